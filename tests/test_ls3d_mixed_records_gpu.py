"""A mixed 3D plan whose replicas get their materials between solves of others: the
FP32 copies are written with each (GPU)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_material_set_after_another_replica_solved():
    # the same replica alone in a plan: the same bits
    import torch
    from mgkmc_b200.linear_elastic_simulator import Ls3dBatch
    shape = (64, 64, 64)
    eb = np.diag([0.01, 0.0, 0.0])
    m = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in W.ls3d_material(*shape, np.random.default_rng(s))]
         for s in (1, 2)]
    scratch = torch.full((8 * 64 ** 3,), np.nan, dtype=torch.float32, device="cuda")  # what freed memory may hold
    del scratch
    torch.cuda.empty_cache()

    def solve(plan, r):
        eps = torch.empty(shape + (3, 3), dtype=torch.float64, device="cuda")
        info = plan.solve([r], [eb], [eps], None, max_iter=200, tol=1e-8)[0]
        return eps.cpu().numpy(), info.iterations, info.status, info.final_diff

    two, one = Ls3dBatch([shape] * 2, precision="mixed"), Ls3dBatch([shape], precision="mixed")
    two.set_material(0, *m[0])
    solve(two, 0)
    two.set_material(1, *m[1])
    one.set_material(0, *m[1])
    a, b = solve(two, 1), solve(one, 0)
    assert a[2] == 0 and a[1:] == b[1:] and np.array_equal(a[0], b[0])
