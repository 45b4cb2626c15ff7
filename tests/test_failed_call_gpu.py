"""A solve on a plan whose last call ended in a timed-out device wait: its CTAs'
arrival counter was left part-way (GPU)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,precision", [((64, 64), "fp64"), ((64, 96), "mixed"), ((12, 6), "fp64"),
                                             ((24, 27, 32), "fp64"), ((64, 64, 64), "mixed"), ((6, 4, 12), "fp64")])
@pytest.mark.parametrize("left", [1, 3])
def test_next_solve_starts_afresh(shape, precision, left):
    # register and CTA-wide passes; the same solve before and after, to the last bit
    import torch
    from mgkmc_b200 import _lib as L
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch, Ls3dBatch
    d = len(shape)
    plan = (Ls2dBatch if d == 2 else Ls3dBatch)([shape], precision=precision)
    leave = L.lib().mgk_ls2d_leave_arrivals if d == 2 else L.lib().mgk_ls3d_leave_arrivals
    E, nu = W.ls2d_problem(*shape, seed=7)[:2] if d == 2 else W.ls3d_material(*shape, np.random.default_rng(7))
    E, nu = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (E, nu))
    plan.set_material(0, E, nu, None)
    eb = np.zeros((d, d))
    eb[0, 0] = 0.01
    out = []
    for again in range(2):
        if again:
            L.check(leave(plan._h, 0, left, L.stream_ptr()), "leave_arrivals")
        eps = torch.empty(shape + (d, d), dtype=torch.float64, device="cuda")
        info = plan.solve([0], [eb], [eps], None, max_iter=200, tol=1e-8)[0]
        out.append((eps.cpu().numpy(), info.iterations, info.status, info.final_diff))
    assert out[0][2] == 0 and out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])
