"""The timing hook on a plan with Anderson mixing that has not solved yet: its first
passes find no mix (GPU)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 64), (12, 6)])
def test_profile_before_the_first_solve(shape):
    import torch
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch
    E, nu, ep, eb = W.ls2d_problem(*shape, seed=1)
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (lam, mu, 0.05 * ep)]
    out = []
    for profiled in (False, True):
        plan = Ls2dBatch([shape])
        plan.set_secant(0.3, 50.0)
        plan.set_anderson(2)
        plan.set_lame(0, *t)
        if profiled:
            assert all(ms > 0 for ms in plan.profile_kernels([0], [eb], n=3))
        eps = torch.empty(shape + (2, 2), dtype=torch.float64, device="cuda")
        info = plan.solve([0], [0.3 * np.asarray(eb)], [eps], None, max_iter=200, tol=1e-8)[0]
        out.append((eps.cpu().numpy(), info.iterations, info.final_diff))
    assert out[0][1:] == out[1][1:] and np.array_equal(out[0][0], out[1][0])
