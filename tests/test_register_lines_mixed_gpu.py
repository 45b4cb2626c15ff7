"""The FP32 passes of the 2D mixed form at every line length with a register FFT, in
both passes, both kinds of rounding and both widths (GPU).

The FP64 phase of a mixed solve would hide a wrong FP32 pass, so the solves are cut
inside the FP32 phase, where the field is the FP32 one, and compared with the FP64
plan's after as many iterations.  Four iterations of two transforms each way (at most 10
passes) and some 20 roundings per point between them stay below 4 (4 x 10 + 20) 2^-24 =
1.4e-5 of the largest strain.  A whole solve takes as many iterations as in FP64, give or
take two."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W
from tests.test_register_lines_gpu import LENGTHS

pytestmark = pytest.mark.gpu
WARP_LENGTHS = [64, 96, 128, 192, 256, 384, 512, 768, 1024]  # plans of these sides alone have roundings of their own
N = 128


def _check(shape):
    import torch
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch
    E, nu, ep, eb = W.ls2d_problem(*shape, seed=sum(shape))
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (E, nu, ep)]

    def solve(precision, copies, max_iter):
        plan = Ls2dBatch([shape] * copies, precision=precision)
        for r in range(copies):
            plan.set_material(r, *t)
        eps = [torch.empty_like(t[2]) for _ in range(copies)]
        info = plan.solve(list(range(copies)), [eb] * copies, eps, None, max_iter=max_iter, tol=1e-8)[-1]
        return eps[-1].cpu().numpy(), info.iterations, info.status

    want, full = solve("fp64", 1, 4)[0], solve("fp64", 1, 300)[1]
    for copies in (1, N):
        got, it, status = solve("mixed", copies, 4)
        assert it == 4 and status == 1
        assert np.max(np.abs(got - want)) < 1.4e-5 * np.max(np.abs(want))
        assert not np.array_equal(got, want)
        assert abs(solve("mixed", copies, 300)[1] - full) <= 2


@pytest.mark.parametrize("n", LENGTHS)
def test_roundings_of_the_cta_wide_passes(n):
    for shape in [(36, n)] + ([(n, 36)] if n % 2 == 0 else []):
        _check(shape)


@pytest.mark.parametrize("n", WARP_LENGTHS)
def test_roundings_of_the_warp_lines(n):
    for shape in {(64, n), (n, 64)}:
        _check(shape)
