"""Small-strain solves whose lines have a register FFT, at every such length and
on each axis, against the oracle; 2D in the narrow form (one small grid) and in
the wide form (a batch that fills the GPU).  Tolerance 1e-9 relative on the
fields (both sides solve to an update norm of 1e-10)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W
from oracle import ls as OL

pytestmark = pytest.mark.gpu
LENGTHS = [24, 27, 32, 36, 48, 54, 64, 72, 81, 96, 108, 128, 144, 162, 192, 216, 243, 256, 288, 324, 384, 432, 486, 512,
           576, 648, 729, 768, 864, 972, 1024]


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _solve(cls, shape, n, E, nu, ep, eb):
    import torch
    B = cls([shape] * n)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (E, nu, ep)]
    eps = [torch.empty_like(t[2]) for _ in range(n)]
    sig = [torch.empty_like(t[2]) for _ in range(n)]
    for r in range(n):
        B.set_material(r, *t)
    B.solve(list(range(n)), [eb] * n, eps, sig, max_iter=300, tol=1e-10)
    return [(eps[r].cpu().numpy(), sig[r].cpu().numpy()) for r in (0, n - 1)]


@pytest.mark.parametrize("n", LENGTHS)
def test_2d(n):
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch
    for shape in [(24, n)] + ([(n, 27)] if n % 2 == 0 else []):
        E, nu, ep, eb = W.ls2d_problem(*shape, seed=n)
        o = OL.spectral_solver(E, nu, eb, ep, max_iter=300, tol=1e-10)
        for copies in (1, 300):
            for eps, sig in _solve(Ls2dBatch, shape, copies, E, nu, ep, eb):
                assert rel(eps, o[0]) < 1e-9 and rel(sig, o[1]) < 1e-9


@pytest.mark.parametrize("shape", [(24, 27, 32), (36, 48, 54), (64, 72, 81), (96, 24, 108), (128, 27, 24), (24, 144, 27),
                                   (162, 24, 36), (24, 24, 192), (216, 27, 24), (24, 243, 24), (2, 27, 243), (256, 3, 128),
                                   (4, 256, 216), (192, 32, 24)])
def test_3d(shape):
    from mgkmc_b200.linear_elastic_simulator import Ls3dBatch
    rng = np.random.default_rng(sum(shape))
    E, nu = W.ls3d_material(*shape, rng)
    ep = W.pure_shear_eigenstrain_3d(*shape, rng)
    eb = np.zeros((3, 3))
    eb[0, 0], eb[0, 1], eb[1, 0] = 0.01, 0.002, 0.002
    o = OL.spectral_solver(E, nu, eb, ep, max_iter=300, tol=1e-10)
    eps, sig = _solve(Ls3dBatch, shape, 1, E, nu, ep, eb)[0]
    assert rel(eps, o[0]) < 1e-9 and rel(sig, o[1]) < 1e-9
