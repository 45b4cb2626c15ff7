"""A replica solved alone (the narrow kernels) and with 127 others (the wide ones):
the same fields, iteration count and update norm to the last bit, at every line
length with a register FFT, in both passes, under every law and precision (GPU)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W
from tests.test_register_lines_gpu import LENGTHS

pytestmark = pytest.mark.gpu
N = 128
LANDAU = (-199.7e9, -75.4e9, -23.1e9, 1432.0e9, 311.0e9, 145.0e9, -273.0e9)
LAWS = {"linear": lambda p: None, "secant": lambda p: p.set_secant(0.3, 50.0), "rose": lambda p: p.set_rose(5.0),
        "landau": lambda p: p.set_landau(LANDAU)}


def _check(shape, precision, law):
    import torch
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch
    E, nu, ep, eb = W.ls2d_problem(*shape, seed=sum(shape))
    a, b = E, nu
    if law != "linear":
        a, b, ep, eb = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu)), 0.05 * ep, 0.3 * np.asarray(eb)
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b, ep)]
    plan = Ls2dBatch([shape] * N, precision=precision)
    LAWS[law](plan)
    for r in range(N):
        (plan.set_material if law == "linear" else plan.set_lame)(r, *t)
    out = []
    for k in (1, N):
        eps, sig = ([torch.empty_like(t[2]) for _ in range(k)] for _ in range(2))
        info = plan.solve(list(range(k)), [eb] * k, eps, sig, max_iter=300, tol=1e-8)[0]
        out.append((eps[0].cpu().numpy(), sig[0].cpu().numpy(), info.iterations, info.final_diff))
    assert out[0][2:] == out[1][2:]
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n", LENGTHS)
def test_selection_size_does_not_change_a_replica(n):
    for shape in [(36, n)] + ([(n, 36)] if n % 2 == 0 else []):
        _check(shape, "fp64", "linear")
        _check(shape, "mixed", "linear")
    for law in ("secant", "rose", "landau"):
        _check((36, n), "fp64", law)
