"""The chunk walk of the exact running sum at its edges, and the barrier pass's
load widths (GPU)."""
import numpy as np
import pytest

from tests.test_kmc2d_gpu import _prefix_gpu

pytestmark = pytest.mark.gpu

CHUNK, WINDOW = 2048, 4096  # rates per chunk, chunks per window of the walk


def _rates(n, seed=11):
    return 1e13 * np.exp(-np.random.default_rng(seed).normal(1.0, 0.15, n) / 0.02585)


@pytest.mark.parametrize("case", ["c-1", "c", "c+1", "c+3", "c+4", "3c+255", "3c+257", "window+", "all_zero",
                                  "leading_zeros", "zeros_between", "subnormal_start", "inf", "step_edges"])
def test_walk_edges_bit_for_bit(case):
    if case.startswith("c") or case.startswith("3c"):
        k, d = (3, case[2:]) if case.startswith("3c") else (1, case[1:])
        r = _rates(k * CHUNK + int(d or 0))
    elif case == "window+":  # a second window that starts with a full chunk and ends with a short one
        r = _rates(WINDOW * CHUNK + CHUNK + 3)
    elif case == "all_zero":
        r = np.zeros(3 * CHUNK + 5)
    elif case == "leading_zeros":
        r = _rates(5 * CHUNK)
        r[:2 * CHUNK + 17] = 0.0
    elif case == "zeros_between":
        r = _rates(5 * CHUNK)
        r[1:3 * CHUNK - 1] = 0.0
    elif case == "subnormal_start":
        r = _rates(2 * CHUNK)
        r[:300] = 5e-324 * np.arange(300)
    elif case == "inf":
        r = _rates(2 * CHUNK + 9)
        r[CHUNK + 700] = np.inf
    else:  # the sum crosses a binade at the first and last rate of warp steps
        r = np.full(2 * CHUNK, 1.0)
        r[255], r[256], r[511], r[768] = 1e3, 1e4, 1e6, 1e9
    p, tot = _prefix_gpu(r)
    ref = np.cumsum(r)
    assert np.array_equal(p.view(np.int64), ref.view(np.int64))
    assert tot == ref[-1]


@pytest.mark.parametrize("M", [1, 3, 8])
def test_barrier_load_widths_agree(M):
    # a catalog and a stress field at 8-byte offsets (scalar loads) against aligned ones
    import torch
    from mgkmc_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(M)
    nx, ny = 6, 9
    f = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)
    sig, cat, Q0 = 1e9 * f(nx, ny, 2, 2), 0.05 * f(nx, ny, M, 2, 2), f(nx, ny, M)
    soft = torch.where(f(nx, ny, 2) > 1.0, f(nx, ny, 2).abs(), torch.zeros((), dtype=torch.float64, device="cuda"))
    when = -f(nx, ny).abs()

    def shifted(t):
        b = torch.empty(t.numel() + 1, dtype=torch.float64, device="cuda")
        b[1:] = t.reshape(-1)
        return b[1:]

    out = []
    for a, b in ((sig, cat), (shifted(sig), shifted(cat))):
        Q = torch.zeros_like(Q0)
        L.check(L.lib().mgk_kmc2d_barrier(nx, ny, M, L.ptr(Q), L.ptr(Q0), L.ptr(a), L.ptr(b), 1.0,
                                          L.ptr(soft.contiguous()), L.ptr(when), 0.5, None, 2.0, 0, 0.7,
                                          L.stream_ptr()), "barrier")
        out.append(Q)
    assert torch.equal(out[0], out[1])
