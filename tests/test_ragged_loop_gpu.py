"""A selection of several shapes, solved with the loop driven from the host (the
caller waits for it) and inside a graph (it does not): the same replicas, to the
last bit, whichever others are selected with them (GPU)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W

pytestmark = pytest.mark.gpu
SHAPES = [(64, 64), (54, 81), (128, 96), (12, 6), (64, 64), (192, 72)]  # (12, 6): the CTA-wide passes


def _plan(precision):
    import torch
    from mgkmc_b200.linear_elastic_simulator import Ls2dBatch
    plan = Ls2dBatch(SHAPES, precision=precision)
    eb = []
    for r, s in enumerate(SHAPES):
        E, nu, ep, e = W.ls2d_problem(*s, seed=r)
        plan.set_material(r, *[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (E, nu, ep)])
        eb.append(e)
    return plan, eb


def _solve(plan, eb, sel, sync, max_iter, stream=None):
    import torch
    out = [torch.full(SHAPES[r] + (2, 2), np.nan, dtype=torch.float64, device="cuda") for r in sel]
    torch.cuda.synchronize()
    infos = plan.solve(sel, [eb[r] for r in sel], out, None, max_iter=max_iter, tol=1e-8, sync=sync, stream=stream)
    if not sync:
        infos = plan.collect(sel, stream=stream)
    return {r: (o.cpu().numpy(), i.iterations, i.status, i.final_diff, tuple(i.sig_mean)) for r, o, i in zip(sel, out, infos)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("max_iter", [200, 5, 1, 0])
def test_host_driven_and_graph_loops_agree(precision, max_iter):
    import torch
    plan, eb = _plan(precision)
    side = torch.cuda.Stream(priority=-1)
    want = _solve(plan, eb, list(range(len(SHAPES))), False, max_iter)
    for sel, stream in (([0, 1, 2, 3, 4, 5], None), ([5, 3], None), ([4, 1, 0], side), ([2, 5, 1, 3], side), ([3], None), ([1, 4], None)):
        got = _solve(plan, eb, sel, True, max_iter, stream)
        for r in sel:
            assert got[r][1:] == want[r][1:], (sel, r)
            assert np.array_equal(got[r][0], want[r][0])
        if max_iter == 200:
            assert all(v[2] == 0 for v in got.values())


def test_host_driven_loop_without_graphs(monkeypatch):
    plan, eb = _plan("mixed")
    want = _solve(plan, eb, [0, 1, 3], False, 200)
    monkeypatch.setenv("MGK_NO_GRAPH_WHILE", "1")
    plan, eb = _plan("mixed")
    for sync in (True, False):
        got = _solve(plan, eb, [0, 1, 3], sync, 200)
        for r in got:
            assert got[r][1:] == want[r][1:] and np.array_equal(got[r][0], want[r][0])


def test_a_repeated_selection_moves_to_its_graph():
    # the first uses of a selection run from the host, later ones as a graph
    plan, eb = _plan("mixed")
    out = [_solve(plan, eb, [0, 1, 3, 5], True, 200) for _ in range(7)]
    for got in out[1:]:
        for r in got:
            assert got[r][1:] == out[0][r][1:] and np.array_equal(got[r][0], out[0][r][0])
