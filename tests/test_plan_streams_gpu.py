"""A new plan used on a stream of its own while the default stream is busy: what
the constructor set up is complete when it returns (GPU)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_finite_strain_plan_on_a_side_stream(precision):
    # both steps solve the same problem with the same kernels: the same bits
    import torch
    from mgkmc_b200.finite_strain_simulator import Fs3dSolver, build_finite_strain_bc_3d
    shape = (24, 27, 32)
    lam, mu, Fp = W.fs3d_material_dev(*shape, 3, "cuda")
    F0 = torch.eye(3, dtype=torch.float64, device="cuda").reshape(3, 3, 1, 1, 1).expand(3, 3, *shape).contiguous()
    Fb, _, Pt, Pm = build_finite_strain_bc_3d((0, 0), 0.005, {(1, 1): 0.0, (2, 2): 0.0})
    side = torch.cuda.Stream()
    out = []
    for stream in (torch.cuda.default_stream(), side):
        torch.cuda.synchronize()
        if stream is side:
            torch.cuda._sleep(200_000_000)  # the default stream, for some 0.1 s
        s = Fs3dSolver(*shape, model="neo_hookean", precision=precision)
        with torch.cuda.stream(stream):
            s.set_material(lam, mu, Fp, stream=stream)
            s.set_F(F0, stream=stream)
            s.step(Fb, (0, 0), Pt, Pm, 90e9, 0.35, 1e-8, 1e-6, 40, 1e6, 40, stream=stream)
            F, P, S = (torch.empty_like(F0) for _ in range(3))
            s.get(F, P, S, stream=stream)
        torch.cuda.synchronize()
        out.append([a.cpu().numpy() for a in (F, P, S)])
    for a, b in zip(*out):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)
