"""GPU parity of the 3D finite-strain Newton-Krylov step (mgk_fs3d_*):
against the reference's golden load step (SVK with F_p) and against the oracle
(SVK / Neo-Hookean, with and without F_p).  Tolerance 1e-9 relative on F, P
and the Cauchy stress (both sides solve to Newton and Krylov tolerances of
1e-10/1e-11, far below it)."""
import numpy as np
import pytest

from mgkmc_b200 import workloads as W
from oracle import fs as OF

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def test_golden_step(golden):
    from mgkmc_b200.finite_strain_simulator import finite_strain_solver_step_3d
    g = golden("fs3d_svk_6")
    lam, mu = OF.lame_3d(g["E"], g["nu"])
    F0 = np.einsum("ij,xyz->ijxyz", np.eye(3), np.ones(g["E"].shape))
    F, P, Sig, K4, Fb = finite_strain_solver_step_3d(
        F0, g["F_bar_in"], Fp=g["Fp"], driving_component=(0, 0), P_target=np.zeros((3, 3)), P_mask=g["P_mask"],
        E_avg=g["E"].mean(), nu_avg=g["nu"].mean(), tol_NW=1e-10, tol_CG=1e-11, max_NW=30, tol_macro=1e3,
        max_iter_macro=30, enable_console=False, model_type="svk", solver="newton_cg", lam=lam, mu=mu)
    assert rel(F, g["F"]) < 1e-9
    assert rel(P, g["P"]) < 1e-9
    assert rel(Sig, g["Sig"]) < 1e-9
    assert np.max(np.abs(Fb - g["F_bar_out"])) < 1e-9


@pytest.mark.parametrize("model,with_fp,shape", [("neo_hookean", True, (16, 16, 16)), ("svk", False, (12, 8, 6)),
                                                 ("neo_hookean", False, (8, 12, 9))])
def test_oracle_step(model, with_fp, shape):
    from mgkmc_b200.finite_strain_simulator import build_finite_strain_bc_3d, finite_strain_solver_step_3d
    rng = np.random.default_rng(sum(shape))
    E, nu, Fp = W.fs3d_material(*shape, rng, fp_frac=0.1)
    Fp = Fp if with_fp else None
    lam, mu = OF.lame_3d(E, nu)
    Fb0, _, Pt, Pm = build_finite_strain_bc_3d((0, 0), 0.02, {(1, 1): 0.0, (2, 2): 0.0})
    F0s = np.broadcast_to(np.eye(3), shape + (3, 3)).copy()
    Fo, Po, So, Fbo = OF.solver_step_3d(F0s, Fb0, E, nu, None if Fp is None else OF.to_spatial(Fp), (0, 0), Pt, Pm,
                                        tol_NW=1e-10, tol_CG=1e-11, max_NW=40, tol_macro=1e3, max_iter_macro=40,
                                        model=model, krylov="cg")
    F0 = OF.to_tensor_first(F0s)
    F, P, Sig, _, Fb = finite_strain_solver_step_3d(
        F0, Fb0, Fp=Fp, driving_component=(0, 0), P_target=Pt, P_mask=Pm, E_avg=E.mean(), nu_avg=nu.mean(),
        tol_NW=1e-10, tol_CG=1e-11, max_NW=40, tol_macro=1e3, max_iter_macro=40, enable_console=False,
        model_type=model, solver="newton_cg", lam=lam, mu=mu)
    assert rel(F, OF.to_tensor_first(Fo)) < 1e-9
    assert rel(P, OF.to_tensor_first(Po)) < 1e-9
    assert rel(Sig, OF.to_tensor_first(So)) < 1e-9
    assert np.max(np.abs(Fb - Fbo)) < 1e-9


def test_load_ramp_runs_and_relaxes_lateral_stress():
    # config-2 shape of the problem at 32^3: F_xx ramped to 1.05 in 10 steps,
    # lateral Cauchy stresses driven to zero
    from mgkmc_b200.finite_strain_simulator import simulate_3d
    rng = np.random.default_rng(2)
    E, nu, Fp = W.fs3d_material(32, 32, 32, rng)
    s, steps = simulate_3d(E, nu, Fp, 0.05, 10, mixed_targets={(1, 1): 0.0, (2, 2): 0.0}, model="neo_hookean",
                           tol_NW=1e-8, tol_CG=1e-6)
    Fb, info = steps[-1]
    assert abs(Fb[0, 0] - 1.05) < 1e-12
    sig = info["sig_mean"]
    assert abs(sig[1, 1]) < 1e6 and abs(sig[2, 2]) < 1e6 and sig[0, 0] > 1e9


@pytest.mark.parametrize("model,with_fp", [("neo_hookean", True), ("svk", False)])
def test_mixed_precision_matches_fp64(model, with_fp):
    # FP32 Krylov matvecs, FP64 Newton residual: the converged fields agree
    # with the FP64 solve within the stated field-error bound of 1e-6 (the
    # macro loop's stress tolerance of 1e3 Pa leaves differences ~1e-8)
    import torch
    from mgkmc_b200.finite_strain_simulator import Fs3dSolver, build_finite_strain_bc_3d
    n = 16
    rng = np.random.default_rng(31)
    E, nu, Fp = W.fs3d_material(n, n, n, rng, fp_frac=0.1)
    lam, mu = OF.lame_3d(E, nu)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    Fb, _, Pt, Pm = build_finite_strain_bc_3d((0, 0), 0.02, {(1, 1): 0.0, (2, 2): 0.0})
    out = {}
    for prec in ("fp64", "mixed"):
        s = Fs3dSolver(n, n, n, model=model, precision=prec)
        s.set_material(t(lam), t(mu), t(Fp) if with_fp else None)
        s.set_F(t(np.einsum("ij,xyz->ijxyz", np.eye(3), np.ones((n, n, n)))))
        Fbo, info = s.step(Fb, (0, 0), Pt, Pm, E.mean(), nu.mean(), 1e-10, 1e-6, 40, 1e3, 40)
        F = torch.empty((3, 3, n, n, n), dtype=torch.float64, device="cuda")
        P = torch.empty_like(F)
        s.get(F, P)
        out[prec] = (F.cpu().numpy(), P.cpu().numpy(), Fbo, info.krylov_iterations)
    assert rel(out["mixed"][0], out["fp64"][0]) < 1e-6
    assert rel(out["mixed"][1], out["fp64"][1]) < 1e-6
    assert np.max(np.abs(out["mixed"][2] - out["fp64"][2])) < 1e-6


def test_host_driven_krylov_loop_matches_graph():
    # the host-driven fallback (no conditional graphs) runs the same arithmetic
    import subprocess, sys, os
    code = ("import numpy as np, torch, sys; sys.path.insert(0, '.');"
            "from mgkmc_b200 import workloads as W; from mgkmc_b200.finite_strain_simulator import simulate_3d;"
            "E, nu, Fp = W.fs3d_material(12, 12, 12, np.random.default_rng(4));"
            "s, st = simulate_3d(E, nu, Fp, 0.01, 2, mixed_targets={(1, 1): 0.0, (2, 2): 0.0});"
            "F = torch.empty((3, 3, 12, 12, 12), dtype=torch.float64, device='cuda'); s.get(F);"
            "np.save(sys.argv[1], F.cpu().numpy())")
    import tempfile
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    outs = []
    with tempfile.TemporaryDirectory() as tmp:
        for flag in ("0", "1"):
            path = os.path.join(tmp, f"F_{flag}.npy")
            env = dict(os.environ, MGK_NO_GRAPH_WHILE=flag)
            subprocess.run([sys.executable, "-c", code, path], cwd=root, env=env, check=True)
            outs.append(np.load(path))
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("shape,model,prec", [((64, 64, 64), "neo_hookean", "fp64"), ((96, 64, 128), "svk", "fp64"),
                                              ((64, 96, 64), "neo_hookean", "mixed")])
def test_warp_line_passes_match_generic(shape, model, prec):
    # the warp-line kernels (sides 64/96/128) against the generic CTA-wide
    # passes, which the oracle tests pin at small sizes: same radix schedule
    # and arithmetic, so the fields agree to rounding
    import subprocess, sys, os, tempfile
    code = ("import numpy as np, torch, sys; sys.path.insert(0, '.');"
            "from mgkmc_b200 import workloads as W; from mgkmc_b200.finite_strain_simulator import simulate_3d;"
            f"sh = {shape!r}; E, nu, Fp = W.fs3d_material(*sh, np.random.default_rng(8));"
            f"s, st = simulate_3d(E, nu, Fp, 0.01, 1, mixed_targets={{(1, 1): 0.0, (2, 2): 0.0}}, model='{model}',"
            f" precision='{prec}', tol_NW=1e-10, tol_CG=1e-8 if '{prec}' == 'fp64' else 1e-6);"
            "F = torch.empty((3, 3) + sh, dtype=torch.float64, device='cuda'); P = torch.empty_like(F); s.get(F, P);"
            "np.save(sys.argv[1], np.stack([F.cpu().numpy(), P.cpu().numpy()]))")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    outs = []
    with tempfile.TemporaryDirectory() as tmp:
        for flag in ("1", "0"):
            path = os.path.join(tmp, f"FP_{flag}.npy")
            subprocess.run([sys.executable, "-c", code, path], cwd=root, env=dict(os.environ, MGK_FS_FAST=flag),
                           check=True)
            outs.append(np.load(path))
    # FP64: the same operations (rounding-level agreement); mixed: FP32
    # matvecs in a different order move the inexact Krylov solves, so the
    # fields agree within the mixed form's stated bound
    tol = (1e-10, 1e-9) if prec == "fp64" else (1e-6, 1e-6)
    assert rel(outs[0][0], outs[1][0]) < tol[0]
    assert rel(outs[0][1], outs[1][1]) < tol[1]


def test_autotune_keeps_results():
    # the finite-strain autotuner picks a kernel family by timing; the next
    # load step gives the same fields whichever family it kept
    import torch
    from mgkmc_b200.finite_strain_simulator import Fs3dSolver, build_finite_strain_bc_3d
    n = 64
    E, nu, Fp = W.fs3d_material(n, n, n, np.random.default_rng(12))
    lam, mu = OF.lame_3d(E, nu)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    Fs = []
    for tune in (False, True):
        s = Fs3dSolver(n, n, n, model="neo_hookean")
        s.set_material(t(lam), t(mu), t(Fp))
        F0 = t(np.einsum("ij,xyz->ijxyz", np.eye(3), np.ones((n, n, n))))
        s.set_F(F0)
        Fb, _, Pt, Pm = build_finite_strain_bc_3d((0, 0), 0.005, {(1, 1): 0.0, (2, 2): 0.0})
        s.step(Fb, (0, 0), Pt, Pm, E.mean(), nu.mean(), 1e-10, 1e-9, 40, 1e3, 40)
        if tune:
            fam, ms = s.autotune(reps=3)
            assert fam in (0, 1) and ms > 0
        Fb2, _, Pt2, Pm2 = build_finite_strain_bc_3d((0, 0), 0.01, {(1, 1): 0.0, (2, 2): 0.0})
        s.set_F(F0)
        s.step(Fb2, (0, 0), Pt2, Pm2, E.mean(), nu.mean(), 1e-10, 1e-9, 40, 1e3, 40)
        F = torch.empty((3, 3, n, n, n), dtype=torch.float64, device="cuda")
        s.get(F)
        Fs.append(F.cpu().numpy())
    assert rel(Fs[1], Fs[0]) < 1e-10


@pytest.mark.parametrize("shape,model,with_fp", [((24, 27, 32), "neo_hookean", True), ((36, 48, 54), "svk", True),
                                                 ((72, 2, 81), "neo_hookean", False), ((96, 3, 108), "svk", False),
                                                 ((128, 4, 144), "neo_hookean", True), ((162, 1, 192), "svk", True),
                                                 ((3, 216, 24), "neo_hookean", True), ((2, 243, 27), "neo_hookean", False),
                                                 ((256, 1, 256), "neo_hookean", True), ((4, 192, 243), "svk", True)])
def test_register_lines_match_general_passes(shape, model, with_fp, monkeypatch):
    # every line length with a register FFT, on each axis beside axes without
    # one, against the general passes (which the oracle tests pin): the same
    # FP64 operations, so the fields of one converged load step agree to
    # rounding (bounds of the test above)
    import torch
    from mgkmc_b200.finite_strain_simulator import Fs3dSolver, build_finite_strain_bc_3d
    lam, mu, Fp = W.fs3d_material_dev(*shape, 3, "cuda")
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("MGK_FS_FAST", flag)
        s = Fs3dSolver(*shape, model=model)
        s.set_material(lam, mu, Fp if with_fp else None)
        F = torch.eye(3, dtype=torch.float64, device="cuda").reshape(3, 3, 1, 1, 1).expand(3, 3, *shape).contiguous()
        s.set_F(F)
        Fb, _, Pt, Pm = build_finite_strain_bc_3d((0, 0), 0.005, {(1, 1): 0.0, (2, 2): 0.0})
        s.step(Fb, (0, 0), Pt, Pm, 90e9, 0.35, 1e-10, 1e-9, 40, 1e3, 40)
        P = torch.empty_like(F)
        s.get(F, P)
        out.append((F.cpu().numpy(), P.cpu().numpy()))
    assert rel(out[0][0], out[1][0]) < 1e-10
    assert rel(out[0][1], out[1][1]) < 1e-9


@pytest.mark.parametrize("shape,model,with_fp", [((24, 27, 32), "neo_hookean", True), ((36, 48, 54), "svk", True),
                                                 ((64, 2, 72), "neo_hookean", False), ((81, 4, 96), "svk", False),
                                                 ((108, 4, 128), "neo_hookean", True), ((144, 1, 162), "svk", True),
                                                 ((3, 192, 216), "neo_hookean", True), ((2, 243, 24), "neo_hookean", False)])
def test_mixed_register_lines_keep_the_general_roundings(shape, model, with_fp, monkeypatch):
    # the mixed form's register FFTs repeat the CTA-wide passes' FP32
    # operations and sums: the same bits, on axes of every length
    import torch
    from mgkmc_b200.finite_strain_simulator import Fs3dSolver, build_finite_strain_bc_3d
    lam, mu, Fp = W.fs3d_material_dev(*shape, 3, "cuda")
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("MGK_FS_FAST", flag)
        s = Fs3dSolver(*shape, model=model, precision="mixed")
        s.set_material(lam, mu, Fp if with_fp else None)
        F = torch.eye(3, dtype=torch.float64, device="cuda").reshape(3, 3, 1, 1, 1).expand(3, 3, *shape).contiguous()
        s.set_F(F)
        Fb, _, Pt, Pm = build_finite_strain_bc_3d((0, 0), 0.005, {(1, 1): 0.0, (2, 2): 0.0})
        _, info = s.step(Fb, (0, 0), Pt, Pm, 90e9, 0.35, 1e-8, 1e-6, 40, 1e6, 40)
        P = torch.empty_like(F)
        s.get(F, P)
        out.append((F.cpu().numpy(), P.cpu().numpy(), info.krylov_iterations))
    assert out[0][2] == out[1][2]
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
