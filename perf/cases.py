"""The calls a user of this framework makes, as measurable cases.

Each case is a dict of plain values; ``listed`` names the fixed ones, ``draw``
gives more of the same ranges.  ``prepare`` builds what a user's program holds
before the call (inputs on the GPU, a plan), ``run`` makes one call through
the public entry points and returns its whole outputs, ``work`` states the
bytes and operations the call cannot do without and ``exact`` its value from
plain torch in 64 bits.

Kinds of cases:

* ``dropin2d``  spectral_solver_2d on numpy arrays, as the reference's own
  drivers call it (one solve per call, host data in and out);
* ``ls2d``      a 2D plan on device-resident fields: one grid or a batch of
  grids per call, linear, secant or Landau material, FP64 or mixed precision,
  cold (material set, solved from the macro strain) or warm (new eigenstrain,
  started from the previous field);
* ``ls3d``      the same in 3D;
* ``fs3d``      one finite-strain load step with stress-controlled lateral
  directions, FP64 or mixed;
* ``rates``     the rate step of a KMC/AQS step: barriers, rates and their
  total, with the reference's sequential sum ("exact") or fused ("fast");
* ``traj2d``    a whole call: a KMC trajectory up to its first events.
"""
import math

import numpy as np
import torch

from mgkmc_b200 import workloads as W
from mgkmc_b200.finite_strain_simulator import Fs3dSolver
from mgkmc_b200.kmc import Kmc2D, pure_shear_modes
from mgkmc_b200.linear_elastic_simulator import Ls2dBatch, Ls3dBatch, spectral_solver_2d

F64 = torch.float64
# Landau coefficients v1, v2, v3, g1, g2, g3, g4 (Pa) of the tests and the benchmark
LANDAU = (-199.7e9, -75.4e9, -23.1e9, 1432.0e9, 311.0e9, 145.0e9, -273.0e9)
SECANT = (0.3, 50.0)  # degradation depth d and rate k of the benchmark's secant law
KB_EV, GPA_NM3_TO_EV = 8.617e-5, 6.241509


def listed():
    return [
        # the smallest call: the reference's KMC driver re-solving a 64^2 grid through the drop-in,
        # numpy in and out, at the drop-in's default tolerance; launches, copies and the host count
        dict(name="dropin2d_64", kind="dropin2d", grids="64x64", tol=1e-6, plane="plane_strain"),
        # the benchmark's workload: 32 different 256^2 problems solved as one mixed-precision batch
        dict(name="ls2d_256x32_mixed", kind="ls2d", grids="256x256*32", law="linear", prec="mixed", warm=False, tol=1e-8,
             plane="plane_strain"),
        # one round of a KMC ensemble in one ragged FP64 plan: the sides of the ensemble workload,
        # new eigenstrains, each replica started from its previous field
        dict(name="ls2d_ragged_warm", kind="ls2d", grids="128x128,192x192,256x256,384x384,512x512", law="linear",
             prec="fp64", warm=True, tol=1e-6, plane="plane_strain"),
        # one large sample solved alone in the mixed form (the serving stream's largest side)
        dict(name="ls2d_1024_mixed", kind="ls2d", grids="1024x1024", law="linear", prec="mixed", warm=False, tol=1e-8,
             plane="plane_strain"),
        # sides that are not powers of two, as a user's sample has them, plane stress
        dict(name="ls2d_odd_fp64", kind="ls2d", grids="288x216,162x243,432x324", law="linear", prec="fp64", warm=False,
             tol=1e-8, plane="plane_stress"),
        # the Landau law with Anderson mixing of depth 5 (the solver's default): one load step
        dict(name="landau2d_256", kind="ls2d", grids="256x256", law="landau", prec="fp64", warm=False, tol=1e-8,
             plane="plane_strain"),
        # a small 3D sample with ragged sides, the reference's arithmetic
        dict(name="ls3d_72x54x48", kind="ls3d", grids="72x54x48", law="linear", prec="fp64", warm=False, tol=1e-6),
        # the 3D trajectory's re-solve at its largest side, FP64 and from the previous field
        dict(name="ls3d_128_warm", kind="ls3d", grids="128x128x128", law="linear", prec="fp64", warm=True, tol=1e-6),
        # one finite-strain load step at a small side in the reference's arithmetic
        dict(name="fs3d_64_fp64", kind="fs3d", n=64, model="neo_hookean", prec="fp64", strain=0.005),
        # one load step of the finite-strain workload at its own side in the mixed form
        dict(name="fs3d_128_mixed", kind="fs3d", n=128, model="neo_hookean", prec="mixed", strain=0.005),
        # the rate step of a 1024^2 x 8 trajectory with the reference's sequential total
        dict(name="rates_1024_exact", kind="rates", nx=1024, ny=1024, M=8, selection="exact", T=300.0),
        # a whole call: the first events of a 128^2 x 8 trajectory with the driver's defaults
        dict(name="traj2d_128", kind="traj2d", n=128, M=8, events=6, T=300.0),
    ]


def _sides(lo, hi, even):
    out = set()
    for a in range(1 if even else 0, 13):
        for b in range(0, 6):
            if lo <= 2 ** a * 3 ** b <= hi:
                out.add(2 ** a * 3 ** b)
    return sorted(out)


def _side(rng, lo, hi, even=False):
    """A supported side (2^a 3^b), near a log-uniform draw."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_sides(lo, hi, even), key=lambda s: abs(math.log(s / v)))


def draw(rng):
    kind = rng.choice(["dropin2d", "ls2d", "ls2d", "ls2d", "ls3d", "ls3d", "fs3d", "rates", "traj2d"])
    if kind == "dropin2d":
        return dict(kind=kind, grids="%dx%d" % (_side(rng, 32, 512, True), _side(rng, 32, 512)), tol=1e-6,
                    plane=rng.choice(["plane_strain", "plane_stress"]))
    if kind == "ls2d":
        law = rng.choice(["linear", "linear", "linear", "secant", "landau"])
        nx, ny = _side(rng, 48, 1024, True), _side(rng, 48, 1024)
        most = max(1, min(32, 2 ** 21 // (nx * ny)))
        reps = 1 if law == "landau" else max(1, min(most, int(math.exp(rng.uniform(0, math.log(32))))))
        if law == "linear":
            return dict(kind=kind, grids="%dx%d*%d" % (nx, ny, reps), law=law, prec=rng.choice(["fp64", "mixed"]),
                        warm=rng.random() < 0.4, tol=1e-8, plane=rng.choice(["plane_strain", "plane_stress"]))
        return dict(kind=kind, grids="%dx%d*%d" % (nx, ny, reps), law=law, prec="fp64", warm=rng.random() < 0.4, tol=1e-8,
                    plane="plane_strain")
    if kind == "ls3d":
        if rng.random() < 0.3:  # the sides of the 3D workloads, which have the mixed form
            n = rng.choice([64, 96, 128])
            return dict(kind=kind, grids="%dx%dx%d" % (n, rng.choice([64, 96, 128]), rng.choice([64, 96])), law="linear",
                        prec=rng.choice(["fp64", "mixed"]), warm=rng.random() < 0.5, tol=1e-8)
        return dict(kind=kind, grids="%dx%dx%d" % (_side(rng, 24, 128, True), _side(rng, 24, 128), _side(rng, 24, 128)),
                    law=rng.choice(["linear", "linear", "secant"]), prec="fp64", warm=rng.random() < 0.5, tol=1e-6)
    if kind == "fs3d":
        return dict(kind=kind, n=_side(rng, 24, 96, True), model=rng.choice(["neo_hookean", "svk"]),
                    prec=rng.choice(["fp64", "mixed"]), strain=round(rng.uniform(0.002, 0.008), 4))
    if kind == "rates":
        return dict(kind=kind, nx=_side(rng, 64, 1024, True), ny=_side(rng, 64, 1024), M=rng.choice([4, 5, 8, 10]),
                    selection=rng.choice(["exact", "fast"]), T=rng.choice([200.0, 300.0, 400.0]))
    return dict(kind=kind, n=_side(rng, 64, 256, True), M=rng.choice([4, 8]), events=rng.choice([4, 6, 8]),
                T=rng.choice([300.0, 350.0, 400.0]))


# ---------------------------------------------------------------- inputs ---

def _grids(case):
    out = []
    for g in case["grids"].split(","):
        g, _, k = g.partition("*")
        out += [tuple(int(v) for v in g.split("x"))] * int(k or 1)
    return out


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _shear(shape, seed, frac=0.05, gamma0=0.1):
    """In-plane pure-shear eigenstrains on a fraction of the voxels."""
    g, d, n = _gen(seed), len(shape), math.prod(shape)
    k = int(round(frac * n))
    at = torch.randperm(n, generator=g, device="cuda")[:k]
    th = torch.rand(k, generator=g, device="cuda", dtype=F64) * math.pi
    ep = torch.zeros((n, d, d), dtype=F64, device="cuda")
    ep[at, 0, 0], ep[at, 1, 1] = 0.5 * gamma0 * torch.cos(2 * th), -0.5 * gamma0 * torch.cos(2 * th)
    ep[at, 0, 1] = ep[at, 1, 0] = 0.5 * gamma0 * torch.sin(2 * th)
    return ep.reshape(shape + (d, d))


def _problem(case, shape, seed):
    """One equilibrium problem: moduli (E, nu; lam, mu for the nonlinear laws),
    eigenstrain, macro strain and, when warm, the previous field."""
    d = len(shape)
    make = W.ls3d_material_dev if d == 3 else (lambda nx, ny, s, dev: W.ls2d_problem_dev(nx, ny, s, dev)[:2])
    a, b = make(*shape, seed, "cuda")
    law = case.get("law", "linear")
    if law != "linear":
        a, b = a * b / ((1 + b) * (1 - 2 * b)), a / (2 * (1 + b))
    # the nonlinear laws are driven elastically, with the eigenstrain amplitude their tests use
    ep = _shear(shape, seed + 1, gamma0=0.1 if law == "linear" else 0.005)
    eb = np.zeros((d, d))
    if law == "linear":
        eb[0, 0] = 0.01
    else:
        eb[0, 0], eb[1, 1], eb[0, 1], eb[1, 0] = 0.02, -0.006, 0.004, 0.004
        if law == "landau":
            eb *= 0.5
    init = None
    if case.get("warm"):
        # the field before the last flip and the last strain step
        before = ep.clone()
        before[tuple(s // 3 for s in shape)] = 0.0
        init = _solve(case, (a, b, before, eb * 0.999, None))[0].contiguous()
    return a.contiguous(), b.contiguous(), ep, eb, init


def _fs_inputs(case, seed):
    n = case["n"]
    lam, mu, Fp = W.fs3d_material_dev(n, n, n, seed, "cuda")
    F0 = torch.eye(3, dtype=F64, device="cuda").reshape(3, 3, 1, 1, 1).expand(3, 3, n, n, n).contiguous()
    Fb = np.eye(3)
    Fb[0, 0] += case["strain"]
    mask = np.zeros((3, 3), bool)
    mask[1, 1] = mask[2, 2] = True
    return lam, mu, Fp, F0, Fb, mask


def _rate_inputs(case, seed):
    """Material, catalog and barriers, and the state the rate step reads: a
    stress field of solved samples' size, softening of past events, their times."""
    nx, ny, M, g = case["nx"], case["ny"], case["M"], _gen(seed + 5)
    E, nu = W.ls2d_problem_dev(nx, ny, seed, "cuda")[:2]
    cat, Q0 = W.kmc2d_state_dev(nx, ny, M, seed, "cuda")
    sig = 3e8 * torch.randn((nx, ny, 2, 2), generator=g, device="cuda", dtype=F64)
    sig = 0.5 * (sig + sig.transpose(2, 3))
    hit = torch.rand((nx, ny), generator=g, device="cuda", dtype=F64) < 0.05
    soft = torch.where(hit[..., None], torch.rand((nx, ny, 2), generator=g, device="cuda", dtype=F64), 0.0).contiguous()
    when = torch.where(hit, 1e-6 * torch.rand((nx, ny), generator=g, device="cuda", dtype=F64), -math.inf)
    return E, nu, cat, Q0, sig.contiguous(), soft, when.contiguous()


_TRAJ = dict(strain_rate=1e6, step_size=1e-5, q_mean=0.6, q_std=0.15, q_min=0.3)


def _traj_inputs(case, seed):
    n = case["n"]
    E, nu = W.ls2d_problem_dev(n, n, seed, "cuda")[:2]
    cat, Q0 = W.kmc2d_state_dev(n, n, case["M"], seed, "cuda", q_mean=_TRAJ["q_mean"], q_std=_TRAJ["q_std"])
    return E, nu, cat, Q0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dropin2d":
        E, nu, ep, eb, _ = _problem(case, _grids(case)[0], seed)
        return dict(case=case, E=E.cpu().numpy(), nu=nu.cpu().numpy(), ep=ep.cpu().numpy(), eb=eb)
    if kind in ("ls2d", "ls3d"):
        sizes = _grids(case)
        probs = [_problem(case, s, seed + 101 * r) for r, s in enumerate(sizes)]
        if kind == "ls2d":
            plan = Ls2dBatch(sizes, plane_mode=case["plane"], precision=case["prec"])
        else:
            plan = Ls3dBatch(sizes, precision=case["prec"])
        if case["law"] == "secant":
            plan.set_secant(*SECANT)
        elif case["law"] == "landau":
            plan.set_landau(LANDAU)
            plan.set_anderson(5)
        if case["warm"]:
            for r, p in enumerate(probs):
                (plan.set_material if case["law"] == "linear" else plan.set_lame)(r, p[0], p[1], p[2])
        return dict(case=case, plan=plan, probs=probs, eps=[torch.empty_like(p[2]) for p in probs],
                    sig=[torch.empty_like(p[2]) for p in probs])
    if kind == "fs3d":
        lam, mu, Fp, F0, Fb, mask = _fs_inputs(case, seed)
        n = case["n"]
        plan = Fs3dSolver(n, n, n, model=case["model"], precision=case["prec"])
        plan.set_material(lam, mu, Fp)
        return dict(case=case, plan=plan, F0=F0, Fb=Fb, mask=mask, out=[torch.empty_like(F0) for _ in range(3)])
    if kind == "rates":
        E, nu, cat, Q0, sig, soft, when = _rate_inputs(case, seed)
        sim = Kmc2D(E, nu, cat, Q0, T=case["T"], selection=case["selection"])
        sim.sig.copy_(sig)
        sim.soft.copy_(soft)
        sim.t_last.copy_(when)
        sim.time = 1.5e-6
        return dict(case=case, sim=sim)
    E, nu, cat, Q0 = _traj_inputs(case, seed)
    return dict(case=case, seed=seed, fields=(E, nu, cat, Q0), plan=Ls2dBatch([(case["n"], case["n"])]))


# ------------------------------------------------------------------ run ---

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dropin2d":
        return spectral_solver_2d(state["E"], state["nu"], state["eb"], eps_plastic=state["ep"], tol=case["tol"],
                                  plane_mode=case["plane"])
    if kind in ("ls2d", "ls3d"):
        plan, probs = state["plan"], state["probs"]
        for r, p in enumerate(probs):
            if case["warm"]:
                plan.set_eigenstrain(r, p[2])
            elif case["law"] == "linear":
                plan.set_material(r, p[0], p[1], p[2])
            else:
                plan.set_lame(r, p[0], p[1], p[2])
        plan.solve(list(range(len(probs))), [p[3] for p in probs], state["eps"], state["sig"],
                   eps_init=[p[4] for p in probs] if case["warm"] else None, max_iter=400, tol=case["tol"])
        if len(probs) > 16:  # one array of each: a batch of equal grids
            return torch.stack(state["eps"]), torch.stack(state["sig"])
        return state["eps"], state["sig"]
    if kind == "fs3d":
        plan, out = state["plan"], state["out"]
        plan.set_F(state["F0"])
        Fb, _ = plan.step(state["Fb"], (0, 0), np.zeros((3, 3)), state["mask"], 90e9, 0.35, 1e-8, 1e-6, 50, 1e6, 20)
        plan.get(*out)
        return out, Fb
    if kind == "rates":
        sim = state["sim"]
        total = sim.barriers_and_rates()
        if case["selection"] == "fast":
            return sim.Q, total
        return sim.Q, sim.rates, sim.indices, sim.prefix, total
    sim = Kmc2D(*state["fields"], T=case["T"], ls=state["plan"], **_TRAJ)
    r = sim.run(np.random.default_rng(state["seed"]), 100, max_events=case["events"])
    return {"events": np.array([e[:3] for e in r["events"]], dtype=np.int64), "steps": r["steps"],
            "solves": r["solves"], "time": r["time"], "eps_macro": r["eps_macro"], "sig": r["sig"], "eps_p": r["eps_p"]}


# ------------------------------------------------------------------ work ---

def work(case):
    kind = case["kind"]
    if kind in ("dropin2d", "ls2d", "ls3d"):
        by = fl = 0.0
        for s in _grids(case):
            n, d = math.prod(s), len(s)
            c = d * (d + 1) // 2
            iters = 4 if case.get("warm") else 10  # fixed-point iterations of the workloads' contrast
            # in: two moduli, the eigenstrain and the previous field; out: strain and stress
            by += 8.0 * n * ((0 if case.get("warm") else 2) + (4 if case.get("warm") else 3) * d * d)
            # an iteration needs the c components' real transforms both ways and the law
            fl += iters * n * (c * 2 * 2.5 * math.log2(n) + 40.0)
        return dict(bytes=by, flops=fl)
    if kind == "fs3d":
        n = case["n"] ** 3
        # about 100 Krylov iterations a load step: 9 components' real transforms both ways, the tangent product
        return dict(bytes=8.0 * n * (2 + 9 + 9 + 27), flops=100.0 * n * (9 * 2 * 2.5 * math.log2(n) + 300.0))
    if kind == "rates":
        n = case["nx"] * case["ny"]
        m = n * case["M"]
        out = 4 if case["selection"] == "exact" else 1
        return dict(bytes=8.0 * (m * (4 + 1 + out) + n * 7), flops=40.0 * m)
    n = case["n"] ** 2
    solves = 3 * case["events"]
    return dict(bytes=8.0 * n * (solves * 12 + 2 * 9 * case["M"] * case["events"]),
                flops=solves * 8.0 * n * (3 * 2 * 2.5 * math.log2(n) + 40.0))


# ----------------------------------------------------------------- exact ---

def _wave(shape):
    q = torch.stack(torch.meshgrid(*[torch.fft.fftfreq(s, dtype=F64, device="cuda") for s in shape], indexing="ij"), -1)
    q2 = (q * q).sum(-1, keepdim=True)
    return torch.where(q2 > 0, q / torch.sqrt(torch.where(q2 > 0, q2, torch.ones_like(q2))), torch.zeros_like(q))


def _hooke(e, lam, mu):
    eye = torch.eye(e.shape[-1], dtype=F64, device=e.device)
    tr = e.diagonal(dim1=-2, dim2=-1).sum(-1)
    return (lam * tr)[..., None, None] * eye + 2 * mu[..., None, None] * e


def _law(case, lam, mu):
    """The stress of an elastic strain field."""
    d = 2 if case["kind"] != "ls3d" else 3
    law = case.get("law", "linear")
    if law == "linear":
        return lambda e: _hooke(e, lam, mu)
    if law == "secant":
        def secant(e):
            e33 = e[..., 2, 2] if d == 3 else torch.zeros_like(e[..., 0, 0])
            tr3 = (e[..., 0, 0] + e[..., 1, 1] + e33) / 3
            ii = (e[..., 0, 0] - tr3) ** 2 + (e[..., 1, 1] - tr3) ** 2 + (e33 - tr3) ** 2
            sh = e[..., 0, 1] ** 2 + ((e[..., 0, 2] ** 2 + e[..., 1, 2] ** 2) if d == 3 else 0.0)
            eq = torch.sqrt((2.0 / 3.0) * (ii + 2 * sh))
            return _hooke(e, lam, mu * (1 - SECANT[0] * (1 - torch.exp(-SECANT[1] * eq))))
        return secant
    v1, v2, v3, g1, g2, g3, g4 = LANDAU

    def landau(e):  # plane strain: e33 = 0
        eye = torch.eye(2, dtype=F64, device=e.device)
        e2 = e @ e
        I1 = e.diagonal(dim1=-2, dim2=-1).sum(-1)
        I2 = e2.diagonal(dim1=-2, dim2=-1).sum(-1)
        I3 = (e2 @ e).diagonal(dim1=-2, dim2=-1).sum(-1)
        cI = lam * I1 + 0.5 * v1 * I1 ** 2 + v2 * I2 + g1 / 6 * I1 ** 3 + g2 * I1 * I2 + 4 / 3 * g3 * I3
        ce = 2 * (mu + v2 * I1 + 0.5 * g2 * I1 ** 2 + g4 * I2)
        return cI[..., None, None] * eye + ce[..., None, None] * e + (4 * (v3 + g3 * I1))[..., None, None] * e2
    return landau


def _solve(case, prob):
    """The Lippmann-Schwinger fixed point of one problem, in 64 bits."""
    a, b, ep, eb, init = prob
    shape = tuple(a.shape)
    axes = tuple(range(len(shape)))
    eb = torch.as_tensor(eb, dtype=F64, device=a.device)
    if case.get("law", "linear") == "linear":
        stress = case.get("plane") == "plane_stress"
        lame = lambda E, nu: (E * nu / (1 - nu ** 2) if stress else E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu)))
        (lam, mu), (lam0, mu0) = lame(a, b), lame(a.mean(), b.mean())
    else:
        lam, mu, lam0, mu0 = a, b, a.mean(), b.mean()
    law = _law(case, lam, mu)
    n = _wave(shape).to(torch.complex128)
    Bc = (lam0 + mu0) / (mu0 * (lam0 + 2 * mu0))
    eps = eb.expand(shape + eb.shape).clone() if init is None else init + (eb - init.mean(axes))
    hg, hf = [], []
    for _ in range(400):
        tau = torch.fft.fftn(law(eps - ep) - _hooke(eps, lam0, mu0.expand(shape)), dim=axes)
        t = (tau @ n[..., None])[..., 0]
        nt = (n * t).sum(-1)
        tau = (n[..., :, None] * t[..., None, :] + t[..., :, None] * n[..., None, :]) / (2 * mu0)
        tau -= (Bc * nt)[..., None, None] * n[..., :, None] * n[..., None, :]
        new = eb - torch.fft.ifftn(tau, dim=axes).real
        f = new - eps
        diff = float(f.norm() / (eps.norm() + 1e-20))
        eps = new
        if diff < case["tol"]:
            break
        if case.get("law") == "landau":  # Anderson mixing of the last five differences
            hg, hf = (hg + [new.flatten()])[-6:], (hf + [f.flatten()])[-6:]
            if len(hf) > 1:
                dF = torch.stack([hf[i + 1] - hf[i] for i in range(len(hf) - 1)], 1)
                dG = torch.stack([hg[i + 1] - hg[i] for i in range(len(hg) - 1)], 1)
                Q, R = torch.linalg.qr(dF)
                eps = new - (dG @ (torch.linalg.pinv(R) @ (Q.T @ hf[-1]))).reshape(new.shape)
    return eps, law(eps - ep)


def _matmul(a, b):
    return torch.einsum("ij...,jk...->ik...", a, b)


def _fs_exact(case, seed):
    """The load step's Newton-Krylov iteration in 64 bits."""
    lam, mu, Fp, F, Fb, mask = _fs_inputs(case, seed)
    n = case["n"]
    Ev, nuv = 90e9, 0.35
    T = lambda x: x.transpose(0, 1)
    inv = lambda x: torch.linalg.inv(x.permute(2, 3, 4, 0, 1)).permute(3, 4, 0, 1, 2).contiguous()
    det = lambda x: torch.linalg.det(x.permute(2, 3, 4, 0, 1))
    eye = torch.eye(3, dtype=F64, device="cuda").reshape(3, 3, 1, 1, 1)
    Fpi = inv(Fp)
    q = _wave((n, n, n))[:, :, : n // 2 + 1].permute(3, 0, 1, 2)
    keep = torch.ones((n, n, n // 2 + 1), dtype=F64, device="cuda")
    if n % 2 == 0:
        keep[n // 2], keep[:, n // 2], keep[:, :, n // 2] = 0, 0, 0
    xi = (q * keep).to(torch.complex128)

    def project(A):
        H = torch.fft.rfftn(A, dim=(2, 3, 4))
        v = torch.einsum("ij...,j...->i...", H, xi)
        return torch.fft.irfftn(v[:, None] * xi[None], s=(n, n, n), dim=(2, 3, 4))

    def material(F):
        Fe = _matmul(F, Fpi)
        C = _matmul(T(Fe), Fe)
        if case["model"] == "svk":
            Eg = 0.5 * (C - eye)
            S, Ci, c = 2 * mu * Eg + lam * torch.einsum("ii...->...", Eg) * eye, None, mu
        else:
            Ci, lnJ = inv(C), torch.log(det(Fe))
            S, c = mu * eye + (lam * lnJ - mu) * Ci, mu - lam * lnJ
        return Fe, Ci, c, _matmul(_matmul(Fpi, S), T(Fpi)), _matmul(_matmul(Fe, S), T(Fpi))

    def tangent(m, d):
        Fe, Ci, c, Sref, _ = m
        X = _matmul(_matmul(T(Fe), d), Fpi)
        Xs = X + T(X)
        if Ci is None:
            Y = c * Xs + lam * torch.einsum("ii...->...", X) * eye
        else:
            Y = lam * torch.einsum("ij...,ij...->...", Ci, X) * Ci + c * _matmul(_matmul(Ci, Xs), Ci)
        return _matmul(Sref, T(d)) + _matmul(_matmul(Fpi, Y), T(Fe))

    Fb, prev = Fb.copy(), None
    for _ in range(20):
        dbar = (torch.as_tensor(Fb, dtype=F64, device="cuda") - F.mean((2, 3, 4))).reshape(3, 3, 1, 1, 1)
        m = material(F)
        for it in range(50):
            r = -project(tangent(m, dbar.expand_as(F))) if it == 0 else -project(m[4])
            x, p = torch.zeros_like(F), r.clone()
            rr = bb = float((r * r).sum())
            for _ in range(150):
                if not rr > 1e-12 * bb:
                    break
                w = project(tangent(m, p))
                alpha = rr / float((p * w).sum())
                x, r = x + alpha * p, r - alpha * w
                new = float((r * r).sum())
                p, rr = r + (new / rr) * p, new
            F = F + x + (dbar if it == 0 else 0)
            m = material(F)
            if it > 0 and float(x.norm()) / float(F.norm()) < 1e-8:
                break
        sig = _matmul(m[4], T(F)) / det(F)
        mean = sig.mean((2, 3, 4)).cpu().numpy()
        err = np.where(mask, -mean, 0.0)
        if np.max(np.abs(err)) < 1e6:
            break
        dF = np.clip((err - nuv * np.trace(err) * np.eye(3)) / Ev, -0.01, 0.01)
        for k in (1, 2):
            step = dF[k, k]
            if prev is not None and abs(Fb[k, k] - prev[0][k]) > 1e-14:
                slope = (mean[k, k] - prev[1][k]) / (Fb[k, k] - prev[0][k])
                if np.isfinite(slope) and slope > 0.01 * Ev:
                    step = min(0.01, max(-0.01, err[k, k] / slope))
            dF[k, k] = step
        prev = (np.diag(Fb).copy(), np.diag(mean).copy())
        for k in (1, 2):
            Fb[k, k] += dF[k, k]
    return [F, m[4], sig], Fb


def _rates_exact(case, seed):
    _, _, cat, Q0, sig, soft, when = _rate_inputs(case, seed)
    tau = 1.0 / (1e13 * math.exp(-0.37 / (KB_EV * case["T"])))
    g = soft[..., 0] + torch.where(soft[..., 1] > 0, soft[..., 1] * torch.exp(-(1.5e-6 - when) / tau), 0.0)
    g = torch.clamp_max(g, 2.0)[..., None]
    w = (sig[:, :, None] * cat).sum((-1, -2))
    Q = Q0 * torch.exp(-g) - 0.5 * (w / 1e9) * GPA_NM3_TO_EV
    beta = 1.0 / (KB_EV * case["T"])
    rates = (1e13 * torch.exp(-torch.clamp_min(Q, 0.0) * beta)).flatten()
    if case["selection"] == "fast":
        return Q, float(rates.sum())
    prefix = torch.cumsum(rates, 0)
    return Q, rates, None, prefix, float(prefix[-1])


def _traj_exact(case, seed):
    """The trajectory's host logic (waiting times, selection, redraws, stress
    control) on 64-bit torch solves."""
    E, nu, cat, Q0 = _traj_inputs(case, seed)
    cat, Q0, n, M = cat.clone(), Q0.clone(), case["n"], case["M"]
    E0, nu0 = float(E.mean()), float(nu.mean())
    rng, ep = np.random.default_rng(seed), torch.zeros((n, n, 2, 2), dtype=F64, device="cuda")
    eb, time, events, solves = np.zeros((2, 2)), 0.0, [], 0
    ls, beta = dict(kind="ls2d", tol=1e-6), 1.0 / (KB_EV * case["T"])
    out = {}

    def elastic():
        out["sig"] = _solve(ls, (E, nu, ep, eb, None))[1]
        return out["sig"].mean((0, 1)).cpu().numpy()

    elastic()
    solves += 1
    dt = _TRAJ["step_size"] / _TRAJ["strain_rate"]
    for done in range(100):
        remaining = dt
        while remaining > 0:
            w = (out["sig"][:, :, None] * cat).sum((-1, -2))
            Q = Q0 - 0.5 * (w / 1e9) * GPA_NM3_TO_EV
            acc = torch.cumsum(1e13 * torch.exp(-torch.clamp_min(Q, 0.0) * beta).flatten(), 0)
            wait = -math.log(rng.random()) / float(acc[-1])
            if wait >= remaining:
                eb[0, 0] += _TRAJ["strain_rate"] * remaining
                time += remaining
                break
            time += wait
            eb[0, 0] += _TRAJ["strain_rate"] * wait
            remaining -= wait
            f = int(torch.searchsorted(acc, rng.random() * acc[-1]))
            x, y, m = f // (n * M), (f // M) % n, f % M
            new = torch.as_tensor(pure_shear_modes(rng.uniform(0.0, np.pi, M), 0.1), device="cuda")
            q0 = np.clip(rng.normal(_TRAJ["q_mean"], _TRAJ["q_std"], M), _TRAJ["q_min"], None)
            ep[x, y] += cat[x, y, m]
            cat[x, y], Q0[x, y] = new, torch.as_tensor(q0, device="cuda")
            events.append((x, y, m))
            elastic()
            solves += 1
            if len(events) >= case["events"]:
                return {"events": np.array(events, dtype=np.int64), "steps": done, "solves": solves, "time": time,
                        "eps_macro": eb, "sig": out["sig"].cpu().numpy(), "eps_p": ep.cpu().numpy()}
        prev = None
        for _ in range(50):
            s = float(elastic()[1, 1])
            solves += 1
            if abs(s) < 1e4:
                break
            step = (-s + nu0 * s) / E0
            if prev is not None and abs(eb[1, 1] - prev[0]) > 1e-14:
                slope = (s - prev[1]) / (eb[1, 1] - prev[0])
                if np.isfinite(slope) and slope > 0.01 * E0:
                    step = -s / slope
            prev = (eb[1, 1], s)
            eb[1, 1] += step
    return None


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dropin2d", "ls2d", "ls3d"):
        probs = [_problem(case, s, seed + 101 * r) for r, s in enumerate(_grids(case))]
        got = [_solve(case, p) for p in probs]
        if kind == "dropin2d":
            e, s = got[0]
            return e, s, e.mean((0, 1)), s.mean((0, 1))
        if len(got) > 16:
            return torch.stack([g[0] for g in got]), torch.stack([g[1] for g in got])
        return [g[0] for g in got], [g[1] for g in got]
    if kind == "fs3d":
        return _fs_exact(case, seed)
    if kind == "rates":
        return _rates_exact(case, seed)
    return _traj_exact(case, seed)
