"""The work that programs using this framework have it do, as cases that can be timed.

Every case goes through the public Python API on seeded synthetic inputs (the distributions of
`shakti.jl_b200/configs.py`, generated on the device).  The kinds:

  step       one timestep (`step`): melt input, Picard loop to convergence, gap update
  parabolic  one timestep of the parabolic head scheme (e_v > 0): one linear solve, fields, gap
  solve      one assembled linear solve (`solve_elliptic_linear_system`), the seam a host program
             with its own Picard loop calls
  fields     the fused field update (`picard_tail`), the other half of that seam
  ensemble   one timestep of a ragged ensemble (`Ensemble.run`)
  train      one training step of the warm-start network: forward, backward, Adam

Steps and solves start from a stored state that is put back first, as a study that branches from a
saved state does, so that every pass does the same work.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

YEAR = 365 * 86400.0
GROUNDED, OCEAN, LAND, OTHER = 0, 1, 2, 3
# Default ModelParameters, as the exact results need them.
RHO_W, RHO_SW, RHO_I, GRAV, NU, OMEGA, LATENT = 1000.0, 1027.0, 910.0, 9.81, 1.787e-6, 1e-4, 334e3
BR, LR, CT, CW = 0.05, 2.0, 7.5e-8, 4.22e3
EVOLVING = ("h", "N", "K", "mdot", "b", "beta", "b_x", "b_y", "pw", "dhdx", "dhdy", "dpwdx", "dpwdy")


def listed():
    return [
        # The plain 64 x 64 workload: Chebyshev(4), Krylov's default tolerances, dt of one hour.
        dict(name="step_chebyshev_64", kind="step", nx=64, ny=64, dx=10e3 / 63, precond="chebyshev", rule="krylov",
             rtol=0.0, gap="implicit", kface="arithmetic", C=1e4, dt=3600.0, melt="constant"),
        # A small odd-sized catchment with the other k-face and gap schemes, Jacobi.
        dict(name="step_jacobi_201x150", kind="step", nx=201, ny=150, dx=156.25, precond="jacobi", rule="relres",
             rtol=1e-12, gap="explicit", kface="harmonic", C=0.25, dt=1800.0, melt="constant"),
        # The 1024 x 1024 drop-in workload (100 km, Harmonic k-faces, dt 1800 s), both plain
        # preconditioners, at the tolerance of a parity run.
        dict(name="step_jacobi_1024", kind="step", nx=1024, ny=1024, dx=100e3 / 1023, precond="jacobi",
             rule="relres", rtol=1e-12, gap="implicit", kface="harmonic", C=1e4, dt=1800.0, melt="constant"),
        dict(name="step_chebyshev_1024", kind="step", nx=1024, ny=1024, dx=100e3 / 1023, precond="chebyshev",
             rule="relres", rtol=1e-12, gap="explicit", kface="harmonic", C=1e4, dt=1800.0, melt="constant"),
        # Its parabolic run (e_v = 1e-3) on a domain that is not square.
        dict(name="parabolic_1000x600", kind="parabolic", nx=1000, ny=600, dx=100e3 / 1023, precond="jacobi",
             rule="relres", rtol=1e-12, gap="implicit", kface="harmonic", C=0.25, dt=1800.0, melt="constant", e_v=1e-3),
        # One tight multigrid solve for a host program's own Picard loop, odd sizes.
        dict(name="solve_multigrid_385x301", kind="solve", nx=385, ny=301, dx=100e3 / 2047, precond="multigrid",
             rule="relres", rtol=1e-12, kface="arithmetic", C=0.25, melt="seasonal"),
        # The seasonal workload in the mixed-precision multigrid form: a small, a mid and the
        # benchmark's own size (200 km at 49 m), rel-res 1e-8.
        dict(name="step_multigrid_256", kind="step", nx=256, ny=256, dx=100e3 / 2047, precond="multigrid",
             rule="relres", rtol=1e-8, gap="implicit", kface="arithmetic", C=0.25, dt=1800.0, melt="seasonal"),
        dict(name="step_multigrid_1024", kind="step", nx=1024, ny=1024, dx=100e3 / 2047, precond="multigrid",
             rule="relres", rtol=1e-8, gap="implicit", kface="arithmetic", C=0.25, dt=1800.0, melt="seasonal"),
        dict(name="step_multigrid_4096", kind="step", nx=4096, ny=4096, dx=200e3 / 4095, precond="multigrid",
             rule="relres", rtol=1e-8, gap="implicit", kface="arithmetic", C=0.25, dt=1800.0, melt="seasonal"),
        # A ragged parameter study, every instance advanced together (128^2 to 512^2).
        dict(name="ensemble_multigrid_20", kind="ensemble", members=20, smallest=128, largest=512,
             precond="multigrid", rule="relres", rtol=1e-8),
        # The field update of a large ragged domain, for a host program's own Picard loop.
        dict(name="fields_2501x1803", kind="fields", nx=2501, ny=1803, dx=100e3 / 2047, C=0.25, melt="seasonal"),
        # Training the warm start: a batch of 32 crops of 32 x 32, as its training run uses.
        dict(name="train_32x32", kind="train", batch=32, side=32),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step"] * 5 + ["parabolic", "solve", "fields", "ensemble", "train"])
    c = dict(kind=kind)
    if kind == "train":
        return dict(c, batch=rng.choice([4, 8, 16, 24, 32, 40]), side=rng.choice([16, 24, 32, 40, 48]))
    if kind == "ensemble":
        lo = rng.choice([65, 96, 128, 160])
        return dict(c, members=rng.randint(4, 20), smallest=lo, largest=rng.choice([193, 256, 300, 384, 512]),
                    precond=rng.choice(["multigrid", "multigrid", "jacobi"]), rule="relres", rtol=1e-8)
    if kind == "fields":
        nx = side(200, 3000)
        return dict(c, nx=nx, ny=max(100, int(nx * rng.uniform(0.5, 1.4))), dx=100e3 / 2047, C=0.25,
                    melt=rng.choice(["seasonal", "constant"]))
    kface, gap = rng.choice(["arithmetic", "harmonic"]), rng.choice(["implicit", "explicit"])
    if kind == "solve":
        nx = side(96, 700)
        return dict(c, nx=nx, ny=max(64, min(700, int(nx * rng.uniform(0.6, 1.5)))), dx=100e3 / 2047,
                    precond=rng.choice(["multigrid", "multigrid", "jacobi", "chebyshev"]), rule="relres", rtol=1e-12,
                    kface=kface, C=0.25, melt="seasonal")
    c.update(gap=gap, kface=kface, C=0.25, dt=1800.0, rule="relres")
    if kind == "parabolic":
        nx = side(80, 1000)
        return dict(c, nx=nx, ny=max(64, min(1000, int(nx * rng.uniform(0.6, 1.4)))), dx=100e3 / 1023,
                    precond=rng.choice(["jacobi", "chebyshev", "multigrid"]), rtol=1e-12, melt="constant", e_v=1e-3)
    if rng.random() < 0.5:  # the plain forms
        nx = side(40, 800)
        return dict(c, nx=nx, ny=max(32, min(1000, int(nx * rng.uniform(0.6, 1.5)))), dx=rng.choice([156.25, 100e3 / 1023]),
                    precond=rng.choice(["jacobi", "chebyshev"]), rtol=1e-12, melt="constant")
    nx = side(96, 2600)
    return dict(c, nx=nx, ny=max(96, int(nx * rng.uniform(0.6, 1.3))), dx=100e3 / 2047, precond="multigrid", rtol=1e-8,
                gap="implicit", kface="arithmetic", melt="seasonal")


# ---------------------------------------------------------------------------------------------
# Inputs.  Device tensors of shape (rows along y, columns along x): the fields' memory order.
# ---------------------------------------------------------------------------------------------
def _blobs(mask, rng, frac):
    """LAND and OTHER_BASIN disks over `frac` of the cells (mask: uint8 array (ny, nx))."""
    ny, nx = mask.shape
    rmax = max(2, min(nx, ny) // 100)
    painted, k = 0, 0
    while painted < frac * nx * ny:
        r = int(rng.integers(max(1, rmax // 4), rmax + 1))
        cx, cy = int(rng.integers(r + 2, nx - r - 1)), int(rng.integers(r, ny - r))
        jj, ii = np.ogrid[-r:r + 1, -r:r + 1]
        sub = mask[cy - r:cy + r + 1, cx - r:cx + r + 1]
        fresh = (ii * ii + jj * jj <= r * r) & (sub == GROUNDED)
        sub[fresh] = (LAND, OTHER)[k % 2]
        painted += int(fresh.sum())
        k += 1


def _inputs(nx, ny, dx, seed, melt, slope=0.01, ieb=1e-8, b0=0.005, spread=0.001):
    gen = torch.Generator("cuda").manual_seed(int(seed) * 7919 + nx * 31 + ny)
    f64 = dict(dtype=torch.float64, device="cuda")
    x = torch.arange(nx, **f64) * dx
    mask = np.zeros((ny, nx), dtype=np.uint8)
    base = torch.zeros((ny, nx), **f64)
    if melt == "seasonal":
        rng = np.random.default_rng(int(seed) + 1)
        _blobs(mask, rng, 0.10)
        grounded = np.flatnonzero(mask.ravel() == GROUNDED)
        n = max(2, min(64, nx * ny // 16384))
        pick = torch.from_numpy(rng.choice(grounded, size=n, replace=False)).cuda()
        base.view(-1)[pick] = torch.from_numpy(rng.uniform(1.0, 20.0, size=n)).cuda() / (dx * dx)
    mask[:, 0] = OCEAN
    base[:, 0] = 0.0
    zb = slope * (dx * (nx - 1) - x) + 5.0 * torch.randn((ny, nx), generator=gen, **f64)
    return dict(mask=torch.from_numpy(mask).cuda().double(), A_visc=torch.full((ny, nx), 5e-25, **f64), zb=zb,
                zs=zb + 6.0 * torch.sqrt(x + 5000.0), b=b0 + spread * (2 * torch.rand((ny, nx), generator=gen, **f64) - 1),
                G=torch.full((ny, nx), 0.05, **f64), ub_x=torch.full((ny, nx + 1), 30.0 / YEAR, **f64),
                ub_y=torch.zeros((ny + 1, nx), **f64), ieb=base if melt == "seasonal" else torch.full((ny, nx), ieb, **f64),
                taub_x=torch.zeros((ny, nx + 1), **f64), taub_y=torch.zeros((ny + 1, nx), **f64))


def _host(t):
    return t.t().contiguous().cpu().numpy()


def _simulation(shk, nx, ny, dx, inputs, case, C, params, dt=1800.0):
    g = shk.Grid(nx, ny, dx * (nx - 1), dx * (ny - 1))
    p = shk.ModelParameters(**params)
    sl = shk.RegularizedCoulombSlidingLaw(C)
    s = shk.State(g)
    shk.set_initial_conditions(s, g, p, sl, **{k: _host(v) for k, v in inputs.items()})
    kw = dict(stop_rule=case["rule"])
    if case["rule"] == "relres":
        kw.update(rtol=case["rtol"], atol=0.0)
    if case["precond"] == "chebyshev":
        kw.update(chebyshev_degree=4)
    ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, multigrid=case["precond"] == "multigrid", **kw)
    ps = shk.PicardSolver(500, 1e-6, ls, g)
    mi = shk.ConstantMeltInput()
    if case.get("melt") == "seasonal" and case["kind"] == "step":
        peak = 5e-8 * YEAR  # a sinusoid of one year, 5e-8 m/s at its peak, over the moulins
        mi = shk.SeasonalBaseMeltInput(inputs["ieb"].t().cpu().numpy(), t_start=0.0, t_end=1.0, amplitude=-peak / 2,
                                       offset=peak / 2, i_min=0.0, seconds_per_year=YEAR)
    return shk.Simulation(g, s, 1, dt, p, case.get("gap", "implicit"), [], mi, sl, ps=ps, ls=ls,
                          k_face_choice=case.get("kface", "arithmetic"))


def _params(case):
    p = dict(b_min=0.002, b_max=1.0) if case.get("melt") == "seasonal" else {}
    if case["kind"] == "parabolic":
        p["e_v"] = case["e_v"]
    return p


def _members(case, seed):
    rng = np.random.default_rng(int(seed) + 5)
    lo, hi = case["smallest"], case["largest"]
    sizes = sorted({lo, hi, int(round(math.sqrt(lo * hi)))})
    return [dict(n=int(sizes[k % len(sizes)]), seed=int(seed) * 100 + k, slope=float(rng.uniform(0.005, 0.02)),
                 ieb=float(rng.uniform(1e-9, 1e-7)), C=float(rng.uniform(0.1, 1.0)), b0=float(rng.uniform(0.003, 0.01)))
            for k in range(case["members"])]


def _training_batch(case, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed) + 11)
    n, s = case["batch"], case["side"]
    X = torch.randn((n, s, s, 16), generator=gen, device="cuda")
    X[..., 7:] = 0.0
    T = torch.randn((n, s, s), generator=gen, device="cuda")
    M = (torch.rand((n, s, s), generator=gen, device="cuda") < 0.9).float()
    return X.bfloat16(), T, M


def prepare(case, seed):
    shk = load_package()
    kind = case["kind"]
    if kind == "train":
        from shakti_b200 import warmstart
        net = warmstart.WarmStartNet(seed=int(seed))
        weights = [net.P[k][f] for k in net.P for f in ("w", "b", "wb", "wt", "mw", "vw", "mb", "vb")]
        return dict(kind=kind, net=net, batch=_training_batch(case, seed), weights=weights,
                    stored=[w.clone() for w in weights])
    if kind == "ensemble":
        sims = []
        for m in _members(case, seed):
            inputs = _inputs(m["n"], m["n"], 156.25, m["seed"], "constant", slope=m["slope"], ieb=m["ieb"], b0=m["b0"],
                             spread=0.2 * m["b0"])
            sims.append(_simulation(shk, m["n"], m["n"], 156.25, inputs, case, m["C"], dict(b_min=0.002, b_max=1.0)))
        ens = shk.Ensemble(sims, autotune_iters=0)
        live = [s.state[f] for s in sims for f in EVOLVING]
        return dict(kind=kind, ens=ens, sims=sims, live=live, stored=[t.clone() for t in live])
    inputs = _inputs(case["nx"], case["ny"], case["dx"], seed, case["melt"])
    full = dict(case, rule=case.get("rule", "krylov"), precond=case.get("precond", "jacobi"))
    sim = _simulation(shk, case["nx"], case["ny"], case["dx"], inputs, full, case["C"], _params(case),
                      case.get("dt", 1800.0))
    if kind == "fields":  # a head that has moved since the fields were set
        sim.state.h += torch.sin(torch.arange(case["ny"], device="cuda").double() * 0.1)
    names = {"solve": ("h",), "fields": ()}.get(kind, EVOLVING)
    live = [sim.state[f] for f in names]
    return dict(kind=kind, shk=shk, sim=sim, live=live, stored=[t.clone() for t in live])


def run(state):
    kind = state["kind"]
    if kind == "train":
        net, (X, T, M) = state["net"], state["batch"]
        torch._foreach_copy_(state["weights"], state["stored"])
        net.step_no = 0
        loss = net.loss_and_grad(X, T, M)
        net.adam_step()
        names = ("enc0a", "enc1b", "enc3a", "enc3b", "dec2a", "dec1b", "dec0a", "head")
        return dict(loss=loss, gradients={k: net.P[k]["gw"] for k in net.P}, bias={k: net.P[k]["gb"] for k in net.P},
                    weights={k: net.P[k]["w"] for k in names})
    if state["live"]:
        torch._foreach_copy_(state["live"], state["stored"])
    if kind == "ensemble":
        state["ens"].run(1)
        return [[s.state.h, s.state.N, s.state.b] for s in state["sims"]]
    shk, sim = state["shk"], state["sim"]
    s = sim.state
    if kind == "solve":
        shk.solve_elliptic_linear_system(sim.ls, s, sim.grid, sim.p, sim.kfs, sim.sl)
        return s.h
    if kind == "fields":
        shk.picard_tail(sim.ls, s, sim.p, sim.sl)
        return {f: s[f] for f in ("pw", "N", "q_x", "q_y", "Re", "shear", "mdot", "K")}
    shk.step(sim)
    return {f: s[f] for f in ("h", "N", "b", "q_x", "q_y", "mdot", "K")}


def work(case):
    kind = case["kind"]
    if kind == "train":
        px = case["batch"] * case["side"] ** 2
        layers = [(16, 32, 1), (32, 32, 1), (32, 64, 4), (64, 64, 4), (64, 128, 16), (128, 128, 16), (128, 256, 64),
                  (256, 256, 64), (256, 128, 64), (128, 128, 16), (128, 64, 16), (64, 64, 4), (64, 32, 4), (32, 32, 1),
                  (32, 16, 1)]
        flops = sum(3 * 2 * 9 * a * b * px / d for a, b, d in layers)
        return {"bytes": px * (16 * 2 + 8) + sum(9 * a * b * 4 * 6 for a, b, _ in layers), "flops": flops}
    if kind == "ensemble":
        cells = sum(m["n"] ** 2 for m in _members(case, 0))
        return {"bytes": 30 * 8 * cells, "flops": 200 * cells}
    cells = case["nx"] * case["ny"]
    # Fields read once and written once: the solve reads 10 and writes h; the field update reads 16
    # and writes 18; a timestep reads 18 and writes 23.
    words = {"solve": 11, "fields": 34}.get(kind, 41)
    return {"bytes": 8 * words * cells, "flops": 100 * cells}


# ---------------------------------------------------------------------------------------------
# The same results in plain 64-bit torch, for the cases where one pass has a closed form: a direct
# solve (block elimination) and the field formulas.
# ---------------------------------------------------------------------------------------------
def _initial_fields(case, seed):
    nx, ny, dx = case["nx"], case["ny"], case["dx"]
    s = _inputs(nx, ny, dx, seed, case["melt"])
    m = s["mask"]
    ok = m != OTHER
    s["valid_x"], s["valid_y"] = torch.ones_like(s["ub_x"]), torch.ones_like(s["ub_y"])
    s["valid_x"][:, 1:-1] = (ok[:, :-1] & ok[:, 1:]).double()
    s["valid_y"][1:-1] = (ok[:-1] & ok[1:]).double()
    gr = m == GROUNDED
    ub = torch.zeros_like(s["ub_x"])
    ub[:, 1:-1] = torch.where(gr[:, :-1] & gr[:, 1:], s["ub_x"][:, 1:-1], 0.0)
    s["ub_x"] = ub
    s["lambda"] = 1.5 * s["A_visc"]
    s["b"] = torch.where(gr, s["b"], 0.0)
    H = s["zs"] - (s["zb"] + s["b"])
    s["beta"] = torch.clamp((BR - s["b"]) / LR, min=0.0)
    s["po"] = RHO_I * GRAV * H
    pw = torch.where(m == OCEAN, -RHO_SW * GRAV * torch.clamp(s["zb"], max=0.0), torch.where(gr, s["po"] / 2, 0.0))
    s["pw"] = pw
    s["N"] = torch.where(gr, s["po"] - pw, 0.0)
    s["h"] = pw / (RHO_W * GRAV) + s["zb"]
    s["abs_ub"] = ((s["ub_x"][:, :-1] + s["ub_x"][:, 1:]) / 2).abs()
    s["b_x"], s["b_y"] = _to_faces(s["b"])
    return s


def _to_faces(c):
    x = torch.cat([c[:, :1], (c[:, 1:] + c[:, :-1]) / 2, c[:, -1:]], dim=1)
    y = torch.cat([c[:1], (c[1:] + c[:-1]) / 2, c[-1:]], dim=0)
    return x, y


def _gradients(c, dx, s):
    x, y = torch.zeros_like(s["b_x"]), torch.zeros_like(s["b_y"])
    x[:, 1:-1] = (c[:, 1:] - c[:, :-1]) / dx
    y[1:-1] = (c[1:] - c[:-1]) / dx
    return x * s["valid_x"], y * s["valid_y"]


def _tail(s, dx, C, from_h=True):
    """The fields that follow from the head, in place."""
    if from_h:
        s["pw"] = RHO_W * GRAV * (s["h"] - s["zb"])
        s["N"] = torch.where(s["mask"] == GROUNDED, s["po"] - s["pw"], 0.0)
    sums = {"Re": 0.0, "ut": [], "qd": [], "qp": []}
    dh, dp = _gradients(s["h"], dx, s), _gradients(s["pw"], dx, s)
    Nf, lf, af = _to_faces(s["N"]), _to_faces(s["lambda"]), _to_faces(s["abs_ub"])
    for k, (b, ub) in enumerate(((s["b_x"], s["ub_x"]), (s["b_y"], s["ub_y"]))):
        D = b ** 3 * GRAV * dh[k].abs() / (12 * NU * NU)
        R = 2 * D / (1 + torch.sqrt(1 + 4 * OMEGA * D))
        q = -torch.sign(dh[k]) * NU * R
        ratio = torch.where(af[k] > 0, af[k] / (af[k] + Nf[k].abs() ** 3 * lf[k]), 0.0)
        tau = torch.where(af[k] > 0, Nf[k] * C * ratio ** (1 / 3) * ub / torch.where(af[k] > 0, af[k], 1.0), 0.0)
        mid = (lambda f: (f[:, 1:] + f[:, :-1])) if k == 0 else (lambda f: f[1:] + f[:-1])
        sums["Re"] = sums["Re"] + mid(R) / 4
        for name, f in (("ut", ub * tau), ("qd", q * dh[k]), ("qp", q * dp[k])):
            sums[name].append(mid(f) / 2)
        s["q_x" if k == 0 else "q_y"] = q
    s["Re"] = sums["Re"]
    s["shear"] = sum(sums["ut"]).abs()
    pot, sens = sum(sums["qd"]).abs(), sum(sums["qp"])
    s["mdot"] = (s["G"] + s["shear"] + RHO_W * GRAV * pot + CT * CW * RHO_W * sens) / LATENT
    s["K"] = s["b"] ** 3 * GRAV / (12 * NU * (1 + OMEGA * s["Re"]))
    return s


def _system(s, dx, kface, e_v, dt):
    """Diagonal, east and north couplings and right-hand side of the assembled system."""
    m, K = s["mask"], s["K"]
    fixed = (m == OCEAN) | (m == LAND)
    free = m == GROUNDED
    head = s["zb"] + torch.where(m == OCEAN, -RHO_SW * GRAV * torch.clamp(s["zb"], max=0.0), 0.0) / (RHO_W * GRAV)

    def coupling(a, b):
        """Face conductance over dx^2 as seen from `a` (a slice) towards its neighbour `b`."""
        if kface == "harmonic":
            k = 2 * K[a] * K[b] / (K[a] + K[b] + np.finfo(float).eps)
        else:
            k = (K[a] + K[b]) / 2
        k = torch.where(fixed[b], K[a], torch.where(m[b] == OTHER, 0.0, k))
        return torch.where(free[a], k / (dx * dx), 0.0)

    full = slice(None)
    lo, hi = slice(None, -1), slice(1, None)
    aP, rhs = torch.zeros_like(K), torch.zeros_like(K)
    aE, aN = torch.zeros_like(K), torch.zeros_like(K)
    for a, b, store in (((full, lo), (full, hi), aE), ((full, hi), (full, lo), None), ((lo, full), (hi, full), aN),
                        ((hi, full), (lo, full), None)):
        c = coupling(a, b)
        aP[a] += c
        rhs[a] += torch.where(fixed[b], c * head[b], 0.0)
        if store is not None:
            store[a] = torch.where(free[b], c, 0.0)
    creep = s["A_visc"] * s["N"] ** 2 * s["b"]
    rhs += s["mdot"] * (1 / RHO_W - 1 / RHO_I) - s["beta"] * s["abs_ub"] + creep * s["N"] + s["ieb"]
    if e_v:
        aP += e_v / dt
        rhs += e_v / dt * s["h"]
    else:
        aP += 3 * RHO_W * GRAV * creep
        rhs += creep * (3 * RHO_W * GRAV * s["h"])
    aP = torch.where(free, aP, 1.0)
    rhs = torch.where(free, rhs, torch.where(fixed, head, s["h"]))
    return aP, aE, aN, rhs


def _direct(aP, aE, aN, rhs):
    """Block elimination along y, with one step of refinement."""
    ny, nx = aP.shape
    inv, below = [], None
    for j in range(ny):
        S = torch.diag(aP[j]) - torch.diag(aE[j, :-1], 1) - torch.diag(aE[j, :-1], -1)
        if j:
            S -= aN[j - 1][:, None] * below * aN[j - 1][None, :]
        below = torch.cholesky_inverse(torch.linalg.cholesky(S))
        inv.append(below)

    def solve(b):
        g = [b[0]]
        for j in range(1, ny):
            g.append(b[j] + aN[j - 1] * (inv[j - 1] @ g[j - 1]))
        x = [None] * ny
        for j in range(ny - 1, -1, -1):
            x[j] = inv[j] @ (g[j] if j == ny - 1 else g[j] + aN[j] * x[j + 1])
        return torch.stack(x)

    def apply(x):
        y = aP * x
        y[:, :-1] -= aE[:, :-1] * x[:, 1:]
        y[:, 1:] -= aE[:, :-1] * x[:, :-1]
        y[:-1] -= aN[:-1] * x[1:]
        y[1:] -= aN[:-1] * x[:-1]
        return y

    x = solve(rhs)
    return x + solve(rhs - apply(x))


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("fields", "solve", "parabolic"):
        return None
    s, dx = _initial_fields(case, seed), case["dx"]
    _tail(s, dx, case["C"], from_h=False)
    if kind == "fields":
        s["h"] = s["h"] + torch.sin(torch.arange(case["ny"], device="cuda").double() * 0.1)[:, None]
        _tail(s, dx, case["C"])
        return {f: s[f].t() for f in ("pw", "N", "q_x", "q_y", "Re", "shear", "mdot", "K")}
    s["h"] = _direct(*_system(s, dx, case["kface"], case.get("e_v", 0.0), case.get("dt", 1.0)))
    if kind == "solve":
        return s["h"].t()
    _tail(s, dx, case["C"])
    dt, grow = case["dt"], s["mdot"] / RHO_I + s["beta"] * s["abs_ub"]
    creep = s["A_visc"] * s["N"] ** 3
    b = (s["b"] + dt * grow) / (1 + dt * creep) if case["gap"] == "implicit" else s["b"] + dt * (grow - creep * s["b"])
    s["b"] = torch.where(s["mask"] == GROUNDED, torch.clamp(b, min=0.0), s["b"])
    return {f: s[f].t() for f in ("h", "N", "b", "q_x", "q_y", "mdot", "K")}
