"""What the time stepping is measured on: calls of the public entry points, over the range of
basins, layers, precisions and solvers that the configurations, tests and benchmark of this
repository use.

``listed`` names the fixed cases, ``draw`` gives further ones of the same ranges, ``prepare``
makes what a user's program holds before the call (the model, its plan and the state on the
GPU), ``run`` is one call, ``work`` what the call cannot do without, and ``exact`` the same
result in 64 bits, in plain torch.
"""

import math

import numpy as np
import torch

import somax_gb300 as sg
from somax_gb300 import testcases

F0, BETA = 9.375e-5, 1.754e-11
BASIN = 5.12e6  # the longer side of a QG basin (m)
RHO0 = 1000.0

# Layer thicknesses and reduced gravities by layer count: one layer of 50 km deformation radius,
# the two layers of the shallow-water jet, the three of the double gyre, the five of the ensemble.
STRAT = {
    1: ((4000.0,), ((F0 * 5.0e4) ** 2 / 4000.0,)),
    2: ((500.0, 4500.0), (9.81, 0.025)),
    3: ((400.0, 1100.0, 2600.0), (9.81, 0.025, 0.0125)),
    5: (tuple(200.0 * 10 ** (k / 4) for k in range(5)), (9.81, 0.030, 0.020, 0.0125, 0.008)),
}
# The ragged ensemble's classes: (layers, share of the members, interior cells per side).
CLASSES = ((1, 96, 64), (3, 96, 128), (3, 48, 256), (5, 16, 256))


# ---- the cases -------------------------------------------------------------------------------
def _qg(kind, nx, ny, nl, precision="fp32", refine=0, solver="ssprk3", steps=1, **more):
    return dict(kind=kind, nx=nx, ny=ny, nl=nl, precision=precision, refine=refine, solver=solver, steps=steps, **more)


def _swm(kind, nx, ny, nl, bc, solver="tsit5", steps=1, **more):
    return dict(kind=kind, nx=nx, ny=ny, nl=nl, bc=bc, solver=solver, steps=steps, **more)


def listed():
    return [
        # one tendency of a small odd basin, as an outside integrator or an analysis asks for it
        dict(_qg("rhs", 40, 33, 3), name="rhs_40x33_fp32"),
        # the barotropic double gyre at its default size, a third of a day: a short run of the
        # smallest model, everything latency
        dict(_qg("step", 64, 64, 0, solver="heun", steps=24), name="barotropic_64_fp32"),
        # the reference user's first call: the three-layer double gyre with every default (FP32,
        # Tsit5 through integrate), two saved states
        dict(_qg("integrate", 128, 128, 3, solver="tsit5", steps=12), name="gyre_128_fp32_tsit5"),
        # the headline basin of the benchmark on the tensor-core passes
        dict(_qg("step", 128, 128, 3, "bf16x3", steps=24), name="basin_128_bf16x3"),
        # an eddy-resolving basin with the default FP32 passes
        dict(_qg("step", 512, 512, 3, steps=4), name="basin_512_fp32"),
        # the largest single basin, refined to FP32 accuracy
        dict(_qg("step", 1024, 1024, 3, "bf16x3", 1, steps=2), name="basin_1024_refined"),
        # a basin with a coastline, of odd proportions
        dict(_qg("masked", 250, 190, 3, "bf16x3", 1, steps=4), name="masked_250x190"),
        # the ragged ensemble of the benchmark: 256 members in one plan
        dict(kind="ensemble", scale=1.0, members=256, solver="ssprk3", steps=4, name="ensemble_256"),
        # data assimilation: the gradient of a misfit in the initial state and the wind
        dict(_qg("gradient", 256, 256, 3, "bf16x3", steps=20), name="gradient_256"),
        # the reference's shallow-water jet run
        dict(_swm("swm", 64, 64, 2, "periodic", steps=60), name="swm_jet_64"),
        # a large wall-bounded shallow-water gyre
        dict(_swm("swm", 1024, 1024, 3, "wall", steps=4), name="swm_gyre_1024"),
        # the gradient of a shallow-water misfit
        dict(_swm("swm_gradient", 64, 64, 2, "periodic", steps=40), name="swm_gradient_64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    nx = _log(rng, lo, hi)
    ny = min(hi, max(lo, int(round(nx * rng.uniform(0.6, 1.6)))))
    return nx, ny


def draw(rng):
    kind = rng.choice(["rhs", "step", "step", "integrate", "masked", "ensemble", "gradient", "swm", "swm", "swm_gradient"])
    nl = rng.choice([1, 2, 3, 3, 5])
    precision, refine = rng.choice([("fp32", 0), ("fp32", 0), ("bf16x3", 0), ("bf16x3", 1)])
    if kind == "rhs":
        return _qg(kind, *_sides(rng, 16, 512), rng.choice([0, nl]), precision, refine)
    if kind in ("step", "integrate"):
        nx, ny = _sides(rng, 24, 1024)
        big = nx * ny * nl > 300_000
        solver = rng.choice(["heun", "ssprk3", "ssprk3", "tsit5", "euler"]) if kind == "step" else "tsit5"
        return _qg(kind, nx, ny, rng.choice([0, nl, nl]), precision, refine, solver, rng.randint(2, 3 if big else 24))
    if kind == "masked":
        return _qg(kind, *_sides(rng, 48, 256), rng.choice([2, 3]), *rng.choice([("fp32", 0), ("bf16x3", 1)]),
                   steps=rng.randint(2, 8))
    if kind == "ensemble":
        return dict(kind=kind, scale=rng.uniform(0.4, 1.0), members=_log(rng, 8, 256), solver=rng.choice(["heun", "ssprk3"]),
                    steps=rng.randint(2, 4))
    if kind == "gradient":
        return _qg(kind, *_sides(rng, 24, 256), rng.choice([1, 3]), rng.choice(["fp32", "bf16x3"]),
                   solver=rng.choice(["heun", "ssprk3"]), steps=rng.randint(5, 20))
    nl = rng.choice([1, 2, 3])
    if kind == "swm":
        nx, ny = _sides(rng, 24, 1024)
        return _swm(kind, nx, ny, nl, rng.choice(["periodic", "wall"]), rng.choice(["tsit5", "tsit5", "heun"]),
                    rng.randint(2, 4) if nx * ny * nl > 300_000 else rng.randint(8, 60))
    return _swm(kind, *_sides(rng, 24, 128), nl, rng.choice(["periodic", "wall"]), steps=rng.randint(5, 40))


# ---- parameters and inputs ---------------------------------------------------------------------
def _extent(case):
    d = BASIN / max(case["nx"], case["ny"])
    return d * case["nx"], d * case["ny"]


def _qg_numbers(case):
    """Everything create() takes for a QG case (nl = 0: the barotropic model)."""
    Lx, Ly = _extent(case)
    wind = 0.08 * 2.0 * math.pi / (RHO0 * Ly)
    p = dict(nx=case["nx"], ny=case["ny"], Lx=Lx, Ly=Ly, f0=F0, beta=BETA, lateral_viscosity=15.0, bottom_drag=1e-7,
             wind_amplitude=wind, biharmonic_viscosity=2e9)
    if case["nl"] == 0:
        p["wind_amplitude"] = wind / 4000.0
    else:
        H, g = STRAT[case["nl"]]
        p.update(n_layers=case["nl"], H=H, g_prime=g)
    return p


DT = 1200.0  # time step of every QG case (s)


def _swm_numbers(case):
    H, g = STRAT[case["nl"]] if case["nl"] > 1 else ((1000.0,), (9.81,))
    d = 1.0e6 / 64 if max(case["nx"], case["ny"]) <= 256 else 4.0e6 / 1024
    wall = case["bc"] == "wall"
    return dict(nx=case["nx"], ny=case["ny"], Lx=d * case["nx"], Ly=d * case["ny"], f0=F0, beta=BETA, n_layers=case["nl"], H=H,
                g_prime=g, lateral_viscosity=100.0 if wall else 1000.0, bottom_drag=1e-7,
                wind_amplitude=8e-5 if wall else 0.0, bc=case["bc"])


def _swm_dt(case):
    p = _swm_numbers(case)
    return float(max(1, int(0.28 * p["Lx"] / p["nx"] / math.sqrt(9.81 * sum(p["H"])))))


def _dst(n, dtype=torch.float64):
    k = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
    return (math.sqrt(2.0 / (n + 1)) * torch.sin(math.pi * torch.outer(k, k) / (n + 1))).to(dtype)


def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _eddies(seed, salt, nl, ny, nx, slope=-1.5):
    """(nl, ny + 2, nx + 2) unit-RMS fields with zero ring, random with a k^-3 power spectrum."""
    k = torch.arange(1, max(nx, ny) + 1, dtype=torch.float32, device="cuda")
    amp = (k[:ny, None] ** 2 + k[None, :nx] ** 2) ** (slope / 2)
    c = torch.randn((nl, ny, nx), generator=_generator(seed, salt), device="cuda") * amp
    f = _dst(ny, torch.float32) @ c @ _dst(nx, torch.float32)
    out = torch.zeros((nl, ny + 2, nx + 2), device="cuda")
    out[:, 1:-1, 1:-1] = f / f.square().mean(dim=(-2, -1), keepdim=True).sqrt()
    return out


def _pv(case, seed, salt=0):
    """Eddying PV with 1e-6 /s in the top layer and less in the thicker layers below."""
    nl = max(1, case["nl"])
    H = torch.tensor(STRAT[nl][0], device="cuda")
    return (1e-6 * _eddies(seed, salt, nl, case["ny"], case["nx"]) * (H[0] / H)[:, None, None]).contiguous()


def _swm_state(case, seed):
    """(h, u, v) of a spun-up basin: a jet of 0.5 m/s with eddies of 0.2 m/s and metres of height."""
    p = _swm_numbers(case)
    nl, nx, ny = case["nl"], case["nx"], case["ny"]
    e = _eddies(seed, 7, 3 * nl, ny, nx, slope=-2.5)
    H = torch.tensor(p["H"], device="cuda")[:, None, None]
    y = torch.arange(ny + 2, device="cuda") / ny - 0.5
    sign = torch.tensor([1.0, -1.0, 1.0], device="cuda")[:nl, None, None]
    jet = 0.5 * torch.exp(-0.5 * (y / 0.05) ** 2)[None, :, None] * sign
    return ((H + 0.5 * e[:nl]).contiguous(), (jet + 0.2 * e[nl:2 * nl]).contiguous(), (0.2 * e[2 * nl:]).contiguous())


def _members(case):
    """The ensemble's members: (layers, cells per side, wind stress in N/m^2)."""
    rng, out = np.random.default_rng(1000), []
    for nl, share, n in CLASSES:
        for _ in range(max(1, round(share * case["members"] / 256))):
            out.append((nl, max(8, int(round(n * case["scale"]))), float(rng.uniform(0.05, 0.12))))
    return out


def _member_case(nl, n):
    return _qg("step", n, n, nl)


def _member_numbers(nl, n, tau):
    p = _qg_numbers(_member_case(nl, n))
    p["wind_amplitude"] = tau * 2.0 * math.pi / (RHO0 * p["Ly"])
    return p


def _land(case):
    return testcases.land_mask(case["ny"], case["nx"], frac=0.15, seed=3)


# ---- what a program holds, and the call -----------------------------------------------------------
def _qg_model(case, **more):
    p = dict(_qg_numbers(case), precision=case["precision"], refine=case["refine"], **more)
    if case["precision"] != "fp32":
        p["persistent"] = False
    return (sg.BaroclinicQG if case["nl"] else sg.BarotropicQG).create(**p)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members = _members(case)
        models = [sg.BaroclinicQG.create(**_member_numbers(*m)) for m in members]
        ens = sg.QGEnsemble(models, precision="bf16x3", persistent=False)
        q = ens.pack([_pv(_member_case(nl, n), seed, k) for k, (nl, n, _) in enumerate(members)])
        return dict(case, model=ens, q=q)
    if kind.startswith("swm"):
        model = sg.MultilayerShallowWater2D.create(**_swm_numbers(case))
        h, u, v = _swm_state(case, seed)
        state = dict(case, model=model, dt=_swm_dt(case), h=h, u=u, v=v)
        if kind == "swm_gradient":
            state["target"] = _swm_state(case, seed + 500_000)[1]
        else:
            model.plan(h.device)
        return state
    if kind == "masked":
        model = _qg_model(case, mask=_land(case))
    else:
        model = _qg_model(case)
    q = _pv(case, seed)
    q = q if case["nl"] else q[0].contiguous()
    model.plan(q.device)
    state = dict(case, model=model, q=q)
    if kind == "gradient":
        state["target"] = _pv(case, seed, 99)
    return state


def run(state):
    kind, model = state["kind"], state["model"]
    if kind == "ensemble":
        return model.step(state["q"].clone(), DT, state["steps"], state["solver"])
    if kind == "swm":
        s = sg.MultilayerSW2DState(h=state["h"], u=state["u"], v=state["v"])
        y = model.integrate(s, 0.0, state["steps"] * state["dt"], state["dt"], solver=state["solver"]).ys
        return {"h": y.h, "u": y.u, "v": y.v}
    if kind == "swm_gradient":
        h, u, v = (state[k].clone().requires_grad_(True) for k in "huv")
        y = model.integrate(sg.MultilayerSW2DState(h=h, u=u, v=v), 0.0, state["steps"] * state["dt"], state["dt"],
                            solver=state["solver"], checkpoint_every=10).ys
        loss = (y.u[0] - state["target"]).square().mean()
        gh, gu, gv = torch.autograd.grad(loss, (h, u, v))
        return {"loss": loss.detach(), "h": gh, "u": gu, "v": gv}
    S = sg.BaroclinicQGState if state["nl"] else sg.BarotropicQGState
    if kind == "rhs":
        return model.vector_field(0.0, S(q=state["q"])).q
    if kind == "integrate":
        half = max(1, state["steps"] // 2)
        return model.integrate(S(q=state["q"]), 0.0, state["steps"] * DT, DT,
                               saveat=sg.SaveAt(ts=[half * DT, state["steps"] * DT])).ys.q
    if kind == "gradient":
        q = state["q"].clone().requires_grad_(True)
        tau = torch.tensor(float(_qg_numbers(state)["wind_amplitude"]), requires_grad=True)
        model.params.wind_amplitude = tau
        qT = model.integrate(S(q=q), 0.0, state["steps"] * DT, DT, solver=state["solver"]).ys.q[-1]
        loss = ((qT - state["target"]) * 1e6).square().mean()
        gq, gt = torch.autograd.grad(loss, (q, tau))
        return {"loss": loss.detach(), "q": gq, "tau": gt}
    return model.step(S(q=state["q"]), DT, state["steps"], state["solver"]).q


# ---- what a call cannot do without -----------------------------------------------------------------
STAGES = {"euler": 1, "heun": 2, "ssprk3": 3, "tsit5": 6}


def _qg_flops(cells, nx, ny, nl):
    """One tendency: two sine transforms along each axis (2.5 N log2 N each), the modal mixes, and
    the Jacobian, Laplacians, forcing and stage update (about 70 operations a cell)."""
    return cells * (2 * 2.5 * (math.log2(nx + 2) + math.log2(ny + 2)) + 4 * nl + 70)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        total, flops = 0, 0.0
        for nl, n, _ in _members(case):
            c = nl * (n + 2) ** 2
            total += c
            flops += _qg_flops(c, n, n, nl)
        return {"bytes": 8.0 * total, "flops": flops * case["steps"] * STAGES[case["solver"]]}
    nl = max(1, case["nl"])
    cells = nl * (case["nx"] + 2) * (case["ny"] + 2)
    n = case["steps"] * STAGES[case["solver"]]
    if kind == "swm":
        return {"bytes": 24.0 * cells, "flops": 110.0 * cells * n}
    if kind == "swm_gradient":  # the state and its gradient; a reverse sweep is about twice a forward one
        return {"bytes": 24.0 * cells, "flops": 330.0 * cells * n}
    flops = _qg_flops(cells, case["nx"], case["ny"], nl)
    if kind == "rhs":
        return {"bytes": 8.0 * cells, "flops": flops}
    if kind == "gradient":
        return {"bytes": 12.0 * cells, "flops": 3 * flops * n}
    return {"bytes": (12.0 if kind == "integrate" else 8.0) * cells, "flops": flops * n}


# ---- the same in 64 bits ------------------------------------------------------------------------
def _inner(a):
    return a[..., 1:-1, 1:-1]


def _pad(a):
    return torch.nn.functional.pad(a, (1, 1, 1, 1))


def _at(a, dj, di):
    ny, nx = a.shape[-2:]
    return a[..., 1 + dj:ny - 1 + dj, 1 + di:nx - 1 + di]


def _lap(a, dx, dy):
    c = _inner(a)
    return _pad((_at(a, 0, 1) - 2 * c + _at(a, 0, -1)) / dx**2 + (_at(a, 1, 0) - 2 * c + _at(a, -1, 0)) / dy**2)


def _jacobian(f, g, dx, dy):
    """The energy- and enstrophy-conserving average of the three second-order forms, f_x g_y - f_y g_x."""
    fe, fw, fn, fs = _at(f, 0, 1), _at(f, 0, -1), _at(f, 1, 0), _at(f, -1, 0)
    ge, gw, gn, gs = _at(g, 0, 1), _at(g, 0, -1), _at(g, 1, 0), _at(g, -1, 0)
    one = (fe - fw) * (gn - gs) - (fn - fs) * (ge - gw)
    two = fe * (_at(g, 1, 1) - _at(g, -1, 1)) - fw * (_at(g, 1, -1) - _at(g, -1, -1))
    two = two - fn * (_at(g, 1, 1) - _at(g, 1, -1)) + fs * (_at(g, -1, 1) - _at(g, -1, -1))
    three = gn * (_at(f, 1, 1) - _at(f, 1, -1)) - gs * (_at(f, -1, 1) - _at(f, -1, -1))
    three = three - ge * (_at(f, 1, 1) - _at(f, -1, 1)) + gw * (_at(f, 1, -1) - _at(f, -1, -1))
    return (one + two + three) / (12.0 * dx * dy)


def _edges_zeroed(q):
    return _pad(_inner(q))


class _ExactQG:
    """The layered QG tendency in float64: (..., nl, Ny, Nx) with the ring, one wind per member."""

    def __init__(self, p, mask=None, tau=None):
        nx, ny = p["nx"], p["ny"]
        self.dx, self.dy, self.p = p["Lx"] / nx, p["Ly"] / ny, p
        self.barotropic = "H" not in p
        f64 = dict(dtype=torch.float64, device="cuda")
        y = torch.arange(ny + 2, **f64) * self.dy
        self.by = (p["beta"] * (y - p["Ly"] / 2))[:, None]
        self.wind = -torch.sin(2 * math.pi * y / p["Ly"])[:, None]
        self.tau = torch.as_tensor(p["wind_amplitude"] if tau is None else tau, **f64)
        self.Sx, self.Sy = _dst(nx + 2), _dst(ny + 2)
        k = lambda n, d: (2 * torch.cos(math.pi * torch.arange(1, n + 1, **f64) / (n + 1)) - 2) / d**2  # noqa: E731
        lap = k(ny + 2, self.dy)[:, None] + k(nx + 2, self.dx)[None, :]
        if self.barotropic:
            self.L = lap
        else:
            H, g = np.asarray(p["H"], float), np.asarray(p["g_prime"], float)
            A = np.zeros((len(H), len(H)))
            for i in range(len(H)):
                A[i, i] += 1 / (H[i] * g[i])
                if i + 1 < len(H):
                    A[i, i] += 1 / (H[i] * g[i + 1])
                    A[i, i + 1] -= 1 / (H[i] * g[i + 1])
                if i:
                    A[i, i - 1] -= 1 / (H[i] * g[i])
            ev, R = np.linalg.eig(A)
            self.Cm2l = torch.tensor(R.real, **f64)
            self.Cl2m = torch.tensor(np.linalg.inv(R.real), **f64)
            self.L = lap - p["f0"] ** 2 * torch.tensor(ev.real, **f64)[:, None, None]
            self.H0 = p["H"][0]
        self.land = None
        if mask is not None:
            land = torch.tensor(np.asarray(mask) == 0, device="cuda")
            land[0], land[-1], land[:, 0], land[:, -1] = False, False, False, False
            ocean = ~land
            ocean[0], ocean[-1], ocean[:, 0], ocean[:, -1] = False, False, False, False
            near = torch.nn.functional.max_pool2d(ocean.double()[None], 3, 1, 1)[0] > 0
            self.land, self.b = land, torch.nonzero((land & near).reshape(-1))[:, 0]
            # psi of a unit source at each coastal land point, seen at all of them
            C = torch.empty((self.L.shape[0], len(self.b), len(self.b)), **f64)
            for a in range(0, len(self.b), 32):
                e = torch.zeros((min(32, len(self.b) - a), land.numel()), **f64)
                e[torch.arange(len(e)), self.b[a:a + 32]] = 1.0
                e = e.reshape(-1, 1, *land.shape)
                C[:, :, a:a + 32] = self.solve(e.expand(-1, self.L.shape[0], -1, -1)).flatten(2)[..., self.b].permute(1, 2, 0)
            self.C = C

    def solve(self, r):
        return self.Sy @ ((self.Sy @ r @ self.Sx) / self.L) @ self.Sx

    def psi(self, q):
        if self.barotropic:
            return self.solve(q)
        qm = torch.einsum("ml,...lyx->...myx", self.Cl2m, q)
        if self.land is None:
            pm = self.solve(qm)
        else:
            qm = torch.where(self.land, 0.0, qm)
            sigma = torch.linalg.solve(self.C, self.solve(qm).flatten(-2)[..., self.b])
            flat = qm.flatten(-2).clone()
            flat[..., self.b] -= sigma
            pm = self.solve(flat.reshape(qm.shape))
        psi = _edges_zeroed(torch.einsum("lm,...myx->...lyx", self.Cm2l, pm))
        return psi if self.land is None else torch.where(self.land, 0.0, psi)

    def rhs(self, q):
        p = self.p
        if self.land is not None:
            q = torch.where(self.land, 0.0, q)
        psi = self.psi(q)
        dq = -_pad(_jacobian(psi, q + self.by, self.dx, self.dy))
        lap = _lap(q, self.dx, self.dy)
        if self.land is not None:
            lap = torch.where(self.land, 0.0, lap)
        dq = dq + p["lateral_viscosity"] * lap - p["biharmonic_viscosity"] * _lap(lap, self.dx, self.dy)
        drag = -p["bottom_drag"] * _lap(psi, self.dx, self.dy)
        if self.barotropic:
            return dq + self.tau * self.wind + drag
        wind = (self.tau[..., None, None] if self.tau.dim() else self.tau) * self.wind / self.H0
        top = torch.zeros(dq.shape[-3], 1, 1, dtype=dq.dtype, device=dq.device)
        bottom = top.clone()
        top[0], bottom[-1] = 1.0, 1.0
        wind = wind.unsqueeze(-3) if wind.dim() > 2 else wind
        dq = dq + top * wind + bottom * drag
        return dq if self.land is None else torch.where(self.land, 0.0, dq)


TSIT5_A = [
    [],
    [0.161],
    [-0.008480655492356989, 0.335480655492357],
    [2.897153057105493, -6.359448489975075, 4.3622954328695815],
    [5.325864828439257, -11.748883564062828, 7.4955393428898365, -0.09249506636175525],
    [5.86145544294642, -12.92096931784711, 8.159367898576159, -0.071584973281401, -0.028269050394068383],
]
TSIT5_B = [0.09646076681806523, 0.01, 0.4798896504144996, 1.379008574103742, -3.290069515436081, 2.324710524099774]
TABLEAU = {
    "euler": ([[]], [1.0]),
    "heun": ([[], [1.0]], [0.5, 0.5]),
    "ssprk3": ([[], [1.0], [0.25, 0.25]], [1 / 6, 1 / 6, 2 / 3]),
    "tsit5": (TSIT5_A, TSIT5_B),
}


def _step(f, y, dt, solver):
    a, b = TABLEAU[solver]
    ks = []
    for row in a:
        z = [yi + dt * sum(c * k[i] for c, k in zip(row, ks)) for i, yi in enumerate(y)]
        ks.append(f(z))
    return [yi + dt * sum(c * k[i] for c, k in zip(b, ks)) for i, yi in enumerate(y)]


def _qg_steps(m, q, steps, solver):
    f = lambda y: [m.rhs(_edges_zeroed(y[0]))]  # noqa: E731
    y = [_edges_zeroed(q)]
    if m.land is not None:
        y = [torch.where(m.land, 0.0, y[0])]
    for _ in range(steps):
        y = _step(f, y, DT, solver)
    return y[0]


class _ExactSWM:
    """The layered shallow-water tendencies in float64, vector-invariant with upwind mass fluxes."""

    def __init__(self, p):
        self.p, self.dx, self.dy = p, p["Lx"] / p["nx"], p["Ly"] / p["ny"]
        f64 = dict(dtype=torch.float64, device="cuda")
        y = torch.arange(p["ny"] + 2, **f64) * self.dy
        f = p["f0"] + p["beta"] * (y - p["Ly"] / 2)
        self.fx = (0.5 * (f[1:-1] + f[2:]))[:, None]
        self.wind = (-torch.cos(2 * math.pi * y / p["Ly"]) * p["wind_amplitude"] / p["H"][0])[:, None]
        self.g = torch.tensor(p["g_prime"], **f64)[:, None, None]

    def edges(self, y):
        h, u, v = (a.clone() for a in y)
        if self.p["bc"] == "periodic":
            out = []
            for a in (h, u, v):
                a = torch.cat([a[..., -2:-1, :], a[..., 1:-1, :], a[..., 1:2, :]], -2)
                out.append(torch.cat([a[..., :, -2:-1], a[..., :, 1:-1], a[..., :, 1:2]], -1))
            return out
        zc = torch.zeros_like(u[..., :1])
        u = torch.cat([zc, u[..., 1:-2], zc, zc], -1)
        u = torch.cat([u[..., 1:2, :], u[..., 1:-1, :], u[..., -2:-1, :]], -2)
        zr = torch.zeros_like(v[..., :1, :])
        v = torch.cat([zr, v[..., 1:-2, :], zr, zr], -2)
        v = torch.cat([v[..., :, 1:2], v[..., :, 1:-1], v[..., :, -2:-1]], -1)
        h = torch.cat([h[..., 1:2, :], h[..., 1:-1, :], h[..., -2:-1, :]], -2)
        return [torch.cat([h[..., :, 1:2], h[..., :, 1:-1], h[..., :, -2:-1]], -1), u, v]

    def rhs(self, y):
        h, u, v = self.edges(y)
        p, dx, dy = self.p, self.dx, self.dy
        fx = u[..., :, :-1] * torch.where(u[..., :, :-1] > 0, h[..., :, :-1], h[..., :, 1:])
        fy = v[..., :-1, :] * torch.where(v[..., :-1, :] > 0, h[..., :-1, :], h[..., 1:, :])
        dh = _pad(-((fx[..., 1:-1, 1:] - fx[..., 1:-1, :-1]) / dx + (fy[..., 1:, 1:-1] - fy[..., :-1, 1:-1]) / dy))
        zeta = (_at(v, 0, 1) - _inner(v)) / dx - (_at(u, 1, 0) - _inner(u)) / dy
        q = _pad((zeta + self.fx) / (0.25 * (_inner(h) + _at(h, 0, 1) + _at(h, 1, 0) + _at(h, 1, 1))))
        uh = _pad(0.5 * (_inner(h) + _at(h, 0, 1)) * _inner(u))
        vh = _pad(0.5 * (_inner(h) + _at(h, 1, 0)) * _inner(v))
        ke = 0.25 * (_inner(u) ** 2 + _at(u, 0, -1) ** 2 + _inner(v) ** 2 + _at(v, -1, 0) ** 2)
        P = _pad(ke) + torch.cumsum(self.g * h, 0)
        vhu = 0.25 * (_inner(vh) + _at(vh, 0, 1) + _at(vh, -1, 0) + _at(vh, -1, 1))
        uhv = 0.25 * (_inner(uh) + _at(uh, 0, -1) + _at(uh, 1, 0) + _at(uh, 1, -1))
        du = _pad(0.5 * (_inner(q) + _at(q, -1, 0)) * vhu - (_at(P, 0, 1) - _inner(P)) / dx)
        dv = _pad(-0.5 * (_inner(q) + _at(q, 0, -1)) * uhv - (_at(P, 1, 0) - _inner(P)) / dy)
        du = du + p["lateral_viscosity"] * _lap(u, dx, dy)
        dv = dv + p["lateral_viscosity"] * _lap(v, dx, dy)
        top = torch.zeros_like(self.g)
        bottom = torch.zeros_like(self.g)
        top[0], bottom[-1] = 1.0, 1.0
        du = du + top * self.wind - p["bottom_drag"] * bottom * u
        return [dh, du, dv - p["bottom_drag"] * bottom * v]

    def run(self, y, dt, steps, solver):
        y = self.edges(y)
        for _ in range(steps):
            y = _step(self.rhs, y, dt, solver)
        return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        members, out = _members(case), []
        classes = sorted({m[:2] for m in members}, key=[m[:2] for m in members].index)
        for nl, n in classes:
            mine = [(k, m) for k, m in enumerate(members) if m[:2] == (nl, n)]
            q = torch.stack([_pv(_member_case(nl, n), seed, k) for k, _ in mine]).double()
            wind = [_member_numbers(*m)["wind_amplitude"] for _, m in mine]
            out.append(_qg_steps(_ExactQG(_member_numbers(*mine[0][1]), tau=wind), q, case["steps"], case["solver"]).reshape(-1))
        return torch.cat(out)
    if kind.startswith("swm"):
        m, y = _ExactSWM(_swm_numbers(case)), [a.double() for a in _swm_state(case, seed)]
        if kind == "swm":
            h, u, v = m.run(y, _swm_dt(case), case["steps"], case["solver"])
            return {"h": h[None], "u": u[None], "v": v[None]}
        y = [a.requires_grad_(True) for a in y]
        u = m.run(y, _swm_dt(case), case["steps"], case["solver"])[1]
        loss = (u - _swm_state(case, seed + 500_000)[1].double()).square().mean()
        gh, gu, gv = torch.autograd.grad(loss, y)
        return {"loss": loss.detach(), "h": gh, "u": gu, "v": gv}
    p = _qg_numbers(case)
    q = _pv(case, seed).double()
    q = q if case["nl"] else q[0]
    if kind == "gradient":
        q.requires_grad_(True)
        tau = torch.tensor(p["wind_amplitude"], dtype=torch.float64, device="cuda", requires_grad=True)
        qT = _qg_steps(_ExactQG(p, tau=tau), q, case["steps"], case["solver"])
        loss = ((qT - _pv(case, seed, 99).double()) * 1e6).square().mean()
        gq, gt = torch.autograd.grad(loss, (q, tau))
        return {"loss": loss.detach(), "q": gq, "tau": gt.cpu()}
    m = _ExactQG(p, mask=_land(case) if kind == "masked" else None)
    if kind == "rhs":
        return m.rhs(q)
    if kind == "integrate":
        half = max(1, case["steps"] // 2)
        first = _qg_steps(m, q, half, "tsit5")
        y = [first]
        for _ in range(case["steps"] - half):
            y = _step(lambda z: [m.rhs(_edges_zeroed(z[0]))], y, DT, "tsit5")
        return torch.stack([first, y[0]])
    return _qg_steps(m, q, case["steps"], case["solver"])
