"""The row engine of qg_step (two FP32 kernels a stage) against the float64 oracle.  A plan without
autotuning steps FP32 members with it wherever they allow it; the sizes select every number of
columns a lane takes (axes of up to 64, 128, 192, 256, 320 points and beyond), 1, 2 and 4 rows per
CTA, the matrix in one piece and in chunks, odd and even axes, axes shorter than a warp, and
several alike members in one plan.

Tolerance: 1e-5 relative L2 on the state after three steps, the bound every stepping path of the
library is held to (a tendency missing on one row of 130 shows as ~1e-4)."""

import ctypes

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import qg as O
from somax_gb300 import testcases as tc

pytestmark = pytest.mark.gpu

H = {1: (4000.0,), 2: (500.0, 4500.0), 3: (400.0, 1100.0, 2600.0), 4: (400.0, 1100.0, 2600.0, 900.0),
     5: (200.0, 356.0, 632.0, 1125.0, 2000.0)}
G = {1: (0.02,), 2: (9.81, 0.025), 3: (9.81, 0.025, 0.0125), 4: (9.81, 0.025, 0.0125, 0.01),
     5: (9.81, 0.03, 0.02, 0.0125, 0.008)}
P = dict(lateral_viscosity=50.0, bottom_drag=1e-7, wind_amplitude=1e-10, biharmonic_viscosity=1e9)


def setup(nx, ny, nl, n_members=1):
    Lx, Ly = 4e6, 4e6 * ny / nx
    if nl == 0:
        o = O.barotropic_model(nx=nx, ny=ny, Lx=Lx, Ly=Ly, **P)
        spec = sg.MemberSpec(nx, ny, Lx, Ly, o.f0, o.beta, [1.0], [1.0], True)
    else:
        o = O.baroclinic_model(nx=nx, ny=ny, Lx=Lx, Ly=Ly, H=H[nl], g_prime=G[nl], **P)
        spec = sg.MemberSpec(nx, ny, Lx, Ly, o.f0, o.beta, H[nl], G[nl])
    plan = sg.Plan([spec] * n_members, "fp32", autotune=False)
    on = ctypes.c_int(0)
    assert plan._L.qg_plan_row_engine(plan.handle, ctypes.byref(on), None) == 0 and on.value == 1
    params = torch.tensor(list(P.values()) * n_members, dtype=torch.float32, device="cuda")
    return o, plan, params


def check(nx, ny, nl, scheme, n_members=1):
    o, plan, params = setup(nx, ny, nl, n_members)
    qs = [tc.kminus3_field(max(nx, ny), 7 * k + nx, max(nl, 1))[:, :ny + 2, :nx + 2].astype(np.float32) * np.float32(1e-6)
          for k in range(n_members)]
    rng = np.random.default_rng(nx)
    for q in qs:  # a ring that the boundary conditions have to clear
        q[:, 0], q[:, :, -1] = 1e-6, 1e-6 * rng.standard_normal((max(nl, 1), ny + 2))
    y = torch.tensor(np.stack(qs), device="cuda").reshape(-1)
    plan.step(y, params, 1200.0, 3, scheme, True)
    assert plan.status() == 0
    got = y.view(n_members, max(nl, 1), ny + 2, nx + 2).cpu().double().numpy()
    for g, q in zip(got, qs):
        q = q.astype(np.float64) if nl else q[0].astype(np.float64)
        ref = O.integrate(o, q, 1200.0, 3, scheme)
        g = g if nl else g[0]
        assert np.linalg.norm(g - ref) / np.linalg.norm(ref) < 1e-5


@pytest.mark.parametrize("nx,ny,nl,scheme", [
    (3, 5, 1, "heun"), (1, 40, 2, "ssprk3"), (62, 63, 3, "tsit5"), (64, 64, 0, "heun"), (65, 30, 4, "ssprk3"),
    (126, 127, 2, "tsit5"), (128, 128, 3, "ssprk3"), (97, 190, 5, "heun"), (190, 191, 3, "ssprk3"), (250, 190, 3, "tsit5"),
    (256, 255, 1, "ssprk3"), (254, 256, 3, "heun"), (318, 140, 1, "tsit5"), (319, 321, 1, "ssprk3"), (510, 40, 2, "heun"),
    (41, 512, 3, "ssprk3"), (700, 64, 1, "ssprk3"),
])
def test_rows_against_oracle(nx, ny, nl, scheme):
    check(nx, ny, nl, scheme)


def test_rows_alike_members():
    check(40, 33, 3, "ssprk3", n_members=3)
    check(64, 66, 1, "tsit5", n_members=5)


def test_rows_nonfinite_and_chunked_calls():
    o, plan, params = setup(40, 33, 3)
    q = torch.tensor(tc.kminus3_field(40, 3, 3)[:, :35, :42] * 1e-6, dtype=torch.float32, device="cuda").reshape(-1)
    a = plan.step(q.clone(), params, 1200.0, 11, "ssprk3", True)
    b = plan.step(q.clone(), params, 1200.0, 4, "ssprk3", True)
    plan.step(b, params, 1200.0, 7, "ssprk3", False)
    assert torch.equal(a, b)
    q[500] = float("nan")
    plan.step(q, params, 1200.0, 1, "ssprk3", True)
    assert plan.status() != 0 and plan.status() == 0
