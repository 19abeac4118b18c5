"""The tiled adjoint of the QG right-hand side at the edges of its 32 x 4 tiles, layers 1 to 8, and in a
plan whose members differ in layers and size, against the float64 transposed Jacobian and parameter
derivatives of the oracle.  Tolerance 1e-4 relative L2, as for every FP32 adjoint of the model."""

import numpy as np
import pytest

import somax_gb300 as sg
from oracle import adjoint as OA
from oracle import qg as O

from test_gpu_adjoint import PHYS, RTOL_VJP, cuda, field, rel

pytestmark = pytest.mark.gpu

H = (400.0, 1100.0, 600.0, 900.0, 300.0, 500.0, 700.0, 800.0)
G = (9.81, 0.025, 0.0125, 0.01, 0.02, 0.015, 0.01, 0.012)
P = dict(lateral_viscosity=PHYS["nu"], bottom_drag=PHYS["kappa"], wind_amplitude=PHYS["tau"],
         biharmonic_viscosity=PHYS["nu4"])


@pytest.mark.parametrize("apply_bc", [False, True])
@pytest.mark.parametrize("sizes", [[(29, 2, 1)], [(30, 3, 2)], [(31, 6, 3)], [(62, 4, 2)], [(5, 15, 4)], [(3, 14, 8)], [(70, 9, 2)],
                                   [(30, 6, 1), (4, 9, 6), (33, 2, 3)]])
def test_rhs_vjp_at_tile_edges(sizes, apply_bc):
    os_, specs, qs, gs = [], [], [], []
    for nx, ny, nl in sizes:
        o = O.baroclinic_model(nx=nx, ny=ny, Lx=1e6, Ly=8e5, H=H[:nl], g_prime=G[:nl], **P)
        os_.append(o)
        specs.append(sg.MemberSpec(nx, ny, 1e6, 8e5, o.f0, o.beta, H[:nl], G[:nl]))
        qs.append(field((nl, ny + 2, nx + 2), nx))
        gs.append(np.random.default_rng(ny).standard_normal((nl, ny + 2, nx + 2)))
    plan = sg.Plan(specs, "fp32")
    par = cuda(np.tile(list(P.values()), len(sizes)))
    qb, pb = plan.rhs_vjp(cuda(np.concatenate([q.ravel() for q in qs])), par,
                          cuda(np.concatenate([g.ravel() for g in gs])), apply_bc)
    qb, at = qb.cpu().double().numpy(), 0
    for k, (o, q, g) in enumerate(zip(os_, qs, gs)):
        want_q, want_p = OA.rhs_vjp(o, q, g, apply_bc=apply_bc)
        assert rel(qb[at:at + q.size], want_q.ravel()) < RTOL_VJP
        got_p = pb.cpu().double().numpy().reshape(len(sizes), 4)[k]
        assert (np.abs(got_p - want_p) <= RTOL_VJP * np.abs(want_p)).all()
        at += q.size
