"""The adjoint of a plan whose members differ in layers: its stencil runs once per layer count, side by
side or one after another, over tiles that lie scattered in the plan's order.  Against the float64
transposed Jacobian of the oracle (1e-4 relative L2, as for every FP32 adjoint); the two ways of launching
and a captured step's replay give the same bits.  Against a plan of the member alone: the FP32 passes add
up a row's products in the same order whatever their tiles, so that the cotangents of q are the same bits,
and the parameters' FP64 sums round to the same FP32 number or its neighbour (2^-23)."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import adjoint as OA
from oracle import qg as O

from test_gpu_adjoint import RTOL_VJP, cuda, field, rel
from test_gpu_vjp_tiles import G, H, P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [(30, 6, 3), (4, 9, 1), (33, 2, 5), (70, 9, 1), (12, 40, 3)],
    [(9, 7, n) for n in (8, 1, 7, 2, 6, 3, 5, 4)],
])
def test_members_of_mixed_layer_counts(sizes):
    os_ = [O.baroclinic_model(nx=nx, ny=ny, Lx=1e6, Ly=8e5, H=H[:nl], g_prime=G[:nl], **P) for nx, ny, nl in sizes]
    plan = sg.Plan([sg.MemberSpec(nx, ny, 1e6, 8e5, o.f0, o.beta, H[:nl], G[:nl]) for o, (nx, ny, nl) in zip(os_, sizes)],
                   "fp32")
    qs = [field((nl, ny + 2, nx + 2), nx) for nx, ny, nl in sizes]
    gs = [np.random.default_rng(ny).standard_normal(q.shape) for q, (_, ny, _) in zip(qs, sizes)]
    q, g = (cuda(np.concatenate([x.ravel() for x in xs])) for xs in (qs, gs))
    par = cuda(np.tile(list(P.values()), len(sizes)))
    qb, pb = plan.rhs_vjp(q, par, g, True)
    step = plan.step_vjp(q, par, 600.0, "ssprk3", g)[0]
    assert torch.equal(step, plan.step_vjp(q, par, 600.0, "ssprk3", g)[0])
    plan.set_parallel_sweep(False)
    assert torch.equal(qb, plan.rhs_vjp(q, par, g, True)[0])
    assert torch.equal(step, plan.step_vjp(q, par, 600.0, "ssprk3", g)[0])
    at = 0
    for k, (o, x, y) in enumerate(zip(os_, qs, gs)):
        mine = qb[at:at + x.size]
        assert rel(mine, OA.rhs_vjp(o, x, y, apply_bc=True)[0].ravel()) < RTOL_VJP
        alone_q, alone_p = sg.Plan([plan.members[k]], "fp32").rhs_vjp(cuda(x.ravel()), par[:4], cuda(y.ravel()), True)
        assert torch.equal(mine, alone_q)
        assert bool(((pb.view(-1, 4)[k] - alone_p).abs() <= 2.0**-23 * alone_p.abs()).all())
        at += x.size
