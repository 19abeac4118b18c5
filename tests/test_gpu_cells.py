"""The kernels that walk a plan's cells without a halo (pack, unpack, Butcher combination): every layer
count, both tile shapes, cells behind the last whole tile, tiles shared by four CTAs and not.

No step of an integration is pack, boundary condition and unpack: exact.  An Euler step against the
plan's own right-hand side: the combination rounds once where the two torch operations round twice,
2^-23 relative to the larger term, 1e-6 with margin."""

import pytest
import torch

import somax_gb300 as sg

pytestmark = pytest.mark.gpu

H = (400.0, 1100.0, 600.0, 900.0, 300.0, 500.0, 700.0, 800.0)
G = (9.81, 0.025, 0.0125, 0.01, 0.02, 0.015, 0.01, 0.012)


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
@pytest.mark.parametrize("stencil", ["tile32x8", "tile64x16"])
@pytest.mark.parametrize("nx,ny,nl", [(29, 6, 1), (30, 14, 2), (31, 15, 3), (62, 17, 4), (63, 30, 5), (64, 31, 6),
                                      (65, 7, 7), (33, 9, 8), (1180, 1100, 1)])
def test_pack_combine_unpack(nx, ny, nl, stencil, precision):
    spec = sg.MemberSpec(nx, ny, 1e6, 1e6 * ny / nx, 1e-4, 1.6e-11, H[:nl], G[:nl])
    plan = sg.Plan([spec], precision, stencil=stencil, cluster=False)
    gen = torch.Generator(device="cuda").manual_seed(nx)
    q = 1e-6 * torch.randn(nl, ny + 2, nx + 2, device="cuda", generator=gen)
    params = torch.tensor([50.0, 1e-7, 1e-10, 1e9], device="cuda")
    closed = torch.zeros_like(q)
    closed[:, 1:-1, 1:-1] = q[:, 1:-1, 1:-1]
    for apply_bc, want in ((False, q), (True, closed)):
        y = q.clone()
        plan.step(y, params, 600.0, 0, "euler", apply_bc)
        assert torch.equal(y, want)
    dq = plan.rhs(closed, params, apply_bc=True)
    y = closed.clone()
    plan.step(y, params, 600.0, 1, "euler", True)
    want = closed.double() + 600.0 * dq.double()
    assert float((y.double() - want).norm() / want.norm()) < 1e-6
    assert plan.status() == 0
