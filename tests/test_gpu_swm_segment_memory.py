"""The memory of the shallow-water segment adjoint: one set of buffers for every segment length of a plan,
as large as the largest needs; a limit on the stage inputs it keeps, and a plan that keeps none where the
device cannot hold them.  Keeping or running the stages again gives the same bits of the state's cotangent;
the parameters' FP64 sums are atomic and round to the same FP32 number or its neighbour."""

import pytest
import torch

import somax_gb300 as sg
from somax_gb300 import swm

pytestmark = pytest.mark.gpu


def setup():
    m = sg.MultilayerShallowWater2D.create(nx=40, ny=33, Lx=4e5, Ly=3.3e5, H=(400.0, 700.0), g_prime=(9.81, 0.02), n_layers=2,
                                           lateral_viscosity=300.0, bottom_drag=1e-5, wind_amplitude=8e-5, bc="wall")
    gen = torch.Generator(device="cuda").manual_seed(3)
    y = 0.05 * torch.randn(3, 2, 35, 42, device="cuda", generator=gen)
    y[0] += torch.tensor((400.0, 700.0), device="cuda").view(2, 1, 1)
    return m, m.plan(), m._param_vector("cuda"), y.reshape(-1).contiguous(), torch.randn(y.numel(), device="cuda", generator=gen)


def same(a, b):
    assert torch.equal(a[0], b[0])
    assert bool(((a[1] - b[1]).abs() <= 2.0**-23 * b[1].abs()).all())


def test_segment_lengths_share_their_buffers():
    lengths = (5, 9, 2, 7, 1, 8)
    _, plan, prm, y, g = setup()
    first = {}
    for k in lengths:  # a plan for each length
        m = setup()
        first[k] = m[1].segment_vjp(y, prm, 20.0, k, "tsit5", g)
    plan.segment_vjp(y, prm, 20.0, 9, "tsit5", g)
    before = torch.cuda.memory_allocated()
    for k in lengths:
        same(plan.segment_vjp(y, prm, 20.0, k, "tsit5", g), first[k])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        same(plan.segment_vjp(y, prm, 20.0, 12, "tsit5", g), setup()[1].segment_vjp(y, prm, 20.0, 12, "tsit5", g))
    torch.cuda.current_stream().wait_stream(side)
    same(plan.segment_vjp(y, prm, 20.0, 7, "ssprk3", g), setup()[1].segment_vjp(y, prm, 20.0, 7, "ssprk3", g))
    grown = 4 * 3 * 6 * y.numel() + 64 * 1024  # three more steps kept (five inputs and a state each)
    assert torch.cuda.memory_allocated() - before <= grown


def test_limit_on_kept_inputs():
    _, plan, prm, y, g = setup()
    kept = plan.segment_vjp(y, prm, 20.0, 6, "tsit5", g)
    size = plan._L.qg_swm_segment_vjp_workspace(plan._h, 3, 6)
    plan.set_kept_inputs(0)
    assert plan._L.qg_swm_segment_vjp_workspace(plan._h, 3, 6) == size - 5 * 5 * y.numel()
    same(plan.segment_vjp(y, prm, 20.0, 6, "tsit5", g), kept)
    plan.set_kept_inputs(4 * 5 * 6 * y.numel())  # just enough
    assert plan._L.qg_swm_segment_vjp_workspace(plan._h, 3, 6) == size
    same(plan.segment_vjp(y, prm, 20.0, 6, "tsit5", g), kept)


def test_out_of_memory_keeps_no_inputs(monkeypatch):
    _, plan, prm, y, g = setup()
    want = setup()[1].segment_vjp(y, prm, 20.0, 6, "tsit5", g)
    size, empty = plan._L.qg_swm_segment_vjp_workspace(plan._h, 3, 6), torch.empty

    def refuse(n, *a, **k):
        if n == size:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(n, *a, **k)

    monkeypatch.setattr(swm.torch, "empty", refuse)
    same(plan.segment_vjp(y, prm, 20.0, 6, "tsit5", g), want)
    assert plan._L.qg_swm_segment_vjp_workspace(plan._h, 3, 6) < size
