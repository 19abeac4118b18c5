"""The tiled adjoint of the shallow-water right-hand side at the edges of its 32 x 4 tiles (rings that
end on, before and behind a tile's edge, layers 1 to 4), against the float64 transposed Jacobian of
the oracle; and a segment's adjoint, with the stage inputs of all steps kept and, beyond 1 GiB of
them, recomputed, against its steps' adjoints one after the other.

Tolerances: 2e-4 relative L2 and 1e-4 for the parameters as for every FP32 adjoint of the model
(sums of up to ~40 terms per entry); the segment runs the same kernels on the same values, its
parameter sums differ by the order of FP64 additions and one FP32 rounding a step: 1e-6."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import swm as W

from test_gpu_swm_adjoint import cuda, pair, rel, state

pytestmark = pytest.mark.gpu

H = (300.0, 500.0, 700.0, 900.0)
G = (9.81, 0.03, 0.02, 0.01)


@pytest.mark.parametrize("bc", ["periodic", "wall"])
@pytest.mark.parametrize("nx,ny,nl", [(29, 2, 1), (30, 3, 2), (31, 2, 3), (32, 6, 1), (33, 7, 2), (3, 5, 4)])
def test_rhs_vjp_at_tile_edges(nx, ny, nl, bc):
    m, o = pair(nx, ny, H[:nl], G[:nl], bc)
    y = state(o, nx + 10 * ny)
    g = np.random.default_rng(nl).standard_normal(y.size)
    yb, pb = m.plan().rhs_vjp(cuda(y), m._param_vector("cuda"), cuda(g), True)
    J = W.rhs_jacobian(o, y)
    P = W.rhs_param_derivatives(o, y) @ g
    assert rel(yb.cpu().double().numpy(), J.T @ g) < 2e-4
    assert (np.abs(pb.cpu().double().numpy() - P) <= 1e-4 * np.maximum(np.abs(P), 1e-30)).all()


@pytest.mark.parametrize("nx,ny,nl,k", [(40, 21, 2, 3), (1000, 700, 3, 9)])
def test_segment_is_its_steps(nx, ny, nl, k):
    kw = dict(nx=nx, ny=ny, Lx=nx * 1e5, Ly=ny * 1e5, f0=1e-4, beta=1.6e-11, H=H[:nl], g_prime=G[:nl],
              lateral_viscosity=300.0, bottom_drag=1e-5, wind_amplitude=2e-3, bc="wall")
    m = sg.MultilayerShallowWater2D.create(n_layers=nl, **kw)
    gen = torch.Generator(device="cuda").manual_seed(nx)
    y = torch.randn(3, nl, ny + 2, nx + 2, device="cuda", generator=gen) * torch.tensor(
        [1.0, 0.05, 0.05], device="cuda").view(3, 1, 1, 1)
    y += torch.cat([torch.tensor(H[:nl]), torch.full((nl,), 0.3), torch.full((nl,), -0.2)]).cuda().view(3, nl, 1, 1)
    y = y.reshape(-1)
    g = torch.randn(y.shape, device="cuda", generator=gen)
    plan, par, dt = m.plan(), m._param_vector("cuda"), 60.0
    sb, sp = plan.segment_vjp(y, par, dt, k, "tsit5", g)
    states = [y]
    for _ in range(k - 1):
        states.append(plan.step(states[-1].clone(), par, dt, 1, "tsit5", False))
    ps = torch.zeros(3, dtype=torch.float64, device="cuda")
    for x in reversed(states):
        g, p = plan.step_vjp(x, par, dt, "tsit5", g)
        g = g.clone()
        ps += p
    assert float((sb - g).norm() / g.norm()) < 1e-6
    assert float(((sp - ps).abs() / ps.abs()).max()) < 1e-6
