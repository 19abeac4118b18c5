"""The shallow-water stage kernels that large basins run with fewer registers, against those of small
ones: on an f-plane without wind a basin whose state repeats a small basin's steps as the small basin
does, away from the small basin's edges (a stage reads two cells on each side, and the ring has no PV).

Tolerance: the two may round a stage's thickness differently, by one unit in its last place; through the
pressure gradient that is g ulp(H) dt / dx of velocity a stage."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg

pytestmark = pytest.mark.gpu

H, G, DX, DT = (400.0, 700.0), (9.81, 0.02), 1e4, 20.0


def model(nx, ny, nl):
    return sg.MultilayerShallowWater2D.create(nx=nx, ny=ny, Lx=nx * DX, Ly=ny * DX, f0=1e-4, beta=0.0, H=H[:nl],
                                              g_prime=G[:nl], n_layers=nl, lateral_viscosity=300.0, bottom_drag=1e-5,
                                              wind_amplitude=0.0, bc="periodic", engine="stages")


@pytest.mark.parametrize("solver,stages", [("heun", 2), ("ssprk3", 3), ("tsit5", 6)])
@pytest.mark.parametrize("nx,ny,nl,kx,ky", [(125, 59, 2, 8, 8), (32, 182, 1, 2, 40)])
def test_large_basin_repeats_a_small_one(nx, ny, nl, kx, ky, solver, stages):
    gen = torch.Generator(device="cuda").manual_seed(nx)
    small = 0.05 * torch.randn(3, nl, ny, nx, device="cuda", generator=gen)
    small[0] += torch.tensor(H[:nl], device="cuda").view(nl, 1, 1)
    out = []
    for m, inner in ((model(nx, ny, nl), small), (model(kx * nx, ky * ny, nl), small.repeat(1, 1, ky, kx))):
        y = torch.nn.functional.pad(inner, (1, 1, 1, 1), mode="circular").contiguous()
        plan = m.plan()
        plan.step(y.view(-1), m._param_vector("cuda"), DT, 1, solver, True)
        assert plan.status() == 0
        e = 2 * stages + 1
        inside = y[..., 1:-1, 1:-1].unflatten(3, (-1, nx)).unflatten(2, (-1, ny))
        out.append(inside[:, :, :, e:-e, :, e:-e].double())
    a, b = out
    ulp = float(np.spacing(np.float32(max(H[:nl]))))
    bound = stages * sum(G[:nl]) * ulp * DT / DX
    for f in range(3):
        rms = float(b[f].pow(2).mean().sqrt())
        assert float((a[f] - b[f]).pow(2).mean().sqrt()) < max(bound, 1e-6 * rms)
