"""The FP32 DST-I passes (even / odd folded, one tile shape per plan chosen by size) against the
float64 inversion, at sizes that select each tile shape and at its edges: axes shorter than a
tile, odd and even lengths (the middle column of an odd axis), one column or row past a tile,
and an ensemble whose members share the shape.

Tolerance: an FP32 transform of length N rounds like a sum of N / 2 products per half, at most
~sqrt(N) * 2^-24 relative in L2 for each of the four passes, and twice that for the modal mixes:
8 * sqrt(514) * 6e-8 = 1.1e-5 is the bound at the largest size here; 2e-6 is the tolerance of
the FP32 inversion elsewhere in the tests and holds for all of them."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import qg as O

pytestmark = pytest.mark.gpu

H = {1: (4000.0,), 2: (500.0, 4500.0), 3: (400.0, 1100.0, 2600.0), 5: (200.0, 356.0, 632.0, 1125.0, 2000.0)}
G = {1: (0.02,), 2: (9.81, 0.025), 3: (9.81, 0.025, 0.0125), 5: (9.81, 0.03, 0.02, 0.0125, 0.008)}


def member(nx, ny, nl):
    kw = dict(nx=nx, ny=ny, Lx=4e6, Ly=4e6 * ny / nx, H=H[nl], g_prime=G[nl])
    return sg.BaroclinicQG.create(n_layers=nl, **kw), O.baroclinic_model(**kw)


def rel(a, b):
    return float(np.linalg.norm(a.cpu().double().numpy() - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nx,ny,nl", [
    (1, 1, 1), (2, 5, 1), (13, 14, 3), (14, 13, 3), (15, 30, 2), (31, 29, 5),   # one or two 16 x 8 tiles
    (126, 127, 2), (128, 128, 3), (97, 201, 1),
    (255, 257, 3), (300, 290, 2),                                               # 32 x 24
    (509, 512, 3), (382, 384, 5),                                               # 64 x 48, 64 x 24
])
def test_fp32_passes(nx, ny, nl):
    m, o = member(nx, ny, nl)
    rng = np.random.default_rng(nx * 1000 + ny)
    q = rng.standard_normal((nl, ny + 2, nx + 2)).astype(np.float32) * np.float32(1e-6)
    psi = m._invert_pv(torch.tensor(q, device="cuda"))
    assert rel(psi, O.invert_pv(o, q.astype(np.float64))) < 2e-6


def test_fp32_passes_ensemble():
    sizes = [(40, 33, 3), (129, 64, 2), (17, 250, 1), (64, 65, 5)]
    models, oracles = zip(*(member(*s) for s in sizes))
    ens = sg.QGEnsemble(models, precision="fp32")
    rng = np.random.default_rng(5)
    qs = [rng.standard_normal((nl, ny + 2, nx + 2)).astype(np.float32) * np.float32(1e-6) for nx, ny, nl in sizes]
    psi = ens.unpack(ens.invert(ens.pack([torch.tensor(q, device="cuda") for q in qs])))
    for p, o, q in zip(psi, oracles, qs):
        assert rel(p, O.invert_pv(o, q.astype(np.float64))) < 2e-6
