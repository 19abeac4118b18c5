"""The wide output tiles of the tensor-core DST passes (176, 208 and 256 columns, 64-byte operand rows),
forced: members shorter than a tile, of exactly one tile, of one column more, of several tiles, one and
several layers, with the refined plan's accumulating last pass and without.

Each output is the sum of the same products in the same steps along k as with 144 columns, so that the two
widths' inversions agree to FP32's rounding of such a sum, sqrt(514) 2^-24 = 1.4e-6; against the float64
inversion the bounds of the narrow widths hold (3e-5 split BF16, 6e-3 TF32).  The persistent kernel takes
128-byte rows only: a plan that asks for it refuses the wide widths, as it did."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import qg as O

pytestmark = pytest.mark.gpu

H = (400.0, 1100.0, 2600.0, 900.0)
G = (9.81, 0.025, 0.0125, 0.01)


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("precision,bound", [("bf16x3", 3e-5), ("tf32", 6e-3)])
@pytest.mark.parametrize("width", [176, 208, 256])
@pytest.mark.parametrize("refine", [0, 1])
@pytest.mark.parametrize("nx,ny,nl", [(3, 5, 2), (40, 33, 3), (174, 175, 1), (206, 207, 2), (254, 255, 3), (300, 17, 4), (512, 350, 1)])
def test_forced_wide_tiles(nx, ny, nl, refine, width, precision, bound):
    o = O.baroclinic_model(nx=nx, ny=ny, Lx=4e6, Ly=4e6 * ny / nx, H=H[:nl], g_prime=G[:nl])
    spec = sg.MemberSpec(nx, ny, 4e6, 4e6 * ny / nx, o.f0, o.beta, H[:nl], G[:nl])
    q = (np.random.default_rng(nx + width).standard_normal((nl, ny + 2, nx + 2)) * 1e-6).astype(np.float32)
    psi = []
    for w in (width, 144):
        plan = sg.Plan([spec], precision, refine, persistent=False, gemm_tile=w)
        assert plan.tuning()["gemm_tile_n"] == w
        psi.append(plan.invert(torch.tensor(q, device="cuda")).cpu().double().numpy())
        assert plan.status() == 0
    assert rel(psi[0], psi[1]) < 1.4e-6
    assert rel(psi[0], O.invert_pv(o, q.astype(np.float64))) < bound


def test_a_reported_width_can_be_given_back():
    spec = sg.MemberSpec(1022, 1022, 4e6, 4e6, 9.4e-5, 1.75e-11, H, G)
    width = sg.Plan([spec], "bf16x3", 1).tuning()["gemm_tile_n"]
    assert sg.Plan([spec], "bf16x3", 1, gemm_tile=width).tuning()["gemm_tile_n"] == width


@pytest.mark.parametrize("width", [176, 208, 256, 64])
def test_the_persistent_kernel_refuses_wide_tiles(width):
    spec = sg.MemberSpec(64, 64, 4e6, 4e6, 9.4e-5, 1.75e-11, H[:1], G[:1])
    with pytest.raises(Exception):
        sg.Plan([spec], "bf16x3", gemm_tile=width)
