"""Every tile shape of the FP32 DST passes, by the sizes that choose it (the plan reports which), against
the float64 inversion: odd and even axes, remainders of rows and columns.

Tolerance: four passes, each rounding like a sum of N products at sqrt(N) 2^-24 relative in L2, and as much
again for the modal mixes: 8 sqrt(N) 2^-24, N the longer axis."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import qg as O

from test_gpu_fp32_passes import member, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nl,tile", [
    (510, 511, 3, (64, 96)), (382, 384, 5, (64, 96)),
    (350, 351, 3, (64, 48)), (700, 97, 5, (64, 48)), (333, 301, 3, (64, 48)), (500, 700, 5, (64, 48)),
    (300, 290, 2, (32, 48)), (255, 257, 3, (32, 48)),
    (128, 127, 3, (16, 16)), (1, 2, 1, (16, 16)),
])
def test_tile_shape(nx, ny, nl, tile):
    m, o = member(nx, ny, nl)
    plan = sg.Plan([m.spec], "fp32", persistent=False)
    t = plan.tuning()
    assert (t["gemm_tile_rows"], t["gemm_tile_n"]) == tile
    q = (np.random.default_rng(nx * 1000 + ny).standard_normal((nl, ny + 2, nx + 2)) * 1e-6).astype(np.float32)
    psi = plan.invert(torch.tensor(q, device="cuda"))
    assert rel(psi, O.invert_pv(o, q.astype(np.float64))) < 8 * (max(nx, ny) + 2) ** 0.5 * 2.0**-24


def test_tensor_core_tile_is_128_rows():
    m, _ = member(64, 64, 1)
    t = sg.Plan([m.spec], "bf16x3", gemm_tile=48).tuning()
    assert (t["gemm_tile_rows"], t["gemm_tile_n"]) == (128, 48)
