"""The wide output tiles of the tensor-core DST passes (64-byte operand rows, rings of four and five
stages): basins whose passes fit one wave of 176, 208 or 256 columns, so that the width is one of those
the plan times and keeps; the refined plan's last pass adds to psi (loads in batches of sixteen).

Tolerance: 3e-5 relative L2 against the float64 oracle, as for the other widths (split BF16 products keep
16 bits a factor); an element added wrongly by the refined plan's last pass is off by its own size."""

import numpy as np
import pytest
import torch

import somax_gb300 as sg
from oracle import qg as O
from somax_gb300 import testcases as tc

pytestmark = pytest.mark.gpu

H = (400.0, 1100.0, 2600.0, 900.0)
G = (9.81, 0.025, 0.0125, 0.01)


@pytest.mark.parametrize("refine", [0, 1])
@pytest.mark.parametrize("n,nl,width", [(1024, 3, 176), (934, 4, 208), (1022, 4, 256)])
def test_wide_tiles(n, nl, width, refine):
    o = O.baroclinic_model(nx=n, ny=n, Lx=4e6, Ly=4e6, H=H[:nl], g_prime=G[:nl])
    spec = sg.MemberSpec(n, n, 4e6, 4e6, o.f0, o.beta, H[:nl], G[:nl])
    plan = sg.Plan([spec], "bf16x3", refine, persistent=False)
    assert plan.tuning()["gemm_ms"][width] > 0
    q = (tc.kminus3_field(n, n, nl) * 1e-6).astype(np.float32)
    psi = plan.invert(torch.tensor(q, device="cuda"))
    ref = O.invert_pv(o, q.astype(np.float64))
    assert np.linalg.norm(psi.cpu().double().numpy() - ref) / np.linalg.norm(ref) < 3e-5
    assert plan.status() == 0
