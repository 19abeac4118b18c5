"""The capacitance correction at the edges of its rows per CTA (8) and of the reads a lane holds in
flight (512 columns): basins whose land is n single cells, so that n is the number of boundary points,
against the oracle's direct sparse solve.  Tolerance 1e-4 relative L2, as for every masked inversion (the
FP32 solve's error passes through the correction)."""

import numpy as np
import pytest
import torch

from oracle import masked as OM

from test_gpu_masked import RTOL_MASK, cuda, field, pair, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,refine", [("fp32", 0), ("fp32", 1), ("bf16x3", 1), ("tf32", 1)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 511, 512, 513, 700])
def test_boundary_points(n, precision, refine):
    nx, ny, nl = 62, 50, 2
    mask = np.ones((ny + 2, nx + 2), dtype=bool)
    cells = [(2 * a + 2, 2 * b + 2) for a in range(24) for b in range(30)][:n]
    for j, i in cells:
        mask[j, i] = False
    m, o = pair(nx, ny, nl, mask, precision, refine=refine)
    q = field((nl, ny + 2, nx + 2), n)
    psi = m._invert_pv(cuda(q))
    assert rel(psi, OM.invert_pv(o, q, mask)) < RTOL_MASK
    assert torch.all(psi[:, torch.as_tensor(OM.land(mask))] == 0)
