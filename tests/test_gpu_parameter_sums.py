"""Parameter cotangents are sums in FP64 of products over the basin.  The products need not be of the size
of the two operands' largest values: here PV and cotangent are largest in different cells of a row, and
the only products that do not vanish are 2^-140 of that bound.

With dx = dy = 1, q at the cell A and a cotangent g there that is zero elsewhere, the second difference of
q at A is -4 q and q at its four neighbours, so that the cotangents of the two viscosities are
-4 g q and -(16 + 4) g q: sums of exact products.  Tolerance: one rounding of the result to FP32, 2^-24."""

import pytest
import torch

import somax_gb300 as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("j,i,far", [(20, 4, 20), (33, 40, 55), (1, 1, 25), (64, 64, 40)])
@pytest.mark.parametrize("layers", [1, 3])
def test_products_far_below_the_largest_operands(layers, j, i, far):
    n = 64
    H = (400.0, 1100.0, 2600.0)[:layers]
    spec = sg.MemberSpec(n, n, float(n), float(n), 0.0, 0.0, H, (9.81, 0.025, 0.0125)[:layers])
    plan = sg.Plan([spec], "fp32", persistent=False)
    q = torch.zeros(layers, n + 2, n + 2, device="cuda")
    g = torch.zeros_like(q)
    q[0, j, i], q[0, j, far] = 1.2345 * 2.0**-100, 1.1 * 2.0**40
    g[0, j, i] = 1.37 * 2.0**40
    bar = plan.rhs_vjp(q.reshape(-1), torch.zeros(4, device="cuda"), g.reshape(-1))[1].double()
    gq = float(g[0, j, i].double() * q[0, j, i].double())
    ring = (j in (1, n)) + (i in (1, n))  # neighbours on the ring have no Laplacian of the cotangent
    assert abs(float(bar[0]) / (-4 * gq) - 1) <= 2.0**-24
    assert abs(float(bar[3]) / (-(20 - ring) * gq) - 1) <= 2.0**-24
