"""The engine of a plan made without the autotuner: the row engine for members few and small enough, the
FP32 passes beyond (1 x 1000 x 1000 x 3 layers steps three times as fast with them)."""

import pytest

import somax_gb300 as sg

pytestmark = pytest.mark.gpu

H, G = (400.0, 1100.0, 2600.0), (9.81, 0.025, 0.0125)


@pytest.mark.parametrize("n,layers,members,rows", [
    (128, 3, 1, True), (128, 3, 8, True), (128, 3, 32, False), (128, 1, 16, True), (64, 3, 16, False),
    (448, 3, 1, True), (512, 3, 1, False), (512, 1, 1, True), (1000, 3, 1, False),
])
def test_untuned_engine_by_size(n, layers, members, rows):
    spec = sg.MemberSpec(n, n, 4e6, 4e6, 9.4e-5, 1.75e-11, H[:layers], G[:layers])
    plan = sg.Plan([spec] * members, "fp32", autotune=False)
    assert plan.engine()["rows"] is rows
    assert plan.launches_per_call(2, "ssprk3") == (14 if rows else 32)
