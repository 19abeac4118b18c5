"""Parameter vectors that reach the device as kernel arguments: the values PyTorch's own conversion
gives, for every split of the length into launches (exact)."""

import math

import pytest
import torch

from somax_gb300.qg import _device_vector

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 3, 8, 9, 1024, 1025, 2500])
def test_device_vector(n):
    vals = [((-1) ** k) * math.exp(k % 171 - 85) for k in range(n)]
    vals[:5] = [math.inf, -0.0, 1e40, 1e-45, math.nan][:min(n, 5)]
    got = _device_vector(vals, "cuda")
    want = torch.tensor(vals, dtype=torch.float32)
    assert got.device.type == "cuda" and got.dtype == torch.float32
    assert torch.equal(got.cpu().view(torch.int32)[want == want], want.view(torch.int32)[want == want])
    assert torch.equal(got.cpu().isnan(), want.isnan())
