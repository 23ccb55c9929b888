"""GPU: the elementwise kernels of the glue at the edges of their vectors and chunks."""
import pytest
import torch

from ternainfer_b200.linear import to_float

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1023, 4096, 4099, 148 * 8 * 4096 + 5])
def test_bf16_to_fp32(lib, n):
    x = torch.randn(n, device="cuda").to(torch.bfloat16)
    y = to_float(x)
    assert y.dtype == torch.float32 and torch.equal(y, x.float())
