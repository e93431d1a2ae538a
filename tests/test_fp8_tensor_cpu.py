"""An FP8 payload without a kernel for it (host memory, another scale type) is dequantised by tensor operations."""
import pytest
import torch

from surogate_b200.runtime.ops_cuda import Fp8Tensor


@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("scale", [torch.tensor([0.5]), torch.tensor(0.5), torch.tensor([0.5], dtype=torch.bfloat16), torch.tensor([0.5], dtype=torch.float64)])
def test_host_payloads(dtype, scale):
    data = (torch.randn(4, 16) * 8).to(dtype)
    assert torch.equal(Fp8Tensor(data, scale).dequantize(), (data.float() * scale).to(torch.bfloat16))
