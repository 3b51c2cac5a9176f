"""The native Python entry points on the host's side: what they take and which Python errors they
raise.  CPU tensors go as far as the library's own checks."""
import pytest
import torch

from relax_b200 import ops


@pytest.mark.gpu
def test_out_of_memory():
    x = torch.empty(1, 64, dtype=torch.float16, device="cuda").expand(1 << 30, 64)
    w = torch.empty(1 << 20, 8, dtype=torch.int32, device="cuda")
    with pytest.raises(torch.OutOfMemoryError):
        ops.gemm_fp16_q4f16(x, w, None)
    torch.empty(16, device="cuda")
