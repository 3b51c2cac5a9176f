"""The library's scratch is filled before the first launch that reads it, whatever streams are busy: a first
call on a side stream (torch's do not wait for the default stream) while the default stream is held for a
while.  A fresh process each time, since the scratch is made once."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import torch
from relax_b200 import ops
m, k, n = %d, %d, %d
g = torch.Generator(device="cuda")
g.manual_seed(3)
w = ops.preprocess_weight_q4f16(torch.randint(-2 ** 31, 2 ** 31 - 1, (n, k // 8), dtype=torch.int32, device="cuda", generator=g))
s = (torch.rand(n, k // 32, device="cuda", generator=g) * 0.01).half()
x = torch.randn(m, k, device="cuda", generator=g).half()
first = torch.empty(m, n, dtype=torch.float16, device="cuda")
side = torch.cuda.Stream()
torch.cuda.synchronize()
torch.cuda._sleep(int(2e8))  # about a tenth of a second of the default stream
with torch.cuda.stream(side):
    ops.gemm_fp16_q4f16(x, w, s, out=first)
side.synchronize()
held = not torch.cuda.default_stream().query()
torch.cuda.synchronize()
second = ops.gemm_fp16_q4f16(x, w, s)
assert torch.equal(first, second), (first.float() - second.float()).abs().max()
print("held" if held else "not held")
"""


# (32 rows of 4096 x 4096 are added up in clusters, without scratch; the others go through it: cut tiles, runs beside whole tiles, pairs)
@pytest.mark.parametrize("m,k,n", [(32, 4096, 4096), (32, 2048, 8192), (64, 1088, 31696), (128, 4096, 4096)])
def test_first_call_beside_a_busy_default_stream(m, k, n):
    r = subprocess.run([sys.executable, "-c", CHILD % (m, k, n)], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))  # loading a kernel waits for the device
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "held", "the default stream was over too early to show anything"
