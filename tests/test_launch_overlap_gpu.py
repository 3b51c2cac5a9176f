"""Launch overlap (programmatic dependent launch) keeps results identical: a chain of dependent
decode matmuls - each consumes the previous one's output - gives bit-identical results with the
switch on and off, eagerly and from a CUDA graph."""
import numpy as np
import pytest
import torch

import relax_b200
from relax_b200 import ops, synth
from tests.test_gemv_gpu import _check_status
from tests.util import to_dev, u32_to_dev

pytestmark = pytest.mark.gpu


def _chain(layers, x):
    for pre, sc in layers:
        x = ops.gemm_fp16_q4f16(x, pre, sc)
    return x


@pytest.mark.parametrize("m", [1, 8, 32])
def test_dependent_chain_is_bit_identical(m):
    g = np.random.Generator(np.random.PCG64(m))
    dims = [(1024, 4096), (4096, 8192), (8192, 1024), (1024, 4096), (4096, 1024)]  # (k, n): both decode kernels
    layers = []
    for k, n in dims:
        c = synth.q4_case(g, 1, k, n, 32)
        layers.append((ops.preprocess_weight_q4f16(u32_to_dev(c.w)), to_dev(c.scales)))
    x = to_dev(g.standard_normal((m, dims[0][0]), dtype=np.float32).astype(np.float16))
    torch.cuda.synchronize()
    assert not relax_b200.get_launch_overlap()
    ref = _chain(layers, x).clone()
    torch.cuda.synchronize()
    relax_b200.set_launch_overlap(True)
    try:
        for _ in range(5):
            got = _chain(layers, x)
        torch.cuda.synchronize()
        _check_status()
        assert torch.equal(got, ref)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _chain(layers, x)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        _check_status()
        assert torch.equal(out, ref)
    finally:
        relax_b200.set_launch_overlap(False)


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("m", [1, 8, 16, 24])
def test_buffers_written_while_a_later_launch_is_resident(m, overlap):
    """Two buffers in turn, small grids: launch i reads the one that launch i - 1 wrote and launch i - 2 read,
    and may be resident since before that write."""
    g = np.random.Generator(np.random.PCG64(50 + m))
    k = n = 512
    layers = []
    for i in range(24):
        c = synth.q4_case(g, 1, k, n, (32, 128, 512)[i % 3])
        scales = (c.scales * 0.72).astype(np.float16)  # results keep the size of their inputs
        layers.append((ops.preprocess_weight_q4f16(u32_to_dev(c.w)), to_dev(scales), c.group))
    x = to_dev(g.standard_normal((m, k), dtype=np.float32).astype(np.float16))
    ref = [x]
    for pre, sc, group in layers:
        ref.append(ops.gemm_fp16_q4f16(ref[-1], pre, sc, group_size=group))
        torch.cuda.synchronize()
    assert torch.isfinite(ref[-1]).all() and ref[-1].abs().max() > 0
    bufs = [x.clone(), torch.empty_like(x)]

    def chain():
        bufs[0].copy_(x)
        for i, (pre, sc, group) in enumerate(layers):
            ops.gemm_fp16_q4f16(bufs[i % 2], pre, sc, group_size=group, out=bufs[(i + 1) % 2])

    before = relax_b200.get_launch_overlap()
    relax_b200.set_launch_overlap(overlap)
    try:
        for _ in range(3):
            chain()
        torch.cuda.synchronize()
        assert torch.equal(bufs[0], ref[-1]) and torch.equal(bufs[1], ref[-2])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain()
        for _ in range(20):
            graph.replay()
        torch.cuda.synchronize()
        _check_status()
        assert torch.equal(bufs[0], ref[-1]) and torch.equal(bufs[1], ref[-2])
    finally:
        relax_b200.set_launch_overlap(before)


@pytest.mark.parametrize("m", [48, 160])
def test_prefill_reads_weights_written_just_before(m):
    """With overlap on, a batch above 32 rows is still ordered behind the kernel that writes its weights."""
    g = np.random.Generator(np.random.PCG64(m))
    k, n = 4096, 4096
    cases = [synth.q4_case(g, 1, k, n, 32) for _ in range(2)]
    src = [u32_to_dev(c.w) for c in cases]
    scales = [to_dev(c.scales) for c in cases]
    x = to_dev(g.standard_normal((m, k), dtype=np.float32).astype(np.float16))
    ref = [ops.gemm_fp16_q4f16(x, ops.preprocess_weight_q4f16(w), s).clone() for w, s in zip(src, scales)]
    sc = torch.empty_like(scales[0])
    outs = [torch.empty_like(r) for r in ref]
    torch.cuda.synchronize()
    relax_b200.set_launch_overlap(True)
    try:
        for rep in range(20):
            for i in (0, 1):
                sc.copy_(scales[i])
                pre = ops.preprocess_weight_q4f16(src[i])  # the block the call before last gave back
                ops.gemm_fp16_q4f16(x, pre, sc, out=outs[i])
                del pre
        torch.cuda.synchronize()
        _check_status()
    finally:
        relax_b200.set_launch_overlap(False)
    for o, r in zip(outs, ref):
        assert torch.equal(o, r)
