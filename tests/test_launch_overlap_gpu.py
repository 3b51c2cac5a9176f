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


def _words(g, *shape):
    return torch.from_numpy(g.integers(-2 ** 31, 2 ** 31, size=shape, dtype=np.int64).astype(np.int32)).cuda()


def _halves(g, shape, lo, hi):
    return to_dev(g.uniform(lo, hi, size=shape).astype(np.float16))


def _loop(passes, calls, reps=20):
    """Every pass alone, with a wait after each of its calls; then, overlap on, the passes in turn without any, each
    taking the blocks the one before has given back.  Same bits."""
    def sync():
        torch.cuda.synchronize()
    ref = [calls(p, sync).clone() for p in passes]
    outs = [torch.zeros_like(r) for r in ref]
    torch.cuda.synchronize()
    before = relax_b200.get_launch_overlap()
    relax_b200.set_launch_overlap(True)
    try:
        for _ in range(reps):
            for p, o in zip(passes, outs):
                o.copy_(calls(p, lambda: None))
        torch.cuda.synchronize()
        _check_status()
    finally:
        relax_b200.set_launch_overlap(before)
    for o, r in zip(outs, ref):
        assert torch.equal(o.view(torch.int16), r.view(torch.int16))


@pytest.mark.parametrize("source", ["zeros_last", "repack_last", "quantise"])
@pytest.mark.parametrize("m", [48, 160])
def test_batches_above_32_rows_read_what_was_prepared_just_before(m, source):
    """AutoGPTQ zero points, repacked weights, quantised weights and scales, each by the kernel directly ahead."""
    g = np.random.Generator(np.random.PCG64(m))
    k, n = 4096, 2048
    x = to_dev(g.standard_normal((m, k), dtype=np.float32).astype(np.float16))
    if source == "quantise":
        passes = [to_dev((g.standard_normal((n, k), dtype=np.float32) * s).astype(np.float16)) for s in (0.01, 0.05)]

        def calls(w, then):
            packed, scales = ops.encode_ft(w, 4)
            then()
            pre = ops.preprocess_weight_ft(packed, True)
            then()
            return ops.gemm_fp16_ft(x, pre, scales, 4)
    else:
        passes = [(_words(g, k // 8, n), _words(g, k // 128, n // 8), _halves(g, (k // 128, n), 0.001, 0.01)) for _ in range(2)]

        def calls(p, then):
            if source == "zeros_last":
                pre = ops.preprocess_weight_autogptq(p[0])
                then()
                zeros = ops.unpack_zeros_autogptq(p[1])
            else:
                zeros = ops.unpack_zeros_autogptq(p[1])
                then()
                pre = ops.preprocess_weight_autogptq(p[0])
            then()
            return ops.gemm_fp16_autogptq(x, pre, p[2], zeros)
    _loop(passes, calls)


@pytest.mark.parametrize("m", [4, 16])
def test_gather_between_the_writer_of_weights_and_a_decode_matmul(m):
    """Act-order: repack, zero points, then one call that gathers x and multiplies.  The matmul reads weights ahead of
    its wait, and the gather lets it start early, but not before the kernels ahead of the gather have ended."""
    g = np.random.Generator(np.random.PCG64(60 + m))
    k, n = 4096, 2048
    perms = [torch.from_numpy(g.permutation(k).astype(np.int32)).cuda() for _ in range(2)]
    passes = [(_words(g, k // 8, n), _words(g, k // 128, n // 8), _halves(g, (k // 128, n), 0.001, 0.01), perms[i],
               to_dev(g.standard_normal((m, k), dtype=np.float32).astype(np.float16))) for i in range(2)]

    def calls(p, then):
        pre = ops.preprocess_weight_autogptq(p[0])
        then()
        zeros = ops.unpack_zeros_autogptq(p[1])
        then()
        return ops.gemm_fp16_autogptq(p[4], pre, p[2], zeros, perm=p[3])
    _loop(passes, calls)


@pytest.mark.parametrize("tokens", [2, 8, 100])
@pytest.mark.parametrize("prepare", [False, True])
def test_expert_layer(tokens, prepare):
    """Route, gather, two grouped matmuls, combine, with resident weights or directly behind their repack; then the
    layer from a graph, whose rows move from expert to expert between replays."""
    g = np.random.Generator(np.random.PCG64(tokens))
    h, f, e, top_k = 1024, 1536, 8, 2
    raw = [[to_dev(g.integers(-128, 128, size=(e, k, n // 2), dtype=np.int8)) for k, n in ((h, f), (f, h))] for _ in range(2)]
    scales = [_halves(g, (e, h // 128, f), 0.001, 0.01), _halves(g, (e, f // 128, h), 0.0001, 0.001)]
    resident = [[ops.preprocess_weight_ft(w, True) for w in r] for r in raw]
    passes = [(i, to_dev(g.standard_normal((tokens, h), dtype=np.float32).astype(np.float16)),
               to_dev(g.standard_normal((tokens, e), dtype=np.float32))) for i in range(2)]

    def calls(p, then):
        i, x, logits = p
        w1, w2 = [ops.preprocess_weight_ft(w, True) for w in raw[i]] if prepare else resident[i]
        then()
        indptr, token_of_row, gate_of_row, row_of_flat = ops.moe_route(logits, top_k)
        then()
        xg = ops.moe_gather(x, token_of_row)
        then()
        y = ops.moe_gemm_ft(xg, w1, scales[0], indptr)
        then()
        y = ops.moe_gemm_ft(y, w2, scales[1], indptr)
        then()
        return ops.moe_combine(y, row_of_flat, gate_of_row, top_k)
    _loop(passes, calls)
    if prepare:
        return
    ref = [calls(p, torch.cuda.synchronize).clone() for p in passes]
    x, logits = torch.empty_like(passes[0][1]), torch.empty_like(passes[0][2])
    relax_b200.set_launch_overlap(True)
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = calls((0, x, logits), lambda: None)
        resident_ref = calls((0,) + passes[1][1:], torch.cuda.synchronize).clone()
        for _ in range(10):
            for p, want in ((passes[0], ref[0]), (passes[1], resident_ref)):
                x.copy_(p[1])
                logits.copy_(p[2])
                graph.replay()
                assert torch.equal(out.view(torch.int16), want.view(torch.int16))
        _check_status()
    finally:
        relax_b200.set_launch_overlap(False)
