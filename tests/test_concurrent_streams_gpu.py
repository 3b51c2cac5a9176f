"""Matmuls whose tiles are cut over several CTAs, launched so that they overlap: on streams of their own, and
as graphs captured on one stream and replayed on two.  Every result has to be the one the call gives alone,
bit for bit: launches that may overlap share no hand-over words."""
import os
import subprocess
import sys

import pytest
import torch

from relax_b200 import ops
from tests.test_gemv_gpu import _check_status

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _calls(seed):
    """(function, output) of several forms: medium and large batches with cut tiles, and an expert layer."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def words(*shape):
        return torch.randint(-2 ** 31, 2 ** 31 - 1, shape, dtype=torch.int32, device="cuda", generator=g)

    def half(lo, hi, *shape):
        return (torch.rand(shape, device="cuda", generator=g) * (hi - lo) + lo).half()

    calls = []
    # tiles shared by a cluster (no words), cut into three, runs beside whole tiles, CTA pairs
    for m, k, n in [(24, 4096, 4096), (64, 4096, 2048), (32, 2048, 8192), (64, 1088, 31696), (128, 4096, 1536), (300, 2048, 3072)]:
        w, s = ops.preprocess_weight_q4f16(words(n, k // 8)), half(1e-3, 1e-2, n, k // 32)
        x, out = torch.randn(m, k, device="cuda", generator=g).half(), torch.empty(m, n, dtype=torch.float16, device="cuda")
        calls.append((lambda x=x, w=w, s=s, out=out: ops.gemm_fp16_q4f16(x, w, s, out=out), out))
    # the same of another decode and drain: int8, one scale per row
    w, s = ops.preprocess_weight_ft(torch.randint(-128, 128, (2048, 3072), dtype=torch.int8, device="cuda", generator=g), False), half(1e-4, 1e-3, 3072)
    x, out = torch.randn(24, 2048, device="cuda", generator=g).half(), torch.empty(24, 3072, dtype=torch.float16, device="cuda")
    calls.append((lambda x=x, w=w, s=s, out=out: ops.gemm_fp16_ft(x, w, s, 8, group_size=-1, out=out), out))
    for rows in (96, 640):
        w = ops.preprocess_weight_ft(torch.randint(-128, 128, (4, 2048, 512), dtype=torch.int8, device="cuda", generator=g), True)
        s, indptr = half(1e-3, 1e-2, 4, 1024), torch.tensor([rows // 4, rows // 2, rows // 2, rows], device="cuda")
        x, out = torch.randn(rows, 2048, device="cuda", generator=g).half(), torch.empty(rows, 1024, dtype=torch.float16, device="cuda")
        calls.append((lambda x=x, w=w, s=s, i=indptr, out=out: ops.moe_gemm_ft(x, w, s, i, out=out), out))
    return calls


def _alone(calls):
    ref = []
    for f, out in calls:
        f()
        torch.cuda.synchronize()
        ref.append(out.clone())
    return ref


def test_two_streams():
    sets = [_calls(1), _calls(2)]
    refs = [_alone(c) for c in sets]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for rep in range(20):
        for i in range(len(sets[0])):
            for j in (0, 1):
                with torch.cuda.stream(streams[j]):
                    sets[j][(i + j * rep) % len(sets[j])][0]()
        torch.cuda.synchronize()
        for c, ref in zip(sets, refs):
            for (_, out), r in zip(c, ref):
                assert torch.equal(out, r)
                out.zero_()
    _check_status()


def test_graphs_of_one_capture_stream_replayed_on_two():
    sets = [_calls(3), _calls(4)]
    refs = [_alone(c) for c in sets]
    graphs = []
    for c in sets:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for f, _ in c:
                f()
        graphs.append(graph)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for s, graph in zip(streams, graphs):
            with torch.cuda.stream(s):
                graph.replay()
    torch.cuda.synchronize()
    _check_status()
    for c, ref in zip(sets, refs):
        for (_, out), r in zip(c, ref):
            assert torch.equal(out, r)


def test_graphs_give_their_words_back():
    calls = _calls(5)
    ref = _alone(calls)

    def one_graph():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for f, _ in calls:
                f()
        graph.replay()
        torch.cuda.synchronize()
        for (_, out), r in zip(calls, ref):
            assert torch.equal(out, r)

    one_graph()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(24):
        one_graph()
    assert free - torch.cuda.mem_get_info()[0] < 200 << 20  # 24 areas would be 460 MB


CHILD = """
import torch
from cuda.bindings import runtime
from relax_b200 import ops
from tests.test_concurrent_streams_gpu import _alone, _calls
calls = _calls(6)
ref = _alone(calls)
for i in range(40):
    err, s = runtime.cudaStreamCreateWithFlags(1)
    assert int(err) == 0
    stream = torch.cuda.ExternalStream(int(s))
    for (f, out), r in zip(calls, ref):
        with torch.cuda.stream(stream):
            out.zero_()
            f()
        stream.synchronize()
        if i < 24:
            assert torch.equal(out, r)
        else:  # the same sums in another order
            d = (out.float() - r.float()).norm() / r.float().norm()
            assert d < 1e-3, (i, d)
print("fine")
"""


def test_more_streams_than_areas():
    """Past the bound a launch computes whole tiles.  In a process of its own: streams keep their areas."""
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stdout + r.stderr
