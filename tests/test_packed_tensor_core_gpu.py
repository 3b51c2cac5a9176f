"""The tensor-core kernels over packed weights (17 to 64 rows: one CTA per tile; above: CTA pairs) where
their tiles and splits can go wrong: rows around 32-row steps, tile widths and the border between the two
kernels, row counts that are no multiple of a 128- or 256-row tile, an odd number of 64-k blocks and a last
chunk of two, every scale source and zero-point form, and experts with more rows than a tile.  Each launch is repeated into a
new output and has to repeat itself bit for bit: the hand-over words are back at rest."""
import numpy as np
import pytest
import torch

from relax_b200 import ops, synth
from tests.test_autogptq_gpu import _case as gptq_case
from tests.test_gemv_gpu import _check_status
from tests.util import assert_close, bits16, to_dev, u32_to_dev

pytestmark = pytest.mark.gpu


def _twice(run):
    a, b = run(), run()
    _check_status()
    assert np.array_equal(bits16(a), bits16(b))
    return a.cpu().numpy()


@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 96, 97, 129, 192, 255, 257])
@pytest.mark.parametrize("k,n,group,zeros", [(704, 144, 32, None), (2304, 400, 96, "int"), (4160, 16, 64, None),
                                             (1024, 272, 128, "any"), (1024, 1040, 32, "int"),
                                             (384, 144, 32, "int"), (1408, 272, 32, None)])
def test_int4(oracle, m, k, n, group, zeros):
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, group, asymmetric=zeros is not None)
    if zeros == "any":
        case.zeros[:, ::2] = np.float16(7.3)  # the subtraction rounds
    pre, s = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales)
    x, z = to_dev(case.x), None if zeros is None else to_dev(case.zeros)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, z, group_size=group))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, group))))


@pytest.mark.parametrize("m", [9, 16])
@pytest.mark.parametrize("n", [12272, 12304])
def test_int4_few_rows(oracle, m, n):
    """either side of the size from which up to 16 rows with zero points per group of 32 come here"""
    k, group = 4096, 32
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + n)), m, k, n, group, asymmetric=True)
    pre, s, z, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.zeros), to_dev(case.x)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, z, group_size=group))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, group))))


@pytest.mark.parametrize("m", [17, 48, 64, 65, 128, 160, 256, 300])
@pytest.mark.parametrize("bits,k,n,group", [(8, 320, 144, -1), (8, 1152, 528, 32), (8, 2112, 272, 64), (4, 4160, 400, -1)])
def test_ft(oracle, m, bits, k, n, group):
    rs = np.random.RandomState(m + k + n)
    x = rs.randn(m, k).astype(np.float16)
    w = rs.randint(-128, 128, size=(k, n * bits // 8)).astype(np.int8)
    s = rs.uniform(1e-4, 1e-3, size=(n,) if group < 0 else (k // group, n)).astype(np.float16)
    pre, xd, sd = ops.preprocess_weight_ft(to_dev(w), bits == 4), to_dev(x), to_dev(s)
    got = _twice(lambda: ops.gemm_fp16_ft(xd, pre, sd, bits, group_size=group))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(x, C.decode_ft_kn(w, s, bits, group), False)))


@pytest.mark.parametrize("rows", [[0, 33, 1, 40], [70, 0, 0, 20], [300, 1, 64, 0], [0, 513, 0, 127]])
@pytest.mark.parametrize("bits,k,n,group", [(4, 448, 272, 64), (8, 320, 144, -1)])
def test_experts(oracle, rows, bits, k, n, group):
    rs = np.random.RandomState(sum(rows) + n)
    total = sum(rows)
    x = rs.randn(total, k).astype(np.float16)
    w = rs.randint(-128, 128, size=(4, k, n * bits // 8)).astype(np.int8)
    s = rs.uniform(1e-3, 1e-2, size=(4, n) if group < 0 else (4, k // group, n)).astype(np.float16)
    indptr = np.cumsum(rows).astype(np.int64)
    pre, xd, sd, ip = ops.preprocess_weight_ft(to_dev(w), bits == 4), to_dev(x), to_dev(s), torch.from_numpy(indptr).cuda()
    got = _twice(lambda: ops.moe_gemm_ft(xd, pre, sd, ip))
    C = oracle.C()
    wq = np.stack([C.decode_ft_kn(w[e], s[e], bits, group).T for e in range(4)])
    assert_close(got, C.epilogue(C.group_gemm_f32(x, np.ascontiguousarray(wq), indptr)))


@pytest.mark.parametrize("m", [24, 64, 65, 128, 176, 256])
@pytest.mark.parametrize("k,n", [(1152, 528), (320, 144)])
def test_int4_groups_of_32_by_columns(oracle, m, k, n):
    """scales, and zero points, whose two groups of a 64-k block are no word: [K/32, N]"""
    test_ft(oracle, m, 4, k, n, 32)
    qweight, qzeros, scales, _, x, bias = gptq_case(m + k, m, k, n, 32)
    pre, zeros = ops.preprocess_weight_autogptq(u32_to_dev(qweight)), ops.unpack_zeros_autogptq(u32_to_dev(qzeros))
    xd, sd, bd = to_dev(x), to_dev(scales), to_dev(bias)
    got = _twice(lambda: ops.gemm_fp16_autogptq(xd, pre, sd, zeros, bias=bd))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(x, C.decode_autogptq(qweight, qzeros, scales, (np.arange(k) // 32).astype(np.uint32)), False), bias))


@pytest.mark.parametrize("m", [24, 64])
@pytest.mark.parametrize("tiles", [236, 238, 246, 248, 295])
@pytest.mark.parametrize("k", [64, 1088])
def test_a_tile_per_sm_and_runs_of_the_rest(oracle, m, tiles, k):
    """either side of the tile counts from which an SM's first CTA keeps a whole tile, with more CTAs than chunks left and fewer"""
    n = tiles * 128 - 48
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, 32)
    pre, s, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.x)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, group_size=32))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, None, 7.0, 32))))
