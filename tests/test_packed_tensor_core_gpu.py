"""The tensor-core kernels over packed weights (17 to 64 rows: one CTA per tile; above: CTA pairs) where
their tiles and splits can go wrong: rows around 32-row steps, tile widths and the border between the two
kernels, row counts that are no multiple of a 128- or 256-row tile, an odd number of 64-k blocks and a last
chunk of two, every scale source and zero-point form, and experts with more rows than a tile.  Each launch is repeated into a
new output and has to repeat itself bit for bit: the hand-over words are back at rest."""
import numpy as np
import pytest
import torch

from relax_b200 import get_launch_overlap, ops, set_launch_overlap, synth
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
@pytest.mark.parametrize("k", [64, 320, 1088])
def test_a_tile_per_sm_and_runs_of_the_rest(oracle, m, tiles, k):
    """either side of the tile counts from which an SM's first CTA keeps a whole tile: two chunks a tile (no fewer CTAs than chunks are
    left then), five, and one, where no tile is cut"""
    n = tiles * 128 - 48
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, 32)
    pre, s, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.x)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, group_size=32))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, None, 7.0, 32))))


@pytest.mark.parametrize("m", [24, 64])
def test_other_forms_of_runs_beside_whole_tiles(oracle, m):
    """zero points, the scale left to the sums, the epilogue's operands and the gated activation behind the same split"""
    k, n = 576, 248 * 128 - 32
    rs, C = np.random.RandomState(m), oracle.C()
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m)), m, k, n, 64, asymmetric=True)
    bias, res = rs.randn(n).astype(np.float16), rs.randn(m, n).astype(np.float16)
    pre, s, z, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.zeros), to_dev(case.x)
    b, r = to_dev(bias), to_dev(res)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, z, bias=b, residual=r, activation="relu", binary_op="plus", group_size=64))
    assert_close(got, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, 64)), bias, res, "relu", "plus"))
    w8, s8 = rs.randint(-128, 128, size=(k, n)).astype(np.int8), rs.uniform(1e-4, 1e-3, size=(n,)).astype(np.float16)
    pre8, s8d = ops.preprocess_weight_ft(to_dev(w8), False), to_dev(s8)
    assert_close(_twice(lambda: ops.gemm_fp16_ft(x, pre8, s8d, 8, group_size=-1)),
                 C.epilogue(C.matmul_f32(case.x, C.decode_ft_kn(w8, s8, 8, -1), False)))
    ffn, sg = n // 2, rs.uniform(1e-3, 1e-2, size=(n, k // 32)).astype(np.float16)
    pre, si = ops.preprocess_weight_gate_up(u32_to_dev(case.w)), ops.interleave_gate_up(to_dev(sg))
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, si, activation="swiglu")).astype(np.float64)
    y = C.matmul_f32(case.x, C.decode_q4_nk(case.w, sg, None, 7.0, 32)).astype(np.float64)
    exp = y[:, :ffn] / (1 + np.exp(-y[:, :ffn])) * y[:, ffn:]
    assert np.linalg.norm(got - exp) <= 1e-3 * np.linalg.norm(exp)


@pytest.mark.parametrize("m", [17, 31, 33, 50, 64, 81])
@pytest.mark.parametrize("k,n", [(2560, 144), (3136, 272), (4160, 1040), (11008, 16)])
def test_parts_of_a_tile_in_a_cluster(oracle, m, k, n):
    """columns that do not divide by the CTAs of a tile, a last tile of few weight rows (81 rows are the pair kernel's)"""
    rs = np.random.RandomState(m + k + n)
    C = oracle.C()
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, 32)
    pre, s, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.x)
    acc = C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, None, 7.0, 32))
    assert_close(_twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, group_size=32)), C.epilogue(acc))
    bias, res = rs.randn(n).astype(np.float16), rs.randn(m, n).astype(np.float16)
    b, r = to_dev(bias), to_dev(res)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, bias=b, residual=r, activation="relu", binary_op="plus", group_size=32))
    assert_close(got, C.epilogue(acc, bias, res, "relu", "plus"))
    w, s8 = rs.randint(-128, 128, size=(k, n)).astype(np.int8), rs.uniform(1e-4, 1e-3, size=(n,)).astype(np.float16)
    pre, s = ops.preprocess_weight_ft(to_dev(w), False), to_dev(s8)
    assert_close(_twice(lambda: ops.gemm_fp16_ft(x, pre, s, 8, group_size=-1)),
                 C.epilogue(C.matmul_f32(case.x, C.decode_ft_kn(w, s8, 8, -1), False)))


@pytest.mark.parametrize("m,k,n,group", [(20, 4160, 1040, 64), (50, 4096, 272, 128), (64, 3072, 144, 32), (12, 14336, 4096, 32)])
def test_zero_points_in_a_cluster(oracle, m, k, n, group):
    """and nine to sixteen rows, which groups of 32 with zero points bring here"""
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, group, asymmetric=True)
    case.zeros[::5, -1] = np.float16(7.3)
    pre, s, z, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.zeros), to_dev(case.x)
    got = _twice(lambda: ops.gemm_fp16_q4f16(x, pre, s, z, group_size=group))
    C = oracle.C()
    assert_close(got, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, group))))


@pytest.mark.parametrize("m,overlap", [(19, False), (32, True), (64, False)])
def test_gate_and_up_rows_of_a_cluster(oracle, m, overlap):
    """the gated activation, gate and up rows eight lanes apart, with overlap of launches where that is switched on"""
    k, ffn = 4096, 144
    rs = np.random.RandomState(m)
    x, w = rs.randn(m, k).astype(np.float16), rs.randint(0, 2 ** 32, size=(2 * ffn, k // 8), dtype=np.uint32)
    s = rs.uniform(1e-3, 1e-2, size=(2 * ffn, k // 32)).astype(np.float16)
    pre, si, xd = ops.preprocess_weight_gate_up(u32_to_dev(w)), ops.interleave_gate_up(to_dev(s)), to_dev(x)
    before = get_launch_overlap()
    set_launch_overlap(overlap)
    try:
        got = _twice(lambda: ops.gemm_fp16_q4f16(xd, pre, si, activation="swiglu")).astype(np.float64)
    finally:
        set_launch_overlap(before)
    y = oracle.C().matmul_f32(x, oracle.C().decode_q4_nk(w, s, None, 7.0, 32)).astype(np.float64)
    exp = y[:, :ffn] / (1 + np.exp(-y[:, :ffn])) * y[:, ffn:]
    assert np.linalg.norm(got - exp) <= 1e-3 * np.linalg.norm(exp)
