"""The small-batch decode kernel (m <= 16, and expert layers of at most 32 rows) where its split can go
wrong: k slices without a chunk, short last chunks and row tiles, odd row-block counts, the four-warp
form of wide weights, scale sources, and experts with more rows than one pass holds."""
import numpy as np
import pytest
import torch

from relax_b200 import ops, synth
from tests.test_gemv_gpu import _check_status
from tests.util import assert_close, to_dev, u32_to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("k,n,group,asym", [(64, 16, 32, False), (704, 48, 32, True), (2304, 1040, 32, False),
                                            (2304, 400, 128, True), (1920, 144, 96, True), (256, 29056, 32, False),
                                            (512, 28688, 256, True), (704, 144, 64, True), (960, 48, 192, False)])
def test_int4_split(oracle, m, k, n, group, asym):
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, group, asymmetric=asym)
    pre = ops.preprocess_weight_q4f16(u32_to_dev(case.w))
    z = to_dev(case.zeros) if asym else None
    out = ops.gemm_fp16_q4f16(to_dev(case.x), pre, to_dev(case.scales), z, group_size=group)
    _check_status()
    C = oracle.C()
    assert_close(out.cpu().numpy(), C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, group))))


@pytest.mark.parametrize("m", [5, 13])
@pytest.mark.parametrize("k,n,group", [(32, 16, -1), (288, 80, -1), (1056, 272, 32), (1152, 144, 64), (128, 28704, -1)])
def test_int8_split(oracle, m, k, n, group):
    rs = np.random.RandomState(k + n)
    x = rs.randn(m, k).astype(np.float16)
    packed = rs.randint(-127, 128, size=(k, n)).astype(np.int8)
    scales = rs.uniform(1e-4, 1e-3, size=(n,) if group < 0 else (k // group, n)).astype(np.float16)
    out = ops.gemm_fp16_ft(to_dev(x), ops.preprocess_weight_ft(to_dev(packed), False), to_dev(scales), 8, group_size=group)
    _check_status()
    C = oracle.C()
    assert_close(out.cpu().numpy(), C.epilogue(C.matmul_f32(x, C.decode_ft_kn(packed, scales, 8, group), False)))


@pytest.mark.parametrize("rows", [[0, 9, 0, 23], [32, 0, 0, 0], [1, 1, 1, 1], [0, 0, 0, 0]])
@pytest.mark.parametrize("bits,k,n", [(4, 384, 144), (8, 320, 16), (4, 128, 7168)])
def test_experts(oracle, rows, bits, k, n):
    rs = np.random.RandomState(sum(rows) + n)
    x = rs.randn(32, k).astype(np.float16)
    w = rs.randint(-128, 128, size=(4, k, n // 2 if bits == 4 else n)).astype(np.int8)
    s = rs.uniform(0.001, 0.01, size=(4, k // 64, n)).astype(np.float16)
    indptr = np.cumsum(rows).astype(np.int64)
    out = torch.full((32, n), -7.0, dtype=torch.float16, device="cuda")
    ops.moe_gemm_ft(to_dev(x), ops.preprocess_weight_ft(to_dev(w), bits == 4), to_dev(s), torch.from_numpy(indptr).cuda(), out=out)
    _check_status()
    C = oracle.C()
    total = int(indptr[-1])
    got = out.cpu().numpy()
    assert np.all(got[total:] == -7.0)  # rows of no expert stay as they are
    if total:
        wq = np.stack([C.decode_ft_kn(w[e], s[e], bits, 64).T for e in range(4)])
        assert_close(got[:total], C.epilogue(C.group_gemm_f32(x[:total], np.ascontiguousarray(wq), indptr)))


@pytest.mark.parametrize("experts,rows", [(128, 32), (160, 9), (65, 1)])
def test_many_experts(oracle, experts, rows):
    """More experts than rows by far: their number is not limited where the rows are few."""
    rs = np.random.RandomState(experts + rows)
    k, n = 128, 48
    x = rs.randn(rows, k).astype(np.float16)
    w = rs.randint(-128, 128, size=(experts, k, n // 2)).astype(np.int8)
    s = rs.uniform(0.001, 0.01, size=(experts, k // 64, n)).astype(np.float16)
    indptr = np.cumsum(np.bincount(rs.randint(0, experts, size=rows), minlength=experts)).astype(np.int64)
    out = ops.moe_gemm_ft(to_dev(x), ops.preprocess_weight_ft(to_dev(w), True), to_dev(s), torch.from_numpy(indptr).cuda())
    _check_status()
    C = oracle.C()
    wq = np.stack([C.decode_ft_kn(w[e], s[e], 4, 64).T for e in range(experts)])
    assert_close(out.cpu().numpy(), C.epilogue(C.group_gemm_f32(x, np.ascontiguousarray(wq), indptr)))


def _forms():
    yield "ft4_row", 4, -1, None
    yield "ft8_row", 8, -1, None
    yield "ft8_64", 8, 64, None
    yield "q4_row_zeros", 4, -1, "int"
    yield "q4_128_zeros", 4, 128, "int"
    yield "q4_64_rounded_zeros", 4, 64, "any"
    yield "q4_32", 4, 32, None


def _call(oracle, name, bits, group, zeros, x, n, seed):
    """One call on random codes; returns (result, decoded weights [n, k] in fp64)."""
    k = x.shape[1]
    rs = np.random.RandomState(seed)
    C = oracle.C()
    if name.startswith("ft"):
        w = rs.randint(-128, 128, size=(k, n * bits // 8)).astype(np.int8)
        s = rs.uniform(1e-4, 1e-3, size=(n,) if group < 0 else (k // group, n)).astype(np.float16)
        out = ops.gemm_fp16_ft(to_dev(x), ops.preprocess_weight_ft(to_dev(w), bits == 4), to_dev(s), bits, group_size=group)
        wq = C.decode_ft_kn(w, s, bits, group).T
    else:
        group = k if group < 0 else group
        case = synth.q4_case(np.random.Generator(np.random.PCG64(seed)), 1, k, n, group, asymmetric=zeros is not None)
        if zeros == "any":
            case.zeros[:, ::2] = np.float16(7.3)
        z = None if zeros is None else to_dev(case.zeros)
        out = ops.gemm_fp16_q4f16(to_dev(x), ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), z, group_size=group)
        wq = C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, group)
    _check_status()
    return out.cpu().numpy().astype(np.float64), wq.astype(np.float64)


@pytest.mark.parametrize("m", [1, 8, 9])
@pytest.mark.parametrize("form", list(_forms()), ids=lambda f: f[0])
def test_activations_with_an_offset(oracle, form, m):
    """Activations far from zero mean over a long k: the zero point has to leave the codes before they are
    summed, or the sums of codes and of zero points cancel.  Bound: a weight that is not rounded to fp16
    differs from the decoded one by at most 2^-11, 2.8e-4 in the mean square, the output's rounding is
    another 2.8e-4, and fp32 sums of k / 128 MMAs add 3e-5: 4e-4 in the 2-norm, and 1e-3 asked."""
    k, n = 28672, 64
    x = (np.abs(np.random.RandomState(m).randn(m, k)) + 4.0).astype(np.float16)
    got, wq = _call(oracle, *form, x, n, 11)
    exp = x.astype(np.float64) @ wq.T
    assert np.linalg.norm(got - exp) <= 1e-3 * np.linalg.norm(exp)


@pytest.mark.parametrize("m", [1, 8, 9])
@pytest.mark.parametrize("form", list(_forms()), ids=lambda f: f[0])
def test_infinite_activation(oracle, form, m):
    """One infinite activation: infinite results with the sign of its weight, NaN where that weight is zero."""
    k, n = 1024, 256
    x = np.random.RandomState(m).randn(m, k).astype(np.float16)
    x[0, 517] = np.inf
    got, wq = _call(oracle, *form, x, n, 12)
    with np.errstate(invalid="ignore"):
        exp = x.astype(np.float64) @ wq.T
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    assert np.array_equal(np.isposinf(got), np.isposinf(exp)) and np.array_equal(np.isneginf(got), np.isneginf(exp))


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("k,n", [(256, 16), (2304, 400), (4096, 4752)])
def test_group_32_with_zero_points(oracle, m, k, n):
    """one row block per pass: a single one, a short last row tile, several passes per CTA"""
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, 32, asymmetric=True)
    pre, s, z, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.zeros), to_dev(case.x)
    out = ops.gemm_fp16_q4f16(x, pre, s, z, group_size=32).cpu().numpy()
    C = oracle.C()
    assert_close(out, C.epilogue(C.matmul_f32(case.x, C.decode_q4_nk(case.w, case.scales, case.zeros, 7.0, 32))))
