"""The int4 kernel of one sequence of units per warp where its split can go wrong: warps without a chunk, chunks that k ends in,
short last row tiles, more row blocks than one meeting of the warps holds, every source of scales and zero points at
either side of its rule, and zero points that do not fit the codes' units."""
import numpy as np
import pytest
import torch

from relax_b200 import get_launch_overlap, ops, set_launch_overlap
from tests.test_gemv_gpu import _check_status
from tests.util import to_dev, u32_to_dev

pytestmark = pytest.mark.gpu


def _exact(case, group, x):
    """Unrounded: codes, zero points and scales in 64 bits."""
    n, k = case.w.shape[0], case.w.shape[1] * 8
    codes = ((case.w[:, :, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15).reshape(n, k).astype(np.float64)
    z = 7.0 if case.zeros is None else np.repeat(case.zeros.astype(np.float64), group, axis=1)
    return x.astype(np.float64) @ ((codes - z) * np.repeat(case.scales.astype(np.float64), group, axis=1)).T


# Weights that are not rounded to fp16 leave the output's own rounding, at most 2^-11 of a value; where calls
# stay with decoded weights another 2^-11 a weight, 2.8e-4 in the mean square.  Zero points that are no
# integers round u - z once more.  3e-5 for fp32 sums.
BOUND = 6e-4


@pytest.mark.parametrize("m,overlap", [(1, False), (4, True), (7, False), (13, True)])
@pytest.mark.parametrize("zeros", [None, "int", "any"])
@pytest.mark.parametrize("k,n,group", [(64, 16, 32), (192, 48, 32), (2304, 400, 32), (1856, 144, 32), (4096, 4752, 32), (256, 47632, 32),
                                       (256, 16, 64), (320, 48, 64), (2304, 400, 64), (4096, 1040, 64), (5504, 144, 64), (256, 47632, 64),
                                       (256, 16, 128), (640, 48, 128), (4096, 400, 128), (1152, 9488, 128), (4352, 144, 128),
                                       (512, 47632, 256), (320, 144, 320)])
def test_rows_of_scales(k, n, group, zeros, m, overlap):
    """scales [N, K / g]"""
    from relax_b200 import synth
    case = synth.q4_case(np.random.Generator(np.random.PCG64(m + k + n)), m, k, n, group, asymmetric=zeros is not None)
    if zeros == "any":  # of some row blocks only
        case.zeros[n // 2::5, -1] = np.float16(7.3)
    pre, s, x = ops.preprocess_weight_q4f16(u32_to_dev(case.w)), to_dev(case.scales), to_dev(case.x)
    z = None if zeros is None else to_dev(case.zeros)
    bias = torch.randn(n, device="cuda").half()
    torch.cuda.synchronize()  # (overlap: the weights are not the preceding kernel's)
    before = get_launch_overlap()
    set_launch_overlap(overlap)
    try:
        out = ops.gemm_fp16_q4f16(x, pre, s, z, bias=bias, group_size=group)
        _check_status()
    finally:
        set_launch_overlap(before)
    exp = _exact(case, group, case.x) + bias.cpu().numpy().astype(np.float64)
    got = out.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - exp) <= BOUND * np.linalg.norm(exp)
    assert np.abs(got - exp).max() <= 4 * BOUND * np.abs(exp).max()


@pytest.mark.parametrize("m", [1, 4, 8, 16])
@pytest.mark.parametrize("k,n,group,zeros", [(4096, 8208, 128, False), (8192, 80, 128, True), (1024, 1040, 128, True), (1152, 144, 128, True), (640, 48, 128, False),
                                             (4096, 8208, 64, False), (4096, 1040, 64, False), (960, 400, 64, False), (4096, 400, 64, True), (768, 144, 384, True),
                                             (1088, 144, -1, False), (64, 16, -1, False)])
def test_columns_of_scales(oracle, k, n, group, zeros, m):
    """scales [K / g, N], zero points beside them"""
    rs = np.random.RandomState(k + n + m)
    x = rs.randn(m, k).astype(np.float16)
    w = rs.randint(-128, 128, size=(k, n // 2)).astype(np.int8)
    groups = 1 if group < 0 else k // group
    s = rs.uniform(1e-3, 1e-2, size=(n,) if group < 0 else (groups, n)).astype(np.float16)
    C = oracle.C()
    if not zeros:
        out = ops.gemm_fp16_ft(to_dev(x), ops.preprocess_weight_ft(to_dev(w), True), to_dev(s), 4, group_size=group)
        wq = C.decode_ft_kn(w, s, 4, group).T.astype(np.float64)
    else:
        z = rs.randint(0, 16, size=(groups, n)).astype(np.float16)
        z[-1, ::3] = 3.7  # (k slices of some warps only)
        qw = rs.randint(0, 2 ** 32, size=(k // 8, n), dtype=np.uint32)
        out = ops.gemm_fp16_autogptq(to_dev(x), ops.preprocess_weight_autogptq(u32_to_dev(qw)), to_dev(s), to_dev(z))
        codes = ((qw[:, None, :] >> (4 * np.arange(8, dtype=np.uint32))[None, :, None]) & 15).reshape(k, n).astype(np.float64)
        wq = ((codes - np.repeat(z.astype(np.float64), group, axis=0)) * np.repeat(s.astype(np.float64), group, axis=0)).T
    _check_status()
    exp = x.astype(np.float64) @ wq.T
    got = out.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - exp) <= BOUND * np.linalg.norm(exp)


@pytest.mark.parametrize("m", [4, 7, 12, 16])
@pytest.mark.parametrize("k,n,group,zeros", [(512, 4736, 128, True), (512, 4752, 128, True), (512, 9488, 128, False), (512, 14224, 128, False),
                                             (512, 4752, 128, False), (1088, 4752, 64, False), (1088, 9488, 64, False), (1152, 4752, 128, True),
                                             (2112, 400, 64, False), (4352, 4752, 128, True)])
def test_either_side_of_the_lines(oracle, k, n, group, zeros, m):
    """one to four row blocks a CTA, and last chunks of one k block, with scales [K / g, N]"""
    test_columns_of_scales(oracle, k, n, group, zeros, m)


@pytest.mark.parametrize("m", [1, 4])
@pytest.mark.parametrize("k", [4096, 1856])
def test_swiglu_and_residual(oracle, m, k):
    """the epilogue's operands in the paired columns: gate and up rows, a residual of each row"""
    ffn, group = 144, 32
    rs = np.random.RandomState(k + m)
    x = rs.randn(m, k).astype(np.float16)
    w = rs.randint(0, 2 ** 32, size=(2 * ffn, k // 8), dtype=np.uint32)
    s = rs.uniform(1e-3, 1e-2, size=(2 * ffn, k // group)).astype(np.float16)
    pre, si = ops.preprocess_weight_gate_up(u32_to_dev(w)), ops.interleave_gate_up(to_dev(s))
    got = ops.gemm_fp16_q4f16(to_dev(x), pre, si, activation="swiglu").cpu().numpy().astype(np.float64)
    C = oracle.C()
    y = C.matmul_f32(x, C.decode_q4_nk(w, s, None, 7.0, group)).astype(np.float64)
    exp = y[:, :ffn] / (1 + np.exp(-y[:, :ffn])) * y[:, ffn:]
    assert np.linalg.norm(got - exp) <= 1e-3 * np.linalg.norm(exp)
    r = rs.randn(m, 2 * ffn).astype(np.float16)
    got = ops.gemm_fp16_q4f16(to_dev(x), ops.preprocess_weight_q4f16(u32_to_dev(w)), to_dev(s), residual=to_dev(r),
                              binary_op="plus").cpu().numpy().astype(np.float64)
    _check_status()
    exp = y + r
    assert np.linalg.norm(got - exp) <= 1e-3 * np.linalg.norm(exp)


@pytest.mark.parametrize("rows", [[0, 9, 0, 23], [1, 2, 0, 5], [32, 0, 0, 0], [0, 0, 0, 0]])
@pytest.mark.parametrize("k,n,group,zeros", [(512, 1040, 32, None), (320, 48, 32, "any"), (512, 9616, 64, "any"), (256, 144, 64, None),
                                             (1024, 144, 128, "int"), (512, 48, 128, None), (640, 144, 128, "any"), (64, 16, 64, None)])
def test_experts(k, n, group, zeros, rows):
    """expert layers: entries of up to eight rows, a CTA's share over several of them, rows of no expert untouched"""
    experts, total = len(rows), 32
    rs = np.random.RandomState(k + n + sum(rows))
    x = rs.randn(total, k).astype(np.float16)
    w = rs.randint(0, 2 ** 32, size=(experts, n, k // 8), dtype=np.uint32)
    s = rs.uniform(1e-3, 1e-2, size=(experts, n, k // group)).astype(np.float16)
    z = None if zeros is None else rs.randint(0, 16, size=s.shape).astype(np.float16)
    if zeros == "any":
        z[1, ::7, -1] = 7.3
    pre = torch.stack([ops.preprocess_weight_q4f16(u32_to_dev(w[e])) for e in range(experts)])
    indptr = np.cumsum(rows).astype(np.int64)
    out = torch.full((total, n), -7.0, dtype=torch.float16, device="cuda")
    ops.moe_gemm_q4f16(to_dev(x), pre, to_dev(s), torch.from_numpy(indptr).cuda(), None if z is None else to_dev(z), group_size=group, out=out)
    _check_status()
    got = out.cpu().numpy().astype(np.float64)
    assert np.all(got[indptr[-1]:] == -7.0)
    codes = ((w[..., None] >> (4 * np.arange(8, dtype=np.uint32))) & 15).reshape(experts, n, k).astype(np.float64)
    wq = (codes - (7.0 if z is None else np.repeat(z.astype(np.float64), group, axis=2))) * np.repeat(s.astype(np.float64), group, axis=2)
    begin = 0
    for e, end in enumerate(indptr):
        exp = x[begin:end].astype(np.float64) @ wq[e].T
        assert np.linalg.norm(got[begin:end] - exp) <= BOUND * np.linalg.norm(exp)
        begin = end


def _zeros_of(kind, rs, shape):
    z = rs.randint(0, 16, size=shape).astype(np.float16)
    if kind == "all":  # sixteenths, below zero and large ones among them
        z = (rs.uniform(0, 15, size=shape)).astype(np.float16)
        z.reshape(-1)[::7] = 5.0625
        z.reshape(-1)[3::11] = -2.7
        z.reshape(-1)[5::13] = 71.3
    return z


@pytest.mark.parametrize("m", [1, 3, 4, 8, 11, 16])
@pytest.mark.parametrize("k,n,group,columns", [(4096, 1040, 32, False), (192, 48, 32, False), (4096, 8208, 32, False), (2368, 400, 32, False),
                                               (4096, 1040, 64, False), (256, 47632, 64, False), (4096, 1040, 128, False), (1152, 9488, 128, False),
                                               (8192, 4112, 128, True), (768, 144, 384, True), (11008, 4112, 128, True)])
def test_fractional_zero_points(k, n, group, columns, m):
    """Every zero point with a fraction: what the codes' units cannot hold is taken off afterwards, from more row blocks than one
    meeting of the warps holds, warps without a chunk and short last chunks among them.  Outputs round to fp16, 2^-11 of a
    value at most; the fractions' 12 bits are less than a tenth of that."""
    rs = np.random.RandomState(m + k + n + group)
    x = rs.randn(m, k).astype(np.float16)
    w = rs.randint(0, 2 ** 32, size=(n, k // 8), dtype=np.uint32)
    s = rs.uniform(1e-3, 1e-2, size=(n, k // group)).astype(np.float16)
    z = _zeros_of("all", rs, s.shape)
    if columns:
        codes = ((w[:, :, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15).reshape(n, k)
        qw = np.zeros((k // 8, n), dtype=np.uint32)
        for i in range(8):
            qw |= codes.T[i::8].astype(np.uint32) << np.uint32(4 * i)
        out = ops.gemm_fp16_autogptq(to_dev(x), ops.preprocess_weight_autogptq(u32_to_dev(qw)), to_dev(np.ascontiguousarray(s.T)),
                                     to_dev(np.ascontiguousarray(z.T)))
    else:
        out = ops.gemm_fp16_q4f16(to_dev(x), ops.preprocess_weight_q4f16(u32_to_dev(w)), to_dev(s), to_dev(z), group_size=group)
        codes = ((w[:, :, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15).reshape(n, k)
    _check_status()
    wq = (codes - np.repeat(z.astype(np.float64), group, axis=1)) * np.repeat(s.astype(np.float64), group, axis=1)
    exp = x.astype(np.float64) @ wq.T
    got = out.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - exp) <= BOUND * np.linalg.norm(exp)
    assert np.abs(got - exp).max() <= 4 * BOUND * np.abs(exp).max()


@pytest.mark.parametrize("k,group", [(1024, 32), (1088, 32), (1024, 64), (1024, 128), (1152, 128), (1024, 256)])
@pytest.mark.parametrize("m", [1, 4, 8, 16])
def test_infinities_beside_fractional_zero_points(k, group, m):
    """An infinite activation has the sign of its weight, also where its code is the zero point's integer; an infinite scale or zero
    point stays with its row."""
    n = 272
    rs = np.random.RandomState(m + group)
    x = rs.randn(m, k).astype(np.float16)
    x[m - 1, 700] = np.inf
    w = rs.randint(0, 2 ** 32, size=(n, k // 8), dtype=np.uint32)
    s = rs.uniform(1e-3, 1e-2, size=(n, k // group)).astype(np.float16)
    z = _zeros_of("all", rs, s.shape)
    z[::2, 700 // group] = np.float16(7.3)

    def call(s, z):
        return ops.gemm_fp16_q4f16(to_dev(x), ops.preprocess_weight_q4f16(u32_to_dev(w)), to_dev(s), to_dev(z), group_size=group).cpu().numpy()

    got = call(s, z)
    with np.errstate(invalid="ignore"):
        exp = (((w[:, 700 // 8] >> (4 * (700 % 8))) & 15) - z[:, 700 // group].astype(np.float64)) * np.inf
    assert np.array_equal(got[m - 1].astype(np.float64), exp, equal_nan=True)
    assert np.isfinite(got[:m - 1]).all()
    s[5, 1], z[18, 2], z[40, 3] = np.inf, np.inf, np.nan
    finite = np.ones((m, n), dtype=bool)
    finite[m - 1], finite[:, [5, 18, 40]] = False, False
    assert np.array_equal(np.isfinite(call(s, z)), finite)


@pytest.mark.parametrize("group", [32, 64, 128])
@pytest.mark.parametrize("m", [1, 8, 16])
def test_fractional_zero_points_take_no_second_pass(group, m):
    """Weights are read once whatever the zero points are: a matmul took 2.6 to 3.4 times as long with fractions in all of them and
    2.3 times with a single one while they were read and decoded again; now 1.2 to 1.5 times and 1.1."""
    k, n = 4096, 22016
    g = torch.Generator(device="cuda")
    g.manual_seed(m + group)
    pre = ops.preprocess_weight_q4f16(torch.randint(-2 ** 31, 2 ** 31 - 1, (n, k // 8), dtype=torch.int32, device="cuda", generator=g))
    s = (torch.rand(n, k // group, device="cuda", generator=g) * 0.009 + 0.001).half()
    whole = torch.randint(0, 16, s.shape, device="cuda", generator=g).half()
    one = whole.clone()
    one[n // 2, 3] = 7.3
    x, out = torch.randn(m, k, device="cuda", generator=g).half(), torch.empty(m, n, dtype=torch.float16, device="cuda")
    times = {}
    graphs = {}
    for name, z in (("whole", whole), ("one", one), ("all", whole + 0.3)):
        graphs[name] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[name]):
            for _ in range(20):
                ops.gemm_fp16_q4f16(x, pre, s, z, group_size=group, out=out)
        times[name] = []
    for _ in range(8):
        for name, graph in graphs.items():
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            times[name].append(a.elapsed_time(b))
    best = {name: min(t) for name, t in times.items()}
    assert best["all"] <= 2.0 * best["whole"] and best["one"] <= 1.5 * best["whole"], best
