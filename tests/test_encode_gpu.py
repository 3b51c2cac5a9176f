"""The GPU quantiser against the numpy restatement of the reference's encode TIR
(tests/python/relax/test_codegen_cutlass.py:1391-1457, :1630-1676, :2043-2109): codes and scales
bit for bit, then the reference tests' whole flow - encode, preprocess, fused decode-matmul -
against the unquantised product at the reference's tolerance."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from relax_b200 import ops
from tests.util import to_dev

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("bits,group,n,k", [(4, -1, 128, 64), (8, -1, 128, 64), (8, 64, 128, 128), (4, 64, 96, 256),
                                            (4, -1, 1000, 2048), (8, 128, 250, 1024)])
def test_encode_matches_reference_quantiser(oracle, bits, group, n, k):
    rs = np.random.RandomState(bits + n)
    y = rs.normal(0, 0.002, size=(n, k)).astype(np.float16)
    y[3, :] = 0  # an all-zero row exercises the 1e-4 floor of the scale
    packed, scales = ops.encode_ft(to_dev(y), bits, group)
    torch.cuda.synchronize()
    exp_packed, exp_scales = oracle.np_encode_ft(y, bits, group)
    assert np.array_equal(scales.cpu().numpy().view(np.uint16), exp_scales.view(np.uint16))
    assert np.array_equal(packed.cpu().numpy(), exp_packed)


def test_reference_flow_entirely_on_gpu():
    """x 64x64, y 128x64 as in test_fp16A_int4B_gemm: encode -> ft_preprocess_weight -> matmul + bias."""
    rs = np.random.RandomState(0)
    x = rs.randn(64, 64).astype(np.float16)
    y = rs.normal(0, 0.002, size=(128, 64)).astype(np.float16)
    bias = rs.randn(1, 128).astype(np.float16)
    packed, scales = ops.encode_ft(to_dev(y), 4)
    pre = ops.preprocess_weight_ft(packed, True, 80)
    out = ops.gemm_fp16_ft(to_dev(x), pre, scales, 4, bias=to_dev(bias))
    ref = np.dot(x.astype(np.float32), y.astype(np.float32).T) + bias.astype(np.float32)
    np.testing.assert_allclose(out.cpu().numpy().astype(np.float32), ref, rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("bits,group", [(4, -1), (8, -1), (4, 64), (8, 64), (8, 24), (4, 512), (8, 768)])
@pytest.mark.parametrize("k", [768, 4608, 12288])
def test_encode_of_long_rows_ties_and_special_values(oracle, bits, group, k):
    """CTAs of 256 and 512 threads, one and several per cluster, groups folded over lanes or not: values on
    and next to rounding boundaries, at the top of the range, infinities and NaN.  n % 32 == 0 takes the
    kernel with the nudged reciprocal; the same rows and two more take the one that divides."""
    if group > 0 and k % group:
        pytest.skip("groups must divide k")
    n = 96
    rs = np.random.RandomState(bits + k)
    y = rs.normal(0, 0.02, size=(n, k)).astype(np.float16)
    g = k if group <= 0 else group
    for r in range(n):  # ties: (2 c + 1) / 2 scales of every group's own maximum, and their neighbours
        m = np.abs(y[r].reshape(-1, g)).max(axis=1, keepdims=True).astype(np.float32)
        c = rs.randint(0, 2 ** (bits - 1), size=(k // g, g // 4))
        t = ((2 * c + 1) * m / 2 ** bits).astype(np.float16)
        t = (t.view(np.uint16) + rs.randint(-1, 2, size=t.shape)).astype(np.uint16).view(np.float16)
        y[r].reshape(-1, g)[:, 1:1 + g // 4] = np.where(np.abs(t) <= m, t, 0) * rs.choice([-1, 1], size=t.shape)
    y[3, :] = 0
    y[5, :] = (y[5] * 2e-3).astype(np.float16)  # below the floor of the scale
    packed, scales = ops.encode_ft(to_dev(y), bits, group)
    exp_packed, exp_scales = oracle.np_encode_ft(y, bits, group)
    assert np.array_equal(scales.cpu().numpy().view(np.uint16), exp_scales.view(np.uint16))
    assert np.array_equal(packed.cpu().numpy(), exp_packed)
    y[7, k - 3] = np.inf
    y[8, 5] = -np.inf
    y[40, 17] = np.nan
    y[41, :] = np.nan
    both = np.concatenate([y, y[:2]])
    want_packed, want_scales = ops.encode_ft(to_dev(both), bits, group)
    packed, scales = ops.encode_ft(to_dev(y), bits, group)
    cols = n // 2 if bits == 4 else n
    assert torch.equal(scales.view(torch.int16), want_scales[..., :n].contiguous().view(torch.int16))
    assert torch.equal(packed, want_packed[:, :cols])


@pytest.mark.parametrize("bits,group", [(4, -1), (8, -1), (8, 64), (4, 24)])
@pytest.mark.parametrize("n,k", [(32 * 701, 1056), (32 * 131, 4104)])
def test_encode_with_several_tiles_per_cta(oracle, bits, group, n, k):
    """More row tiles than run at once: every buffer and every place for the maxima is used again, several
    times over, with row maxima that differ from tile to tile."""
    if group > 0 and k % group:
        k = k // group * group
    rs = np.random.RandomState(bits)
    y = (rs.standard_normal((n, k)).astype(np.float32) * rs.uniform(0.001, 0.2, size=(n, 1)).astype(np.float32)).astype(np.float16)
    exp_packed, exp_scales = oracle.np_encode_ft(y, bits, group)
    w = to_dev(y)
    for _ in range(3):
        packed, scales = ops.encode_ft(w, bits, group)
        assert np.array_equal(scales.cpu().numpy().view(np.uint16), exp_scales.view(np.uint16))
        assert np.array_equal(packed.cpu().numpy(), exp_packed)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("k", [512, 4096, 12288])
def test_row_maximum_without_the_nans(oracle, bits, k):
    """One scale per row, one, eight and sixteen CTAs a cluster: whole vectors of NaN, and NaN at the even or the
    odd places of one only, in the first, a middle and the last slice.  NaN is no maximum, in any pattern."""
    n, finite = 64, np.random.RandomState(k + bits).normal(0, 0.02, size=(64, k)).astype(np.float16)
    nan = np.zeros((n, k), dtype=bool)
    for r, (at, places) in enumerate([(at, p) for at in (0, k // 2 // 8 * 8, k - 8)
                                      for p in (slice(0, 8), slice(0, 8, 2), slice(1, 8, 2), slice(3, 4))]):
        nan[2 * r, at:at + 8][places] = True
    nan[25, :k // 2] = True
    nan[27, 1::2] = True
    y = finite.copy()
    y[nan] = np.float16(np.nan)
    y[4] = -y[4]  # NaN with the sign set
    got, scales = ops.encode_ft(to_dev(y), bits)
    want, want_scales = ops.encode_ft(to_dev(np.concatenate([y, y[:2]])), bits)  # the any-shape kernel
    assert torch.equal(scales.view(torch.int16), want_scales[:n].view(torch.int16))
    assert torch.equal(got, want[:, :n // 2 if bits == 4 else n])
    finite[nan] = 0
    finite[4] = -finite[4]
    exp, exp_scales = oracle.np_encode_ft(finite, bits, -1)
    assert np.array_equal(scales.cpu().numpy().view(np.uint16), exp_scales.view(np.uint16).reshape(-1))

    def codes(p):  # [n, k]
        p = p.view(np.uint8).T
        return np.stack([p & 15, p >> 4], axis=1).reshape(n, k) if bits == 4 else p
    assert np.array_equal(codes(got.cpu().numpy())[~nan], codes(exp)[~nan])


@pytest.mark.parametrize("bits,group", [(4, 8), (8, 8), (4, 16), (8, 1024)])
def test_encode_of_the_smallest_and_largest_groups(oracle, bits, group):
    """Groups of 8 have the most scales in shared memory, one CTA of sixteen warps an SM."""
    test_encode_of_long_rows_ties_and_special_values(oracle, bits, group, 4096)
    test_encode_with_several_tiles_per_cta(oracle, bits, group, 32 * 131, 4096)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("n,k", [(32, 16384), (32, 16392), (32 * 40, 18944), (64, 24576), (64, 24584), (32 * 40, 28672),
                                 (32, 50176), (32, 50184)])
def test_encode_of_rows_beyond_three_buffers(oracle, bits, n, k):
    """Two buffers or one a CTA, one and several row tiles a cluster, and the first length that is left to the
    kernel for any shape."""
    rs = np.random.RandomState(bits + k)
    y = (rs.standard_normal((n, k)).astype(np.float32) * rs.uniform(0.001, 0.2, size=(n, 1)).astype(np.float32)).astype(np.float16)
    exp_packed, exp_scales = oracle.np_encode_ft(y, bits, -1)
    w = to_dev(y)
    for _ in range(3):
        packed, scales = ops.encode_ft(w, bits)
        assert np.array_equal(scales.cpu().numpy().view(np.uint16), exp_scales.view(np.uint16))
        assert np.array_equal(packed.cpu().numpy(), exp_packed)


FIRST_CALL = """
import ctypes
import torch
from relax_b200 import _lib, ops
lib, st = _lib.load(), ctypes.c_int(-1)
assert lib.rb200_check_async_error(None, ctypes.byref(st)) == 0 and st.value == 0  # before there is any status word
w = torch.randn(1024, 4096, device="cuda").half()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    packed, scales = ops.encode_ft(w, 4)
graph.replay()
torch.cuda.synchronize()
assert lib.rb200_check_async_error(None, ctypes.byref(st)) == 0 and st.value == 0
again, scales_again = ops.encode_ft(w, 4)
assert torch.equal(packed, again) and torch.equal(scales, scales_again)
assert lib.rb200_check_async_error(None, ctypes.byref(st)) == 0 and st.value == 0
"""


def test_quantising_is_the_first_call_of_a_process():
    """Its waits report through a status word that needs no earlier call, here under capture."""
    r = subprocess.run([sys.executable, "-c", FIRST_CALL], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
