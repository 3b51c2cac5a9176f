"""The weight-loading kernels at the edges of their tiles: the quantiser's row slices (one CTA, a
cluster of two to eight, slices of whole groups) and values on rounding boundaries; the repack's
stage runs with short last row tiles and short last k-chunks, in every source layout.  All exact."""
import numpy as np
import pytest
import torch

from relax_b200 import ops, synth
from tests.layout_ref import fragment_layout
from tests.util import to_dev, u32_to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,group,n,k", [(4, -1, 32, 8), (8, -1, 64, 1024), (4, -1, 32, 1032), (8, -1, 32, 4104),
                                            (4, -1, 64, 14336), (8, 64, 32, 1088), (4, 24, 64, 2064), (8, 1024, 32, 3072)])
def test_encode_slices(oracle, bits, group, n, k):
    rs = np.random.RandomState(bits * 1000 + k)
    y = rs.normal(0, 0.02, size=(n, k)).astype(np.float16)
    y[1, :] = 0
    y[2, :] = rs.choice([-1, 1], size=k) * 2.0 ** -24   # below the scale's floor
    # exact ties: absmax 1 gives the scale 1/8 (1/128), odd multiples of half of it are boundaries
    y[3, :] = ((2 * rs.randint(-4, 4, size=k) + 1) / (16.0 if bits == 4 else 256.0)).astype(np.float16)
    y[3, ::max(1, (group if group > 0 else k))] = 1.0
    packed, scales = ops.encode_ft(to_dev(y), bits, group)
    exp_packed, exp_scales = oracle.np_encode_ft(y, bits, group)
    assert np.array_equal(scales.cpu().numpy().view(np.uint16), exp_scales.view(np.uint16))
    assert np.array_equal(packed.cpu().numpy(), exp_packed)


def _gate_up_rows(codes):
    n = codes.shape[0]
    j = np.arange(n)
    src = np.where(j % 16 < 8, 8 * (j // 16) + j % 16, n // 2 + 8 * (j // 16) + j % 16 - 8)
    return codes[src]


@pytest.mark.parametrize("n,k", [(32, 64), (160, 320), (128, 256), (288, 832)])
@pytest.mark.parametrize("source", ["q4", "gptq", "ft4", "ft8", "q4_gate_up", "ft4_gate_up", "ft8_gate_up"])
def test_repack_stage_runs(oracle, source, n, k):
    bits = 8 if source.startswith("ft8") else 4
    rs = np.random.RandomState(n + k)
    codes = rs.randint(0, 1 << bits, size=(n, k)).astype(np.uint8)
    if source.startswith("q4"):
        src = u32_to_dev(synth.pack_q4_nk(codes))
        pre = ops.preprocess_weight_gate_up(src) if source.endswith("gate_up") else ops.preprocess_weight_q4f16(src)
    elif source == "gptq":
        words = synth.pack_q4_nk(np.ascontiguousarray(codes))   # [N, K/8]
        pre = ops.preprocess_weight_autogptq(u32_to_dev(np.ascontiguousarray(words.T)))
    else:
        c = codes.T.astype(np.int16) - (8 if bits == 4 else 128)  # signed [K, N]
        src = (c[:, 0::2] & 15) | ((c[:, 1::2] & 15) << 4) if bits == 4 else c
        src = to_dev((src & 255).astype(np.uint8).view(np.int8))
        pre = ops.preprocess_weight_gate_up(src, ops.LAYOUT_FT_KN, bits == 4) if source.endswith("gate_up") \
            else ops.preprocess_weight_ft(src, bits == 4)
    rows = _gate_up_rows(codes) if source.endswith("gate_up") else codes
    got = pre.cpu().numpy().view(np.uint8).reshape(-1)
    assert np.array_equal(got, fragment_layout(np.ascontiguousarray(rows), bits))


def test_repack_of_a_source_without_vector_alignment():
    """A view that starts in the middle of a 16-byte line takes the element-wise kernel."""
    rs = np.random.RandomState(7)
    n, k = 48, 96
    flat = to_dev(rs.randint(-128, 128, size=k * n + 4).astype(np.int8))
    view = flat[4:4 + k * n].view(k, n)
    assert torch.equal(ops.preprocess_weight_ft(view, False), ops.preprocess_weight_ft(view.clone(), False))
