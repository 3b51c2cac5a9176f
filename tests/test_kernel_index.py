"""Index arithmetic shared by host and device code, compiled here for the host and checked over whole ranges:
what stays inside a tensor cannot be seen from results where the value read is not used."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "relax_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    src, so = str(d / "index.cc"), str(d / "index.so")
    with open(src, "w") as f:
        f.write('#include "umma_index.h"\n#include "encode_plan.h"\n'
                'extern "C" int pairs_fit_rows(int k, int bits) { return rb200::us::pairs_fit_rows(k, bits); }\n'
                'static rb200::FitCache cache;\n'
                'extern "C" int clusters_fit(int dev, int ranks, long smem, int answer, int* asked) {\n'
                '  return cache.get(dev, ranks, smem, [&] { ++*asked; return answer; }); }\n'
                'extern "C" int encode_rows(long k, int* out) { rb200::EncodePlan p; if (!rb200::plan_encode_rows(k, &p)) return 0;\n'
                '  out[0] = p.slice, out[1] = p.slices, out[2] = p.bufs, out[3] = p.threads, out[4] = (int)p.smem; return 1; }\n'
                'extern "C" int encode_groups(long k, long group, int* out) { rb200::EncodePlan p;\n'
                '  if (!rb200::plan_encode_groups(k, group, &p)) return 0;\n'
                '  out[0] = p.slice, out[1] = p.slices, out[2] = p.bufs, out[3] = p.threads, out[4] = (int)p.smem; return 1; }\n')
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I" + CSRC, src, "-o", so])
    return ctypes.CDLL(so)


@pytest.mark.parametrize("bits,chunk_blocks", [(4, 4), (8, 2)])
def test_scale_pairs_stay_in_their_row(lib, bits, chunk_blocks):
    """Group 32: where scales are fetched for pairs of 64-k blocks, every pair of every chunk is in the row."""
    fitting = 0
    for k in range(64, 32768 + 1, 64):
        if not lib.pairs_fit_rows(k, bits):
            continue
        fitting += 1
        k_blocks = k // 64
        for chunk in range(-(-k_blocks // chunk_blocks)):
            for kb in range(chunk * chunk_blocks, (chunk + 1) * chunk_blocks, 2):
                assert kb % 2 == 0 and kb + 2 <= k_blocks, (k, kb)
    assert fitting == 32768 // (64 * chunk_blocks)


def test_a_cluster_that_does_not_fit_leaves_other_shapes_alone(lib):
    """The answer for one launch shape is never given for another, in particular not a 0."""
    asked = ctypes.c_int(0)

    def fit(dev, ranks, smem, answer):
        return lib.clusters_fit(dev, ranks, ctypes.c_long(smem), answer, ctypes.byref(asked))
    shapes = [(0, 8, 99000), (0, 16, 99000), (0, 8, 200000), (1, 8, 99000)]
    for answer, shape in enumerate(shapes):
        assert fit(*shape, answer) == answer
        assert fit(*shape, 77) == answer  # kept, a 0 too
    assert fit(*shapes[0], 18) == 18 and fit(*shapes[1], 0) == 0 and fit(*shapes[0], 18) == 18
    assert asked.value == 7


def test_rows_up_to_50176_are_read_once(lib):
    """The quantiser's slices cover every row, none of them empty, in shared memory that a CTA can have; the kernel
    that reads twice is left to rows beyond what one buffer of sixteen CTAs holds."""
    out, most = (ctypes.c_int * 5)(), {1: 0, 2: 0, 3: 0}
    for k in range(8, 60001, 8):
        planned = lib.encode_rows(ctypes.c_long(k), out)
        assert planned == (k <= 50176), k
        if not planned:
            continue
        piece, pieces, bufs, threads, smem = out
        assert piece % 8 == 0 and piece * pieces >= k > piece * (pieces - 1) and pieces <= 16, k
        assert bufs * 32 * -(-piece // 64) * 128 < smem <= 200 * 1024, k
        assert threads == (256 if piece <= 512 else 512), k  # two CTAs an SM, or one
        most[bufs] = max(most[bufs], k)
    assert most == {3: 16384, 2: 24576, 1: 50176}


@pytest.mark.parametrize("group", list(range(8, 1025, 8)))
def test_groups_are_whole_in_a_slice_and_an_sm_has_sixteen_warps(lib, group):
    out = (ctypes.c_int * 5)()
    for k in (group * 2, group * 3, group * 130):
        assert lib.encode_groups(ctypes.c_long(k), ctypes.c_long(group), out)
        piece, pieces, bufs, threads, smem = out
        assert bufs == 3 and piece % group == 0 and piece * pieces >= k > piece * (pieces - 1)
        assert 3 * 32 * -(-piece // 64) * 128 < smem <= 200 * 1024
        two = 2 * (smem + 1536) <= 228 * 1024
        assert threads == (256 if two else 512) and (group == 8) == (piece <= 512 and not two)
