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
        f.write('#include "umma_index.h"\n'
                'extern "C" int pairs_fit_rows(int k, int bits) { return rb200::us::pairs_fit_rows(k, bits); }\n')
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
