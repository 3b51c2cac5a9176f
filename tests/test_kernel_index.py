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
                'extern "C" int pair_in_row(int kb, int k_blocks) { return rb200::us::pair_in_row(kb, k_blocks); }\n')
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I" + CSRC, src, "-o", so])
    return ctypes.CDLL(so)


def test_scale_pairs_stay_in_their_row(lib):
    """Group 32, k a multiple of 128: every pair of blocks a decode group asks for, in all chunks of four."""
    for k in range(128, 32768 + 1, 128):
        k_blocks = k // 64
        for chunk in range((k_blocks + 3) // 4):
            for kb in (chunk * 4, chunk * 4 + 2):
                at = lib.pair_in_row(kb, k_blocks)
                assert at % 2 == 0 and 0 <= at and at + 2 <= k_blocks, (k, kb, at)
                assert at == kb or kb >= k_blocks
