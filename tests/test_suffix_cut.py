"""How the fused shared-prefix kernel cuts a request's own tokens into pieces (csrc/suffix_cut.cuh), built for the host."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "single_gpu_inference_lab_b200/csrc"
SHIM = """
#include "suffix_cut.cuh"
extern "C" void cut(int pairs, int slots, int* out) {
  const pfd::SuffixCut c = pfd::suffix_cut(pairs, slots);
  out[0] = c.pieces; out[1] = c.pairs;
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("suffix_cut")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ftrapv", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "shim.so"), str(d / "shim.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "shim.so"))

    def call(pairs, slots):
        out = (ctypes.c_int * 2)()
        lib.cut(pairs, slots, out)
        return tuple(out)

    return call


def test_the_pieces_cover_the_pairs_within_the_slots(cut):
    big = 2**31 // 32
    for pairs in (*range(0, 70), 255, 256, 257, 4097, big - 1, big):
        for slots in (1, 2, 3, 4, 7, 16, 25, 1000, 2**31 - 1):
            pieces, each = cut(pairs, slots)
            assert 0 <= pieces <= slots
            assert pieces * each >= pairs
            if pairs == 0:
                assert pieces == 0
            else:
                assert (pieces - 1) * each < pairs  # the last piece has work, so every piece's first token is a live one
                assert each >= min(2, pairs)
