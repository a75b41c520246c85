"""Which shared-prefix calls the fused kernel takes (csrc/suffix_cut.cuh, fused_pays), built for the host."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "single_gpu_inference_lab_b200/csrc"
SHIM = """
#include "suffix_cut.cuh"
extern "C" int pays(const int64_t* x) {
  return pfd::fused_pays(pfd::FusedShape{x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7] != 0}, 148);
}
"""


@pytest.fixture(scope="module")
def pays(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fused_rule")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ftrapv", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "shim.so"), str(d / "shim.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "shim.so"))

    def call(batch, q_heads, kv_heads, prefix, own, split, alone=0, grouped=False):
        shape = (batch, q_heads // kv_heads, kv_heads, -(-prefix // 256), max(1, -(-own // split)), own, alone, grouped)
        return bool(lib.pays((ctypes.c_int64 * 8)(*shape)))

    return call


def test_a_long_context_in_no_group_is_left_to_the_two_kernels(pays):
    """Its slots are few and a piece is one warp's: hardly more than half as long as the tiles take, no longer."""
    assert pays(64, 16, 2, 5120, 512, 128, alone=5632, grouped=True)
    for context in (16384, 32768, 131072, 2**31 - 16):
        assert not pays(64, 16, 2, 5120, 512, 128, alone=context, grouped=True)
    assert not pays(64, 16, 2, 256, 16, 64, alone=4096, grouped=True)
    assert not pays(12, 32, 8, 256, 16, 64, alone=4000, grouped=True)


@pytest.mark.parametrize("q_heads,kv_heads", [(16, 2), (28, 4), (32, 8)])
def test_own_tokens_that_outweigh_the_tiles_are_left_to_the_two_kernels(pays, q_heads, kv_heads):
    assert pays(128, q_heads, kv_heads, 8192, 512, 128)
    assert not pays(64, q_heads, kv_heads, 256, 2048, 512)
    assert not pays(16, q_heads, kv_heads, 256, 8192, 512)
    # the longer the own tokens of a call whose prefix is long, the less: none is taken beyond one that is not
    for prefix in (256, 1024, 4096, 8192):
        for batch in (8, 64, 256):
            for grouped, alone in ((False, 0), (True, 0), (True, 400)):
                taken = [pays(batch, q_heads, kv_heads, prefix, own, own, alone=alone, grouped=grouped) for own in range(64, 8192, 64)]
                assert taken[taken.index(True):] == sorted(taken[taken.index(True):], reverse=True) if True in taken else True


# (batch, q heads, kv heads, prefix, own tokens, split, longest context if some may be in no group): us with the two kernels, fused
MEASURED = [
    ((64, 16, 2, 4096, 512, 128, 0), 15.6, 16.4),
    ((16, 16, 2, 8192, 1024, 256, 0), 14.6, 17.4),
    ((8, 8, 8, 2048, 1024, 256, 0), 12.8, 17.2),
    ((64, 8, 1, 4096, 1024, 256, 0), 13.8, 18.9),
    ((128, 8, 8, 2048, 128, 64, 0), 18.4, 21.5),
    ((128, 16, 2, 8192, 512, 256, 0), 50.9, 48.4),
    ((256, 32, 16, 4096, 128, 64, 0), 130.0, 87.0),
    ((64, 16, 2, 4096, 512, 128, 4608), 21.8, 18.7),
    ((64, 16, 2, 5120, 512, 128, 5632), 28.2, 23.3),
    ((256, 28, 4, 4096, 16, 64, 4112), 107.0, 92.4),
    ((256, 16, 2, 320, 128, 64, 448), 22.8, 25.9),
]


@pytest.mark.parametrize("shape,two_kernels,fused", MEASURED)
def test_the_rule_takes_the_faster_side_of_what_was_measured(pays, shape, two_kernels, fused):
    batch, q_heads, kv_heads, prefix, own, split, alone = shape
    assert pays(batch, q_heads, kv_heads, prefix, own, split, alone=alone, grouped=alone > 0) == (fused < two_kernels)


def test_the_largest_call_stays_within_64_bits(pays):
    assert not pays(2048, 8, 2**20, 256, 2**31 - 16, 16, alone=2**31 - 16, grouped=True)
