"""How many of a request's own tokens the fused shared-prefix kernel attends (csrc/suffix_cut.cuh), built for the host:
never a page beyond the block-table row, whatever the lengths on the device say."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "single_gpu_inference_lab_b200/csrc"
SHIM = """
#include "suffix_cut.cuh"
extern "C" int own(int seq_len, int kv0, int cols, int splits, int split_size) {
  return pfd::own_length(seq_len, kv0, cols, splits, split_size);
}
"""


@pytest.fixture(scope="module")
def own(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("own_length")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ftrapv", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "shim.so"), str(d / "shim.cpp")],
                   check=True)
    return ctypes.CDLL(str(d / "shim.so")).own


@pytest.mark.parametrize("max_seq_len", [16, 17, 300, 4096, 4608, 131072, 2**31 - 16])
def test_own_tokens_stay_inside_the_block_table_row(own, max_seq_len):
    cols = -(-max_seq_len // 16)
    for kv0 in {k for k in (0, 16, 256, 4096, max_seq_len // 16 * 16) if k <= max_seq_len}:
        for splits, size in ((0, 64), (1, 16), (1, 512), (4, 128), (9, 64), (1000, 2**20)):
            for seq_len in (0, 1, kv0, kv0 + 1, max_seq_len - 1, max_seq_len, cols * 16, cols * 16 + 1, kv0 + splits * size, 2**31 - 1):
                seq_len = min(seq_len, 2**31 - 1)
                live = own(seq_len, kv0, cols, splits, size)
                assert 0 <= live <= max(seq_len - kv0, 0)
                assert live == 0 or (kv0 + live - 1) // 16 < cols
                # a request within the caller's bounds loses nothing
                if seq_len <= max_seq_len and (splits == 0 or seq_len - kv0 <= splits * size):
                    assert live == max(seq_len - kv0, 0)
