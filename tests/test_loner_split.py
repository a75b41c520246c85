"""How a grouped shared-prefix decode cuts up the requests in no group: the arithmetic of launch and kernels
(csrc/loner_split.cuh), built for the host, at bounds far beyond what a test could allocate."""

import ctypes
import itertools
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "single_gpu_inference_lab_b200/csrc"
SHIM = """
#include "loner_split.cuh"
extern "C" void split(long long max_seq_len, long long slots, long long ns, long long kv_heads, long long sms, int loners, int* out) {
  const pfd::LonerGrid g = pfd::loner_grid(max_seq_len, slots, ns, kv_heads, sms);
  const int size = pfd::loner_split_size(g, loners);
  out[0] = g.rows; out[1] = g.least; out[2] = size; out[3] = pfd::loner_split_count(g, size);
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("loner_split")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ftrapv", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "shim.so"), str(d / "shim.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "shim.so"))

    def call(max_seq_len, slots, ns, kv_heads, sms, loners):
        out = (ctypes.c_int * 4)()
        lib.split(*(ctypes.c_longlong(x) for x in (max_seq_len, slots, ns, kv_heads, sms)), loners, out)
        return list(out)

    return call


@pytest.mark.parametrize("max_seq_len", [0, 1, 15, 255, 256, 257, 4000, 5632, 131072, 1 << 19, 1 << 20, (1 << 20) + 5, (1 << 30) + 1, (1 << 31) - 16])
def test_every_split_lies_inside_the_bound_on_the_lengths(split, max_seq_len):
    for prefix, suffix, split_size in ((4096, 512, 128), (1 << 20, 1 << 20, 512), (1 << 20, 4096, 64), (256, 40, 64), (0, 100, 512)):
        chunks = -(-min(prefix, max_seq_len) // 256)
        ns = max(-(-min(suffix, max_seq_len) // split_size), 1)
        slots = chunks + ns
        for kv_heads, sms, loners in itertools.product((1, 2, 8, 32), (74, 148), (0, 1, 2, 8, 32, 64, 128, 1776, 2048)):
            rows, least, size, count = split(max_seq_len, slots, ns, kv_heads, sms, loners)
            what = f"max={max_seq_len} slots={slots} ns={ns} heads={kv_heads} sms={sms} loners={loners}: {rows} {least} {size} {count}"
            assert 3 * sms <= rows * ns * kv_heads < 3 * sms + ns * kv_heads, what
            assert size >= least >= 256 and size % 16 == 0, what
            assert 1 <= count <= slots and (count - 1) * size < max(max_seq_len, 1) <= max(count * size, 1), what  # the first token of the last split
            assert loners * kv_heads * count < 1 << 31, what  # items
            # the work of the requests is spread over the CTAs: size x items a head, at most some twice what an even share is
            if size > least and size < max_seq_len <= 1 << 21:
                assert size <= loners * (max_seq_len * kv_heads // (rows * ns * kv_heads)) + 63, what
                assert loners * kv_heads * count <= 3 * rows * ns * kv_heads + loners * kv_heads, what


def test_splits_at_sizes_whose_product_left_32_bits(split):
    """(Splits counted for the smallest size, the size that follows from the number of requests: 4096 x 599168 and the like.)"""
    for max_seq_len, kv_heads, loners in ((1 << 20, 8, 32), (1 << 20, 8, 64), (1 << 19, 8, 128), (131072, 8, 2048)):
        chunks, ns = max_seq_len // 256, max_seq_len // 512
        _, _, size, count = split(max_seq_len, chunks + ns, ns, kv_heads, 148, loners)
        assert count == -(-max_seq_len // size) and (count - 1) * size < max_seq_len
