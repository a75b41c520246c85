"""A build in which the fused shared-prefix kernel came out with other registers than its warps share out sends every call to
the two kernels, which need no such number (csrc/suffix_cut.cuh, fused_takes; built for the host)."""

import ctypes
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "single_gpu_inference_lab_b200/csrc"
SHIM = """
#include "suffix_cut.cuh"
static int asked = 0;
extern "C" int times_asked() { return asked; }
extern "C" int takes(int regs, int own) {
  return pfd::fused_takes(pfd::FusedShape{128, 8, 2, 32, 2, own, 0, false}, 148, [regs] { ++asked; return regs; });
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("fused_registers")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def test_other_registers_leave_the_call_to_the_two_kernels(shim):
    assert [r for r in range(0, 256) if shim.takes(r, 512)] == list(range(89, 97))  # (handed out in eights)


def test_a_call_that_would_not_take_the_kernel_does_not_load_it(shim):
    before = shim.times_asked()
    assert not shim.takes(96, 65536)
    assert shim.times_asked() == before


def test_the_register_shares_add_up_to_the_launch():
    source = (CSRC / "shared_prefix_fused.cuh").read_text()
    up, = re.findall(r"setmaxnreg\.inc\.sync\.aligned\.u32 (\d+);", source)
    down, = re.findall(r"setmaxnreg\.dec\.sync\.aligned\.u32 (\d+);", source)
    regs, = re.findall(r"constexpr int kFusedRegs = (\d+);", (CSRC / "suffix_cut.cuh").read_text())
    assert 4 * int(down) + int(up) == 5 * int(regs)  # four warpgroups of dense warps, one of the others


def test_launching_the_fused_kernel_refuses_no_call_for_its_registers():
    source = (CSRC / "paged_decode_abi.cu").read_text()
    body = source[source.index("int launch_fused("):source.index("int launch_decode(")]
    assert "numRegs" in body and not re.search(r"fail\([^;]*numRegs", body)
