"""A kernel that hands registers from one warpgroup to others is not launched if the compiler gave it fewer than the split needs:
the increase would wait for ever.  The launchers' check, against a fake of the CUDA runtime."""

from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "dilution-attention_b200", "csrc")

HEAD = r"""
#include <cstdio>
#include "once_per_device.cuh"
using dil::OncePerDevice;
enum cudaError_t { cudaSuccess = 0, cudaErrorFake = 1 };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize };
struct cudaFuncAttributes { int numRegs; };
static int regs_built, fail_attributes, opt_ins;
static cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
static cudaError_t cudaFuncSetAttribute(const void*, int, int) { ++opt_ins; return cudaSuccess; }
static cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  a->numRegs = regs_built;
  return fail_attributes ? cudaErrorFake : cudaSuccess;
}
static const char* cudaGetErrorString(cudaError_t) { return "fake"; }
"""

MAIN = r"""
int main() {
  char err[256], few = 0, enough = 0, none = 0;
  regs_built = 88;
  for (int i = 0; i < 2; ++i)
    if (set_smem_attr(&few, 1024, err, sizeof err, 96) == 0) return 1;        // refused, and again
  if (opt_ins) return 2;
  regs_built = 96;
  if (set_smem_attr(&few, 1024, err, sizeof err, 96) || set_smem_attr(&enough, 1024, err, sizeof err, 96)) return 3;
  fail_attributes = 1;
  if (set_smem_attr(&none, 1024, err, sizeof err, 96) == 0) return 4;
  if (set_smem_attr(&none, 1024, err, sizeof err)) return 5;                  // no split: not asked
  return opt_ins == 3 ? 0 : 6;
}
"""


def _text(name):
    return open(os.path.join(CSRC, name)).read()


def test_a_build_with_too_few_registers_is_refused(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    body = _text("tc_kernels.cuh")
    body = body[body.index("inline int set_smem_attr("):]
    (tmp_path / "main.cpp").write_text(HEAD + body[:body.index("\n}\n") + 3] + MAIN)
    exe = tmp_path / "main"
    subprocess.run([cxx, "-std=c++17", "-I", CSRC, "-o", str(exe), str(tmp_path / "main.cpp"), "-pthread"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_every_launch_of_a_split_asks():
    """Kernels with a register split, and how many of their launches there are."""
    kernels = {"tc_fused_forward.cuh": "kFusedRegs", "tc_kernels.cuh": "kBwdRegs", "tc_wide_kernels.cuh": "kBwdRegs"}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cuh") and "setmaxnreg.inc" in _text(name):
            assert name in kernels, name
    for name, launches in (("tc_fused_forward.cuh", 1), ("tc_kernels.cuh", 1), ("tc_wide_kernels.cuh", 3)):
        asks = re.findall(r"set_smem_attr\(\(const void\*\)\w[^;]*" + kernels[name] + r"[^;]*;", _text(name))
        assert len(asks) == launches, (name, asks)


def test_the_reverse_pass_in_slices_asks_too():
    """tc_kernels.cuh has a second kernel with a split, and one launch of it; no third."""
    text = _text("tc_kernels.cuh")
    assert len(re.findall(r"set_smem_attr\(\(const void\*\)\w[^;]*kSliceRegs[^;]*;", text)) == 1
    assert text.count("setmaxnreg.inc") == 2 and "static_assert(4 * 104 + 64 <= 5 * kSliceRegs" in text
