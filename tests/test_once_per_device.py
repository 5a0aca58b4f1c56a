"""The opt-in to large shared memory is made once per kernel and device, however many kernels there are."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include "once_per_device.cuh"
int main() {
  static char kernels[300];
  dil::OncePerDevice table;
  for (int pass = 0; pass < 2; ++pass)
    for (int k = 0; k < 300; ++k)
      for (int dev : {0, 7, 63}) {
        if (table.done(kernels + k, dev) != (pass == 1)) return 1;
        table.set(kernels + k, dev);
      }
  if (table.done(kernels, 1) || table.done(kernels, -1) || table.done(kernels, 64)) return 2;
  table.set(kernels, 64);
  return table.done(kernels, 64) ? 3 : 0;
}
"""


def test_three_hundred_kernels(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    csrc = os.path.join(ROOT, "dilution-attention_b200", "csrc")
    subprocess.run([cxx, "-std=c++17", "-I", csrc, "-o", str(exe), str(tmp_path / "main.cpp"), "-pthread"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_the_launchers_use_it():
    text = open(os.path.join(ROOT, "dilution-attention_b200", "csrc", "tc_kernels.cuh")).read()
    body = text[text.index("inline int set_smem_attr("):]
    assert "OncePerDevice" in body[:body.index("\n}\n")]
