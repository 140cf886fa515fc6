"""Shared memory above 48 KB is allowed once on every device (csrc/grants.h), and every launcher asks through that one place."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

from sleuth_b200.kernels.library import CSRC, find_nvcc

PROGRAM = r"""
#include "grants.h"
#include <initializer_list>
static int device, asked[70], refuse;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  if (refuse) return cudaErrorInvalidValue;
  ++asked[device];
  return cudaSuccess;
}
int main() {
  static std::atomic<unsigned long long> one, other;
  for (int turn = 0; turn < 3; ++turn)
    for (int d : {0, 1, 63}) { device = d; if (slb::allow_shared(nullptr, 65536, one) != cudaSuccess) return 1; }
  if (asked[0] != 1 || asked[1] != 1 || asked[63] != 1) return 2;
  device = 5; refuse = 1;
  if (slb::allow_shared(nullptr, 65536, one) == cudaSuccess) return 3;
  refuse = 0;                                      // a refusal is not remembered, and no kernel has another's grant
  if (slb::allow_shared(nullptr, 65536, one) != cudaSuccess || asked[5] != 1) return 4;
  if (slb::allow_shared(nullptr, 65536, other) != cudaSuccess || asked[5] != 2) return 5;
  device = 64;                                     // beyond the word: asked every time
  slb::allow_shared(nullptr, 65536, one); slb::allow_shared(nullptr, 65536, one);
  return asked[64] == 2 ? 0 : 6;
}
"""


def test_allowed_once_per_device(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    include = Path(find_nvcc()).resolve().parent.parent / "include"
    (tmp_path / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(include), str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")], check=True)
    assert subprocess.run([str(tmp_path / "p")]).returncode == 0


def test_no_launcher_keeps_a_flag_of_its_own():
    for f in sorted(CSRC.iterdir()):
        if f.name != "grants.h":
            assert not re.search(r"cudaFuncSetAttribute\s*\(", f.read_text()), f.name
