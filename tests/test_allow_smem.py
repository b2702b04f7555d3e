"""The opt-in to more than 48 KB of shared memory holds for one device: it is made once on every
device that a kernel runs on, and again after an error. The function is compiled alone, against
stand-ins for the two calls that it makes."""
import os
import re
import shutil
import subprocess

import pytest

from mormot2_ai_b200.csrc import build

MAIN = r"""
#include <cassert>
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
static int device, set_calls, fail;
static cudaError_t cudaGetDevice(int* d) { *d = device; return 0; }
static cudaError_t cudaFuncSetAttribute(const void*, int, int) { ++set_calls; return fail; }
%s
int main() {
  unsigned long long done = 0;
  const int order[] = {0, 0, 1, 0, 1, 7, 7, 63, 63}, calls[] = {1, 1, 2, 2, 2, 3, 3, 4, 4};
  for (int i = 0; i < 9; ++i) {
    device = order[i];
    assert(mb_allow_smem(0, 1, &done) == 0 && set_calls == calls[i]);
  }
  device = 64;      // beyond the bits: asked for every time
  for (int i = 1; i < 3; ++i) assert(mb_allow_smem(0, 1, &done) == 0 && set_calls == 4 + i);
  device = 2, fail = 5;
  for (int i = 1; i < 3; ++i) assert(mb_allow_smem(0, 1, &done) == 5 && set_calls == 6 + i);
  fail = 0;
  assert(mb_allow_smem(0, 1, &done) == 0 && set_calls == 9);
  assert(mb_allow_smem(0, 1, &done) == 0 && set_calls == 9);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_once_a_device(tmp_path):
    text = open(os.path.join(build.HERE, "common.cuh")).read()
    function = re.search(r"static inline cudaError_t mb_allow_smem\(.*?\n}\n", text, re.S).group()
    source, program = tmp_path / "main.cpp", tmp_path / "main"
    source.write_text(MAIN % function)
    subprocess.run(["g++", "-o", str(program), str(source)], check=True)
    subprocess.run([str(program)], check=True)
