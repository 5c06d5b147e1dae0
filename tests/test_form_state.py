"""Optional kernel forms on the CPU: a device that refuses one is asked once, the plan does
without it, and no error stays behind.  The refusal is a fake's error code."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include "msx_form.h"
#include <cstdio>
int main() {
  int asked = 0;
  msx::FormState refused, taken;
  for (int i = 0; i < 3; ++i)
    if (refused.ready([&] { ++asked; return cudaErrorInvalidConfiguration; })) return printf("taken\n"), 1;
  if (asked != 1 || refused.state != -1) return printf("asked %d times\n", asked), 1;
  for (int i = 0; i < 3; ++i)
    if (!taken.ready([&] { ++asked; return cudaSuccess; })) return printf("refused\n"), 1;
  if (asked != 2 || taken.state != 1) return printf("asked again\n"), 1;
  return 0;
}
'''


def test_refusal_is_remembered(tmp_path):
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc not found')
    src, exe = tmp_path / 'form.cu', tmp_path / 'form'
    src.write_text(SRC)
    r = subprocess.run([nvcc, '-std=c++17', '-O1', '-w', '-I', os.path.join(ROOT, 'namsa_gb300', 'csrc'), str(src),
                        '-o', str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

