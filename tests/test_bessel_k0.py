"""K0 of the atom windows on the CPU, against the same integral with a step four times finer in
long double (exact to its rounding).

Bound, in half roundings of a double (2^-53): x + 1/2 from rounding the arguments x cosh u (their
mean under the integrand), about two from the exponentials and the last product, up to five from
adding some thirty terms."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include "msx_bessel.cuh"
#include <cstdio>
int main() {
  static const msx::CoshTable t{};
  for (int i = 0; i <= 20000; ++i) {
    const double x = 0.1 * pow(300.0, i / 20000.0);
    long double sum = 0.5L * expl(-(long double)x);
    for (int k = 1; k < 300; ++k) sum += expl(-(long double)x * coshl(k / 32.0L));
    sum /= 32;
    const double err = fabs((double)((msx::bessel_k0(x, t.v) - sum) / sum));
    if (err > (x + 8) * ldexp(1.0, -53)) return printf("x %.6f error %.3e\n", x, err), 1;
  }
  return 0;
}
'''


def test_k0(tmp_path):
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc not found')
    src, exe = tmp_path / 'k0.cu', tmp_path / 'k0'
    src.write_text(SRC)
    r = subprocess.run([nvcc, '-std=c++17', '-O2', '-w', '-I', os.path.join(ROOT, 'namsa_gb300', 'csrc'), str(src),
                        '-o', str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
