"""Register codelets and the two-stage line schedules on the CPU against a direct DFT.

Each transform is within a few float32 roundings per butterfly level: the bound
5e-7 on the relative L2 error is the one of the schedule check in
tests/fft_host_check.cu (measured errors are about 2e-7)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include "msx_fft.cuh"
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
using namespace msx;
static double error(const std::vector<float2>& x, const std::vector<float2>& y, bool inv) {
  const int n = (int)x.size();
  double num = 0, den = 0;
  for (int k = 0; k < n; ++k) {
    double re = 0, im = 0;
    for (int j = 0; j < n; ++j) {
      const double a = (inv ? 2 : -2) * M_PI * double((long)j * k % n) / n;
      re += x[j].x * cos(a) - x[j].y * sin(a);
      im += x[j].x * sin(a) + x[j].y * cos(a);
    }
    num += (y[k].x - re) * (y[k].x - re) + (y[k].y - im) * (y[k].y - im);
    den += re * re + im * im;
  }
  return sqrt(num / den);
}
template <int R, bool INV> double codelet(std::mt19937& g) {
  std::uniform_real_distribution<float> u(-1, 1);
  std::vector<float2> x(R), y(R);
  for (auto& e : x) e = make_float2(u(g), u(g));
  float2 v[R];
  for (int i = 0; i < R; ++i) v[i] = x[i];
  Dft<R, INV>::run(v);
  for (int i = 0; i < R; ++i) y[i] = v[i];
  return error(x, y, INV);
}
template <int R> double both(std::mt19937& g) {
  const double e = fmax(codelet<R, false>(g), codelet<R, true>(g));
  printf("radix %d: %.2e\n", R, e);
  return e;
}
template <int N, int T, int... Rs> double line(std::mt19937& g) {
  using F = LineFFT<N, T, Radices<Rs...>>;
  std::vector<float2> tw(F::tw_words() + 1), x(N), y;
  F::host_twiddles(tw.data());
  std::uniform_real_distribution<float> u(-1, 1);
  for (auto& e : x) e = make_float2(u(g), u(g));
  y = x;
  F::template host_run<false>(y.data(), tw.data());
  double w = error(x, y, false);
  y = x;
  F::template host_run<true>(y.data(), tw.data());
  w = fmax(w, error(x, y, true));
  printf("line %d: %.2e\n", N, w);
  return w;
}
int main() {
  std::mt19937 g(7);
  double w = 0;
  for (double e : {both<2>(g), both<3>(g), both<4>(g), both<6>(g), both<8>(g), both<12>(g), both<16>(g), both<24>(g),
                   both<32>(g), both<48>(g)})
    w = fmax(w, e);
  w = fmax(w, line<768, 16, 48, 16>(g));
  w = fmax(w, line<384, 8, 48, 8>(g));
  return w < 5e-7 ? 0 : 1;
}
'''


def test_codelets_match_a_direct_dft(tmp_path):
    nvcc = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'
    if not os.path.exists(nvcc):
        pytest.skip('nvcc not found')
    src, exe = tmp_path / 'codelets.cu', tmp_path / 'codelets'
    src.write_text(SRC)
    r = subprocess.run([nvcc, '-std=c++17', '-O1', '-w', '-I', os.path.join(ROOT, 'namsa_gb300', 'csrc'), str(src),
                        '-o', str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
