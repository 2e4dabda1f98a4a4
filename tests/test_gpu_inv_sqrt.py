"""The reciprocal square root of the LTS solve (inv_sqrt in tfm.cuh) against CUDA's
double-precision 1 / sqrt, over its stated range.

Two Newton steps from rsqrtf's value (2 units in the last place: 2^-22, squared
twice) leave the roundings of the last step, 1.5 x 2^-53 relative; 1 / sqrt has two
of 2^-53.  They may differ by 3.5 x 2^-53; the bound is 4 x 2^-53.
"""
import subprocess

import pytest

from mirorr_b200 import build as mb_build

pytestmark = pytest.mark.gpu

SRC = r'''
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "tfm.cuh"

__global__ void both(const double *x, double *a, double *b, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    a[i] = mb2::inv_sqrt(x[i]);
    b[i] = 1.0 / sqrt(x[i]);
  }
}

int main() {
  std::mt19937_64 rng(1);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  std::vector<double> x = {1e-36, 1e36, 0.5, 1.0, 2.0, 4.0, std::nextafter(1.0, 0.0),
                           std::nextafter(1.0, 2.0), std::nextafter(4.0, 0.0), 4e-36, 8.0};
  while (x.size() < (1u << 21)) {
    x.push_back(std::pow(10.0, 72.0 * u(rng) - 36.0));  // the whole range
    x.push_back(0.5 + 0.5 * u(rng));                    // the half-angle's cosine
    x.push_back(std::ldexp(1.0 + u(rng) * 1e-6, (int)(rng() % 200) - 100));
  }
  const int n = (int)x.size();
  double *d = nullptr;
  std::vector<double> a(n), b(n);
  if (cudaMalloc(&d, sizeof(double) * 3 * n) != cudaSuccess) return 2;
  cudaMemcpy(d, x.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
  both<<<296, 256>>>(d, d + n, d + 2 * n, n);
  cudaMemcpy(a.data(), d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(b.data(), d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  if (cudaGetLastError() != cudaSuccess) return 2;
  double worst = 0.0, at = 0.0;
  for (int i = 0; i < n; ++i) {
    const double e = std::fabs(a[i] - b[i]) / b[i];
    if (!(e <= worst)) { worst = e; at = x[i]; }
  }
  std::printf("%.3g x 2^-53 at %.17g\n", std::ldexp(worst, 53), at);
  cudaFree(d);
  return worst <= std::ldexp(4.0, -53) ? 0 : 1;
}
'''


def test_against_cuda(tmp_path):
    src, exe = tmp_path / "inv_sqrt.cu", tmp_path / "inv_sqrt"
    src.write_text(SRC)
    subprocess.check_call([mb_build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3",
                           "-std=c++17", "--expt-relaxed-constexpr", "-I", mb_build.SRC, str(src),
                           "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
