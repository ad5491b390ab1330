"""Reciprocal square roots from the FP32 one (GPU) against 1 / sqrt over all exponents and the values where there is
none. Two roundings of an operand near 1 and the last one: within 2^-52."""
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "rsqrt.cuh"
__global__ void all_kernel(const double* d, int n, double* full, double* refined) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  full[i] = ttgb::rsqrt_full(d[i]);
  refined[i] = ttgb::rsqrt_refined(d[i]);
}
int main() {
  std::vector<double> d;
  std::mt19937_64 g(1);
  for (int e = 1; e < 2047; ++e)
    for (int q = 0; q < 256; ++q) {
      const unsigned long long frac = q == 0 ? 0ull : q == 1 ? (1ull << 52) - 1 : g() >> 12;
      const unsigned long long b = (unsigned long long)e << 52 | frac;
      double v;
      std::memcpy(&v, &b, 8);
      d.push_back(v);
    }
  const int normal = (int)d.size();
  for (double v : {0.0, -0.0, 4.9406564584124654e-324, 1e-310, (double)INFINITY, -1.0, (double)NAN}) d.push_back(v);
  const int n = (int)d.size();
  double* p;
  if (cudaMalloc((void**)&p, 3 * n * 8) || cudaMemcpy(p, d.data(), n * 8, cudaMemcpyHostToDevice)) return 2;
  all_kernel<<<(n + 255) / 256, 256>>>(p, n, p + n, p + 2 * n);
  std::vector<double> r(2 * n);
  if (cudaMemcpy(r.data(), p + n, 2 * n * 8, cudaMemcpyDeviceToHost)) return 3;
  double worst[2] = {0, 0};
  for (int i = 0; i < normal; ++i) {
    const long double ref = 1.0L / sqrtl((long double)d[i]);
    worst[0] = std::fmax(worst[0], (double)(fabsl(r[i] - ref) / ref));
    if (d[i] >= 1.1754943508222875e-38 && d[i] <= 1.7e38)
      worst[1] = std::fmax(worst[1], (double)(fabsl(r[n + i] - ref) / ref));
  }
  int same = 0;
  for (int i = normal; i < n; ++i) {
    const double ref = 1.0 / std::sqrt(d[i]);
    same += std::isnan(ref) ? std::isnan(r[i]) : r[i] == ref;
  }
  std::printf("%.4e %.4e %d %d\n", worst[0], worst[1], same, n - normal);
  return 0;
}
"""


def test_all_exponents(cuda, tmp_path):
    from torchtt_gb300 import build
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + build.FLAGS + ["-I" + build.CSRC, str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out
    full, refined, same, others = out.stdout.split()
    assert float(full) <= 2.0 ** -52 and float(refined) <= 2.0 ** -52 and same == others
