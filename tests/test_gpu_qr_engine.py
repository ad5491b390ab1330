"""QR under the double-float engine of the mixed path (GPU): matrices below 1024 rows with m n^2 < 4e5, and wide
ones, are factored with FP64 products whatever the engine, so that Q is orthonormal to rounding."""
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "contract.cuh"
#include "linalg.cuh"
using namespace ttgb;
int main() {
  const int sizes[][2] = {{600, 16}, {1000, 19}, {300, 33}, {200, 44}, {73, 73}, {48, 200}, {100, 130}, {160, 170}};
  double* part; unsigned* counter; int *status, *host;
  if (cudaMalloc((void**)&part, 8 * 1024 * 128) || cudaMalloc((void**)&counter, 64) || cudaMemset(counter, 0, 64) ||
      cudaMalloc((void**)&status, 16) || cudaMemset(status, 0, 16) || cudaMallocHost((void**)&host, 16))
    return 2;
  RedWS red;
  red.partial = part; red.counter = counter; red.cap_blocks = 1024; red.cap_vec = 127;
  for (const auto& z : sizes)
    for (int tuned = 0; tuned < 2; ++tuned) {
      set_autotune(tuned);
      const int m = z[0], n = z[1], k = m < n ? m : n;
      std::vector<double> a((size_t)m * n), q((size_t)m * k);
      for (double& v : a) v = std::rand() / (double)RAND_MAX - 0.5;
      double *A, *Q, *R;
      if (cudaMalloc((void**)&A, a.size() * 8) || cudaMalloc((void**)&Q, q.size() * 8) ||
          cudaMalloc((void**)&R, (size_t)k * n * 8) || cudaMemcpy(A, a.data(), a.size() * 8, cudaMemcpyHostToDevice))
        return 3;
      LinalgWS ws;
      ws.status = status; ws.h_status = host;
      {
        Fp64EngineScope df(kFp64DoubleFloat);
        qr(A, m, m, n, Q, R, ws, red, nullptr);
      }
      if (cudaMemcpy(q.data(), Q, q.size() * 8, cudaMemcpyDeviceToHost)) return 4;
      double s = 0.0;
      for (int i = 0; i < k; ++i)
        for (int j = 0; j < k; ++j) {
          double t = i == j ? -1.0 : 0.0;
          for (int r = 0; r < m; ++r) t += q[(size_t)i * m + r] * q[(size_t)j * m + r];
          s += t * t;
        }
      std::printf("%d %d %.3e\n", m, n, std::sqrt(s));
      cudaFree(A); cudaFree(Q); cudaFree(R);
    }
  return 0;
}
"""


def test_small_and_wide_factors_stay_fp64(cuda, tmp_path):
    from torchtt_gb300 import build
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + build.FLAGS + ["-cudart", "shared", "-I" + build.CSRC, str(src),
                   "-o", str(exe), build.LIB, "-Xlinker", "-rpath=" + build.HERE], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0
    rows = [line.split() for line in out.stdout.splitlines()]
    assert len(rows) == 16
    for m, n, err in rows:
        # norms and inner products of k columns within a few roundings each: FP64 products give 1.6 to 3.1
        # sqrt(k) 2^-52, Householder reflections up to 3.8, double-float products up to 5.5
        assert float(err) <= 4 * min(int(m), int(n)) ** 0.5 * 2.0 ** -52, (m, n, err)
