"""A structured stage refuses a grouping of the nonzeros that was not built (GPU). The core is zero, so that the stage
would have nothing to read from the missing arrays."""
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "sparse_a.cuh"
using namespace ttgb;
int main() {
  const int64_t s = 2, m = 3, n = 4, S = 2;
  double *core, *in, *out;
  if (cudaMalloc((void**)&core, 48 * 8) || cudaMemset(core, 0, 48 * 8) || cudaMalloc((void**)&in, 4096) ||
      cudaMalloc((void**)&out, 4096))
    return 2;
  SparseCore c;
  c.build(core, s, m, n, S, nullptr, SparseCore::kLp);
  const StageDims g{1, 1, 1, 1, 1, 1, 1};
  if (!c.use) return 3;
  sparse_stage(c.lp, in, out, g, nullptr);   // built
  int refused = 0;
  for (const SparseCsr* q : {&c.fw, &c.bk, &c.rh})
    try {
      sparse_stage(*q, in, out, g, nullptr);
    } catch (const Error& e) {
      refused += e.status == kInvalidArgument;
    }
  if (cudaDeviceSynchronize()) return 4;
  std::printf("refused %d\n", refused);
  return 0;
}
"""


def test_unbuilt_groupings_are_refused(cuda, tmp_path):
    from torchtt_gb300 import build
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + build.FLAGS + ["-cudart", "shared", "-I" + build.CSRC, str(src),
                   "-o", str(exe), build.LIB, "-Xlinker", "-rpath=" + build.HERE], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (out.returncode, out.stdout) == (0, "refused 3\n")
