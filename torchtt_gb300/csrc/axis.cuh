// An index i = i1 e0 + i0 with address offset i1 s1 + i0 s0, as the GEMM kernels take it (struct Ax of contract.cuh with
// a 32-bit inner extent).
#pragma once

#include <cstdint>

namespace ttgb {

struct AxD {
  int e0 = 1 << 30;
  int64_t s1 = 0, s0 = 1;
};

#ifdef __CUDACC__
__device__ __forceinline__ int64_t ax_off(const AxD& a, int i) {
  const int i1 = i / a.e0;
  return (int64_t)i1 * a.s1 + (int64_t)(i - i1 * a.e0) * a.s0;
}

// Offsets of consecutive indexes: one division at the start.
struct AxWalk {
  int64_t off;
  int i0;
  __device__ __forceinline__ AxWalk(const AxD& a, int i) : off(ax_off(a, i)), i0(i % a.e0) {}
  __device__ __forceinline__ void next(const AxD& a) {
    off += a.s0;
    if (++i0 == a.e0) { i0 = 0; off += a.s1 - (int64_t)a.e0 * a.s0; }
  }
};
#endif

}  // namespace ttgb
