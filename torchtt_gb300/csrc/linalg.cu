// FP64 dense linear algebra: CholeskyQR with a Householder fallback, one-sided Jacobi thin SVD.
//
// GB300 note: FP64 runs at ~1.9 FMA/clock/SM (measured), so every O(m n^2) step is expressed as a
// GEMM on the contraction engine (spread over all SMs); only O(n^3) steps on the small n x n
// factors run on few SMs: Cholesky + triangular inverse in one block, the Jacobi of n < 16 in one
// warp, the block Jacobi of 16 <= n <= 160 on an 8-CTA cluster, larger ones one grid-wide round per
// launch, all from 16 on after FP32 sweeps in one block that leave them two or three sweeps. Small
// QRs (the kickrank-wide blocks) run all their passes in one block.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "contract.cuh"
#include "linalg.cuh"
#include "reduce.cuh"
#include "rsqrt.cuh"

namespace cg = cooperative_groups;

namespace ttgb {

namespace {

constexpr double kEps = 2.220446049250313e-16;

__device__ double block_sum_d(double v, double* sh) {
  v = red::warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += sh[i];
  __syncthreads();
  return r;   // valid in all threads
}

__device__ double block_max_d(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r = fmax(r, sh[i]);
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------------------------------------
// Cholesky of the symmetric n x n matrix G (row-major, in place -> upper R with G = R^T R).
// shift_rows > 0 adds the sCholQR3 shift 11 (m n + n (n+1)) eps ||A||_F^2 with m = shift_rows
// (Fukaya, Kannan, Nakatsukasa, Yamamoto, Yanagisawa, SIAM J. Sci. Comput. 2020).
// check_identity: flag status=2 when max |G - I| > 0.1 (the third pass of CholeskyQR3 sees the
// Gram matrix of an already orthonormalised Q).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(512) chol_kernel(double* G, int n, int64_t shift_rows,
                                                   int check_identity, int* status) {
  stream_wait();
  __shared__ double sh[32];
  __shared__ int bad;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) bad = 0;
  __syncthreads();
  if (check_identity) {
    double mx = 0.0;
    for (int64_t t = tid; t < (int64_t)n * n; t += nt) {
      const int i = (int)(t / n), k = (int)(t % n);
      if (k < i) continue;   // the Gram matrix is formed (and read) in its upper triangle only
      const double v = G[t] - (i == k ? 1.0 : 0.0);
      mx = fmax(mx, isfinite(v) ? fabs(v) : 1e300);
    }
    mx = block_max_d(mx, sh);
    if (tid == 0 && !(mx <= 0.1)) *status = 2;
  }
  if (shift_rows > 0) {
    double tr = 0.0;
    for (int i = tid; i < n; i += nt) tr += G[(int64_t)i * n + i];
    tr = block_sum_d(tr, sh);
    const double sft = 11.0 * ((double)shift_rows * n + (double)n * (n + 1)) * kEps * tr;
    for (int i = tid; i < n; i += nt) G[(int64_t)i * n + i] += sft;
  }
  __syncthreads();
  __shared__ double piv_inv;   // pivot reciprocal, computed once per step (see chol_inv_smem)
  for (int j = 0; j < n; ++j) {
    if (tid == 0) {
      const double d = G[(int64_t)j * n + j];
      if (!(d > 0.0) || !isfinite(d)) { bad = 1; *status = 1; }
      else { const double rd = sqrt(d); G[(int64_t)j * n + j] = rd; piv_inv = 1.0 / rd; }
    }
    __syncthreads();
    if (bad) break;
    const double inv = piv_inv;
    for (int k = j + 1 + tid; k < n; k += nt) G[(int64_t)j * n + k] *= inv;
    __syncthreads();
    const int w = n - j - 1;
    for (int64_t t = tid; t < (int64_t)w * w; t += nt) {
      const int i = j + 1 + (int)(t / w), k = j + 1 + (int)(t % w);
      if (k < i) continue;
      G[(int64_t)i * n + k] = fma(-G[(int64_t)j * n + i], G[(int64_t)j * n + k], G[(int64_t)i * n + k]);
    }
    __syncthreads();
  }
  __syncthreads();
  for (int64_t t = tid; t < (int64_t)n * n; t += nt) {
    const int i = (int)(t / n), k = (int)(t % n);
    if (k < i) G[t] = 0.0;
  }
}

// Fused, shared-memory resident Cholesky + triangular inverse for n <= kCholSmemMax, one block:
// G (row-major, global) -> R (upper, G = R^T R) to Rout, R^{-1} to Riout; one n x n array holds R in
// its upper and L^{-1} = R^{-T} in its strictly lower triangle.
//
// A column at a time, every step waits for a square root and a division and for three barriers, and
// that chain, not the n^3 / 3 multiply-adds, set the time (133 us at n = 77). By panels of 16 the chain
// runs over a 16 x 32 block [G_JJ | I] with one element per thread: row j is scaled by its warp (the
// reciprocal square root from FP32 with a correction of third order) and published, one barrier per
// step, which gives R_JJ and L_JJ^{-1}; the other columns of the panel's rows and the rows below are
// then two plain products.
//
// pass 0 factors without a shift first (condition of A up to ~1e5: the next pass then sees a matrix
// near the identity); a pivot below kPivotTol of the largest diagonal entry starts over with the shift
// of sCholQR3. pass 1 sets *done when its G is near enough to the identity that Q needs no third
// pass. pass 2 sets *status = 2 when max |G - I| > 0.1. Gin is cleared (the next Gram product
// accumulates into it); Rout and Riout must not overlap it.
constexpr int kCholSmemMax = 160;
constexpr int kCholNb = 16;
constexpr double kNearIdentity = 1e-9;   // max |G - I| below which the first-order factor is used
constexpr double kPivotTol = 1e-11;

// Largest |G - I| and largest diagonal entry of an upper triangle by their high words (upper bounds
// within 2^-20; 1e300 for an infinity or a NaN), and the trace. FP64 comparisons and block-wide FP64
// reductions would hold the FP64 pipe for microseconds; these are integer maxima.
struct GramStats {
  unsigned mx, dmax;
  double tr;
};

__device__ __forceinline__ double from_high_word(unsigned hi) {
  return hi >= 0x7ff00000u ? 1e300 : __hiloint2double((int)hi + 1, 0);
}

// All threads; st is cleared by the caller before a barrier, valid after the next one.
__device__ __forceinline__ void gram_stats(const double* g, int n, int pitch, bool identity, GramStats* st) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  unsigned mx = 0u, dmax = 0u;
  for (int t = tid; t < n * n; t += nt) {
    const int i = t / n, k = t - i * n;
    if (k < i) continue;
    const double v = g[i * pitch + k];
    if (i == k) dmax = max(dmax, (unsigned)__double2hiint(v));
    if (identity) mx = max(mx, (unsigned)__double2hiint(i == k ? v - 1.0 : v) & 0x7fffffffu);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  dmax = __reduce_max_sync(0xffffffffu, dmax);   // a negative diagonal entry counts as infinite
  if (lane == 0) {
    atomicMax(&st->mx, mx);
    atomicMax(&st->dmax, dmax);
  }
  if (tid < 32) {
    double tr = 0.0;
    for (int i = lane; i < n; i += 32) tr += g[i * pitch + i];
    tr = red::warp_sum(tr);
    if (lane == 0) st->tr = tr;
  }
}

// 2^-e, 2^(e/2) and 2^(-e/2) for the even e with 2^e <= d < 2^(e+2) (1 when d is not a normal number)
__device__ __forceinline__ void even_scale(double d, double& sc, double& root, double& inv_root) {
  int e = ((__double2hiint(d) >> 20) & 0x7ff) - 1023;
  if (!(d > 0.0) || d >= 1e300 || e < -1000) e = 0;
  e &= ~1;
  sc = __hiloint2double((1023 - e) << 20, 0);
  root = __hiloint2double((1023 + e / 2) << 20, 0);
  inv_root = __hiloint2double((1023 - e / 2) << 20, 0);
}

// Shared memory of chol_panels.
struct CholShared {
  double rowbuf[2][2 * kCholNb];
  double Ls[kCholNb][kCholNb + 1];   // L_JJ^{-1} of the panel
  double xd[kCholSmemMax];           // diagonal of L^{-1}
  int bad;                           // a pivot not above floor_d (cleared by the caller)
};

// The factorisation described at chol_inv_smem_kernel, by the 512 threads of a block: A (shared, pitch
// n + 1) holds G in its upper triangle and zeros below; on return R and, below the diagonal, L^{-1}.
__device__ void chol_panels(double* A, int n, double floor_d, CholShared& ch) {
  const int ld = n + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int j0 = 0; j0 < n; j0 += kCholNb) {
    const int w = min(kCholNb, n - j0);
    {   // [R_JJ | L_JJ^{-1}] of the diagonal block: element (i, c) = (warp, lane)
      const int i = warp, c = lane;
      double v = (i == (c & 15)) ? 1.0 : 0.0;   // also the padding of the last panel
      if (c < w && i < w) v = c >= i ? A[(j0 + i) * ld + j0 + c] : A[(j0 + c) * ld + j0 + i];
#pragma unroll 1
      for (int j = 0; j < w; ++j) {
        if (i == j) {
          const double d = __shfl_sync(0xffffffffu, v, j);
          // d > floor_d >= 0 and finite, as integers: an FP64 comparison is a round trip to a busy pipe
          const long long bits = __double_as_longlong(d);
          if (bits <= __double_as_longlong(floor_d) || bits >= 0x7ff0000000000000ll)
            ch.bad = 1;   // the same in every lane
          v *= rsqrt_refined(d);
          ch.rowbuf[j & 1][c] = v;
        }
        __syncthreads();
        if (i > j) v = fma(-ch.rowbuf[j & 1][i], ch.rowbuf[j & 1][c], v);
      }
      if (i < w) {
        if (c < w && c >= i) A[(j0 + i) * ld + j0 + c] = v;
        if (c >= kCholNb) {
          const int q = c - kCholNb;
          ch.Ls[i][q] = v;   // zero above the diagonal
          if (q < i) A[(j0 + i) * ld + j0 + q] = v;
          if (q == i) ch.xd[j0 + i] = v;
        }
      }
    }
    __syncthreads();
    if (ch.bad) return;
    {   // the panel's rows of the other columns: L_JJ^{-1} [X | G]
      const int cols = n - w;
      constexpr int kPer = kCholNb * kCholSmemMax / 512;
      double y[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const int t = tid + u * 512;
        double sum = 0.0;
        if (t < w * cols) {
          const int i = t / cols, q = t - i * cols;
          const double* col = A + j0 * ld + (q < j0 ? q : q + w);
          for (int k = 0; k <= i; ++k) sum = fma(ch.Ls[i][k], col[k * ld], sum);
        }
        y[u] = sum;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const int t = tid + u * 512;
        if (t < w * cols) {
          const int i = t / cols, q = t - i * cols;
          A[(j0 + i) * ld + (q < j0 ? q : q + w)] = y[u];
        }
      }
    }
    __syncthreads();
    // rows below: columns left of the panel and the panel's own (L^{-1}), and from the diagonal on (G)
    const int r0 = j0 + w;
    for (int i = r0 + warp; i < n; i += 16) {
      double f[kCholNb];
#pragma unroll
      for (int k = 0; k < kCholNb; ++k) f[k] = k < w ? A[(j0 + k) * ld + i] : 0.0;
      for (int q = lane; q < r0 + (n - i); q += 32) {
        const int c = q < r0 ? q : q - r0 + i;
        double v = A[i * ld + c];
        if (c >= j0 && c < r0) {
#pragma unroll
          for (int k = 0; k < kCholNb; ++k)
            if (k < w) v = fma(-f[k], ch.Ls[k][c - j0], v);
        } else {
#pragma unroll
          for (int k = 0; k < kCholNb; ++k)
            if (k < w) v = fma(-f[k], A[(j0 + k) * ld + c], v);
        }
        A[i * ld + c] = v;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(512) chol_inv_smem_kernel(double* Gin, int n,
                                                            int64_t shift_rows, int pass, double* Rout,
                                                            double* Riout, int* status, int* done) {
  stream_wait();
  extern __shared__ double A[];
  const int ld = n + 1;
  __shared__ CholShared ch;
  __shared__ GramStats st;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) { st.mx = 0u; st.dmax = 0u; }
  for (int t = tid; t < n * n; t += nt) {
    const int i = t / n, k = t - i * n;
    A[i * ld + k] = k < i ? 0.0 : Gin[t];   // the Gram matrix is formed in its upper triangle only
  }
  __syncthreads();
  gram_stats(A, n, ld, pass > 0, &st);
  __syncthreads();
  const double mx = from_high_word(st.mx), dmax = from_high_word(st.dmax), tr = st.tr;
  if (pass > 0) {
    if (tid == 0) {
      if (pass == 2 && !(mx <= 0.1)) *status = 2;
      if (pass == 1) *done = (n * mx <= 0.5) ? 1 : 0;
    }
    if (mx <= kNearIdentity) {
      // First-order factor: R = I + U with U the strict upper triangle of E plus half its
      // diagonal (U + U^T = E), and R^{-1} = I - U. Both are exact to O(n max|E|^2) <= 1.6e-16
      // for max|E| <= 1e-9, so the pass costs O(n^2).
      for (int t = tid; t < n * n; t += nt) {
        const int i = t / n, k = t - i * n;
        const double e = (k >= i) ? A[i * ld + k] - (i == k ? 1.0 : 0.0) : 0.0;
        const double u = (k > i) ? e : (k == i ? 0.5 * e : 0.0);
        const double id = (i == k) ? 1.0 : 0.0;
        Rout[t] = id + u;
        Riout[t] = id - u;
        Gin[t] = 0.0;
      }
      return;
    }
  }
  double sc, rsc, irsc;   // a power of four takes the diagonal into the FP32 range
  even_scale(dmax, sc, rsc, irsc);
  bool shifted = false;
  while (true) {
    if (tid == 0) ch.bad = 0;
    const double sft =
        shifted ? 11.0 * ((double)shift_rows * n + (double)n * (n + 1)) * kEps * tr : 0.0;
    for (int t = tid; t < n * n; t += nt) {
      const int i = t / n, k = t - i * n;
      A[i * ld + k] = (k < i) ? 0.0 : (Gin[t] + (i == k ? sft : 0.0)) * sc;
    }
    const double floor_d = (pass == 0 && !shifted) ? kPivotTol * dmax * sc : 0.0;
    __syncthreads();
    chol_panels(A, n, floor_d, ch);
    if (!ch.bad) break;
    __syncthreads();   // every thread has read `bad`
    if (pass > 0 || shifted) break;
    shifted = true;
  }
  if (ch.bad) {
    if (tid == 0) *status = 1;
    for (int t = tid; t < n * n; t += nt) Gin[t] = 0.0;
    return;
  }
  for (int t = tid; t < n * n; t += nt) {
    const int i = t / n, k = t - i * n;
    Rout[t] = k >= i ? A[i * ld + k] * rsc : 0.0;
    Riout[t] = k > i ? A[k * ld + i] * irsc : (k == i ? ch.xd[i] * irsc : 0.0);
    Gin[t] = 0.0;   // ready for the next Gram product
  }
}

// Ri = R^{-1} for the upper-triangular row-major R (one thread per column of Ri).
__global__ void trinv_kernel(const double* R, double* Ri, int n) {
  stream_wait();
  for (int j = threadIdx.x + blockIdx.x * blockDim.x; j < n; j += blockDim.x * gridDim.x) {
    for (int i = n - 1; i >= 0; --i) {
      double v = (i == j) ? 1.0 : 0.0;
      if (i <= j) {
        for (int k = i + 1; k <= j; ++k) v = fma(-R[(int64_t)i * n + k], Ri[(int64_t)k * n + j], v);
        v /= R[(int64_t)i * n + i];
      }
      Ri[(int64_t)i * n + j] = (i <= j) ? v : 0.0;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Single-block Householder QR (LAPACK dgeqrf/dorgqr scheme): W (m x n col-major, ld m) is
// overwritten; outputs Q (m x k, ld m) and R (k x n, ld k), k = min(m, n).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void householder_body(double* W, int m, int n, double* Q, double* R,
                                                 double* tau) {
  __shared__ double sh[32];
  __shared__ double refl[3];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int k = min(m, n);
  for (int j = 0; j < k; ++j) {
    double* col = W + (int64_t)j * m;
    double xs = 0.0;
    for (int i = j + 1 + tid; i < m; i += nt) xs = fma(col[i], col[i], xs);
    xs = block_sum_d(xs, sh);
    if (tid == 0) {   // reflector scalars once per column (FP64 sqrt/division are DFMA sequences)
      const double alpha = col[j];
      double tj = 0.0, beta = alpha, scale = 0.0;
      if (xs > 0.0) {
        beta = -copysign(sqrt(alpha * alpha + xs), alpha);
        tj = (beta - alpha) / beta;
        scale = 1.0 / (alpha - beta);
      }
      refl[0] = tj; refl[1] = beta; refl[2] = scale;
    }
    __syncthreads();
    const double tj = refl[0], beta = refl[1], scale = refl[2];
    for (int i = j + 1 + tid; i < m; i += nt) col[i] *= scale;
    __syncthreads();
    if (tid == 0) { col[j] = beta; tau[j] = tj; }
    __syncthreads();
    if (tj != 0.0) {
      for (int c = j + 1 + warp; c < n; c += nw) {
        double* cc = W + (int64_t)c * m;
        const double c0 = cc[j];   // read by every lane before lane 0 updates it
        double w = 0.0;
        for (int i = j + 1 + lane; i < m; i += 32) w = fma(col[i], cc[i], w);
        w = red::warp_sum(w) + c0;
        const double tw = tj * w;
        if (lane == 0) cc[j] -= tw;
        for (int i = j + 1 + lane; i < m; i += 32) cc[i] = fma(-tw, col[i], cc[i]);
      }
    }
    __syncthreads();
  }
  // R = upper part
  for (int64_t t = tid; t < (int64_t)k * n; t += nt) {
    const int i = (int)(t % k), c = (int)(t / k);
    R[t] = (i <= c) ? W[(int64_t)c * m + i] : 0.0;
  }
  // Q = H_0 ... H_{k-1} [I; 0]
  for (int64_t t = tid; t < (int64_t)m * k; t += nt) {
    const int i = (int)(t % m), c = (int)(t / m);
    Q[t] = (i == c) ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int j = k - 1; j >= 0; --j) {
    const double tj = tau[j];
    if (tj == 0.0) continue;
    const double* col = W + (int64_t)j * m;
    for (int c = j + warp; c < k; c += nw) {
      double* qc = Q + (int64_t)c * m;
      const double q0 = qc[j];
      double w = 0.0;
      for (int i = j + 1 + lane; i < m; i += 32) w = fma(col[i], qc[i], w);
      w = red::warp_sum(w) + q0;
      const double tw = tj * w;
      if (lane == 0) qc[j] -= tw;
      for (int i = j + 1 + lane; i < m; i += 32) qc[i] = fma(-tw, col[i], qc[i]);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(512) householder_kernel(double* W, int m, int n, double* Q,
                                                          double* R, double* tau) {
  stream_wait();
  householder_body(W, m, n, Q, R, tau);
}

// The same factorisation with W, Q and tau in shared memory (m * n + m * k + k doubles), read
// straight from A (ld lda): every step of the column sweep is a shared-memory access instead of an
// L2 round trip, which is what bounds the small QRs of the enrichment blocks (m <= 1024, n <= 16).
constexpr int kHouseholderSmemBytes = 200 * 1024;

__global__ void __launch_bounds__(512, 1) householder_smem_kernel(const double* A,
                                                               int64_t lda, int m, int n,
                                                               double* Qout, double* R) {
  stream_wait();
  extern __shared__ double hs[];
  const int k = min(m, n);
  double* W = hs;
  double* Q = W + (int64_t)m * n;
  double* tau = Q + (int64_t)m * k;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int64_t t = tid; t < (int64_t)m * n; t += nt) {
    const int64_t i = t % m, j = t / m;
    W[t] = A[j * lda + i];
  }
  __syncthreads();
  householder_body(W, m, n, Q, R, tau);
  __syncthreads();
  for (int64_t t = tid; t < (int64_t)m * k; t += nt) Qout[t] = Q[t];
}

// ---------------------------------------------------------------------------------------------
// CholeskyQR of a small matrix in one launch (512 threads, everything in shared memory): the passes of
// qr() below without their launches and host wait, and the Householder factorisation in the same
// launch when they break down. A Householder sweep pays two reductions over the block and a chain of
// square root and divisions per column, twice (once more to form Q): 27 us for 48 x 4, 131 us for
// 128 x 16. Here a pass is one Gram product, whose sums run over the lanes of a few threads each, the
// n steps of the 16 x 16 block factorisation, and one triangular product.
// ---------------------------------------------------------------------------------------------
constexpr int kCholQrSmallN = 32;

__global__ void __launch_bounds__(512, 1) cholqr_small_kernel(const double* A, int64_t lda,
                                                              int m, int n, double* Qout, double* Rout) {
  stream_wait();
  extern __shared__ double hs[];
  const int ldq = m | 1;   // odd pitch of the columns
  double* X = hs;                            // m x n, this pass's input
  double* Y = X + (int64_t)ldq * n;          // its output
  double* G = Y + (int64_t)ldq * n;          // n x (n + 1)
  double* R = G + n * (n + 1);               // product of the R factors, upper, row-major pitch n
  double* S = R + n * n;
  __shared__ CholShared ch;
  __shared__ GramStats st;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int ld = n + 1;
  for (int t = tid; t < m * n; t += nt) {
    const int j = t / m, i = t - j * m;
    X[j * ldq + i] = A[(int64_t)j * lda + i];
  }
  for (int t = tid; t < n * n; t += nt) R[t] = (t / n == t % n) ? 1.0 : 0.0;
  __syncthreads();
  const int pairs = n * (n + 1) / 2;
  const int lpe = pairs <= 16 ? 32 : pairs <= 64 ? 8 : pairs <= 256 ? 4 : 2;   // lanes per Gram entry
  bool ok = true;
  for (int pass = 0; pass < 3; ++pass) {
    if (tid == 0) { st.mx = 0u; st.dmax = 0u; }
    // G = X^T X, upper triangle: lpe lanes share an entry's rows
    for (int e0 = warp * (32 / lpe); e0 < pairs; e0 += (nt / 32) * (32 / lpe)) {
      const int e = min(e0 + lane / lpe, pairs - 1);
      int k = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);   // column of entry e = k (k + 1) / 2 + i
      while (k * (k + 1) / 2 > e) --k;
      while ((k + 1) * (k + 2) / 2 <= e) ++k;
      const int i = e - k * (k + 1) / 2;
      const double* x = X + i * ldq;
      const double* y = X + k * ldq;
      double s0 = 0.0, s1 = 0.0;
      int r = lane % lpe;
      for (; r + lpe < m; r += 2 * lpe) {
        s0 = fma(x[r], y[r], s0);
        s1 = fma(x[r + lpe], y[r + lpe], s1);
      }
      if (r < m) s0 = fma(x[r], y[r], s0);
      s0 += s1;
      for (int o = lpe >> 1; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if (lane % lpe == 0 && e0 + lane / lpe < pairs) {
        S[i * n + k] = s0;
      }
    }
    __syncthreads();
    gram_stats(S, n, n, pass > 0, &st);
    __syncthreads();
    const double mx = from_high_word(st.mx), dmax = from_high_word(st.dmax), tr = st.tr;
    if (pass == 2 && !(mx <= 0.1)) { ok = false; break; }
    double rsc = 1.0, irsc = 1.0;
    if (pass > 0 && mx <= kNearIdentity) {   // first-order factor, see chol_inv_smem_kernel
      for (int t = tid; t < n * n; t += nt) {
        const int i = t / n, k = t - i * n;
        const double e = S[i <= k ? i * n + k : k * n + i] - (i == k ? 1.0 : 0.0);
        G[i * ld + k] = i == k ? 1.0 + 0.5 * e : (k > i ? e : -e);   // R above, L^{-1} = R^{-T} below
        if (i == k) ch.xd[i] = 1.0 - 0.5 * e;
      }
      __syncthreads();
    } else {
      double sc;
      even_scale(dmax, sc, rsc, irsc);
      for (int shifted = 0; shifted < 2; ++shifted) {
        const double sft = shifted ? 11.0 * ((double)m * n + (double)n * (n + 1)) * kEps * tr : 0.0;
        __syncthreads();
        if (tid == 0) ch.bad = 0;
        for (int t = tid; t < n * n; t += nt) {
          const int i = t / n, k = t - i * n;
          G[i * ld + k] = (k < i) ? 0.0 : (S[t] + (i == k ? sft : 0.0)) * sc;
        }
        __syncthreads();
        chol_panels(G, n, (pass == 0 && !shifted) ? kPivotTol * dmax * sc : 0.0, ch);
        __syncthreads();
        if (!ch.bad || pass > 0) break;
      }
      if (ch.bad) { ok = false; break; }
    }
    // Y = X R^{-1}, columns k and n - 1 - k by one thread (n + 1 terms)
    const int half = (n + 1) / 2;
    for (int t = tid; t < m * half; t += nt) {
      const int p = t / m, r = t - p * m;
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        const int k = side ? n - 1 - p : p;
        if (side && k == p) break;
        double s0 = X[k * ldq + r] * ch.xd[k], s1 = 0.0;
        int i = 0;
        for (; i + 1 < k; i += 2) {
          s0 = fma(X[i * ldq + r], G[k * ld + i], s0);
          s1 = fma(X[(i + 1) * ldq + r], G[k * ld + i + 1], s1);
        }
        if (i < k) s0 = fma(X[i * ldq + r], G[k * ld + i], s0);
        Y[k * ldq + r] = (s0 + s1) * irsc;
      }
    }
    // R <- R_pass R (through S)
    for (int t = tid; t < n * n; t += nt) {
      const int i = t / n, k = t - i * n;
      double v = 0.0;
      for (int l = i; l <= k; ++l) v = fma(G[i * ld + l], R[l * n + k], v);
      S[t] = v * rsc;
    }
    __syncthreads();
    for (int t = tid; t < n * n; t += nt) R[t] = S[t];
    double* tmp = X; X = Y; Y = tmp;
    __syncthreads();
    if (pass == 1 && n * mx <= 0.5) break;   // near enough to the identity: X is orthonormal
  }
  if (ok) {
    for (int t = tid; t < m * n; t += nt) {
      const int j = t / m, i = t - j * m;
      Qout[t] = X[j * ldq + i];
    }
    for (int t = tid; t < n * n; t += nt) {   // column-major
      const int k = t / n, i = t - k * n;
      Rout[t] = R[i * n + k];
    }
    return;
  }
  __syncthreads();
  double* W = hs;
  double* Q = W + (int64_t)m * n;
  for (int t = tid; t < m * n; t += nt) {
    const int j = t / m, i = t - j * m;
    W[t] = A[(int64_t)j * lda + i];
  }
  __syncthreads();
  householder_body(W, m, n, Q, Rout, Q + (int64_t)m * n);
  __syncthreads();
  for (int t = tid; t < m * n; t += nt) Qout[t] = Q[t];
}

size_t cholqr_small_smem(int64_t m, int64_t n) {
  return (size_t)(2 * (m | 1) * n + n * (n + 1) + 2 * n * n) * sizeof(double);
}

// ---------------------------------------------------------------------------------------------
// Batched R-only Householder QR, one block per matrix: block b factors W + b * stride (rows x n,
// column-major, ld rows) in place and writes its R factor as the n x n column-major block
// Rout + b * n * n (upper triangle; rows >= min(rows, n) and the lower part zero). The levels of
// the TSQR reduction in qr_r are launches of this kernel.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(512) householder_r_kernel(double* Wall, int64_t stride, int rows,
                                                            int n, double* Rout) {
  __shared__ double sh[32];
  __shared__ double refl[3];
  double* W = Wall + (int64_t)blockIdx.x * stride;
  double* R = Rout + (int64_t)blockIdx.x * n * n;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int k = min(rows, n);
  for (int j = 0; j < k; ++j) {
    double* col = W + (int64_t)j * rows;
    double xs = 0.0;
    for (int i = j + 1 + tid; i < rows; i += nt) xs = fma(col[i], col[i], xs);
    xs = block_sum_d(xs, sh);
    if (tid == 0) {   // reflector scalars once per column (FP64 sqrt/division are DFMA sequences)
      const double alpha = col[j];
      double tj = 0.0, beta = alpha, scale = 0.0;
      if (xs > 0.0) {
        beta = -copysign(sqrt(alpha * alpha + xs), alpha);
        tj = (beta - alpha) / beta;
        scale = 1.0 / (alpha - beta);
      }
      refl[0] = tj; refl[1] = beta; refl[2] = scale;
    }
    __syncthreads();
    const double tj = refl[0], beta = refl[1], scale = refl[2];
    for (int i = j + 1 + tid; i < rows; i += nt) col[i] *= scale;
    __syncthreads();
    if (tid == 0) col[j] = beta;
    __syncthreads();
    if (tj != 0.0) {
      for (int c = j + 1 + warp; c < n; c += nw) {
        double* cc = W + (int64_t)c * rows;
        const double c0 = cc[j];
        double w = 0.0;
        for (int i = j + 1 + lane; i < rows; i += 32) w = fma(col[i], cc[i], w);
        w = red::warp_sum(w) + c0;
        const double tw = tj * w;
        if (lane == 0) cc[j] -= tw;
        for (int i = j + 1 + lane; i < rows; i += 32) cc[i] = fma(-tw, col[i], cc[i]);
      }
    }
    __syncthreads();
  }
  for (int64_t t = tid; t < (int64_t)n * n; t += nt) {
    const int i = (int)(t % n), c = (int)(t / n);
    R[t] = (i <= c && i < k) ? W[(int64_t)c * rows + i] : 0.0;
  }
}

// Level-0 gather of TSQR: block b = rows [b*mb, b*mb + mb) of A (zero past m), column-major mb x n.
__global__ void tsqr_gather_kernel(const double* __restrict__ A, int64_t lda, int64_t m, int n,
                                   int mb, int nblk, double* W) {
  const int64_t per = (int64_t)mb * n, total = per * nblk;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / per, rem = t - b * per;
    const int64_t j = rem / mb, i = rem - j * mb;
    const int64_t row = b * mb + i;
    W[t] = (row < m) ? A[j * lda + row] : 0.0;
  }
}

// Next TSQR level: block b = [R_{2b}; R_{2b+1}] (2n x n column-major; zero when 2b+1 is missing).
__global__ void tsqr_stack_kernel(const double* __restrict__ R, int n, int nin, double* W) {
  const int nout = (nin + 1) / 2;
  const int64_t per = (int64_t)2 * n * n, total = per * nout;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / per, rem = t - b * per;
    const int64_t j = rem / (2 * n), i = rem - j * 2 * n;
    const int64_t src = 2 * b + (i >= n ? 1 : 0);
    const int64_t ii = i >= n ? i - n : i;
    W[t] = (src < nin) ? R[src * n * n + j * n + ii] : 0.0;
  }
}

// Rotation (c, s) of one-sided Jacobi for a column pair with squared norms a, b and inner product
// g (Demmel-Veselic formulas): false when the pair is orthogonal to `tol`. The angle comes from FP32
// arithmetic (relative error ~1e-7: the pair is left orthogonal to ~1e-7 and a later sweep finishes
// it); its cosine and sine, taken to FP64, are divided by their norm to FP64 accuracy with the series
// of 1 / sqrt(1 - d) for d = 1 - c^2 - s^2 ~ 1e-7, so (c, s) is orthogonal to rounding. An FP64 square
// root or division is a sequence of DFMA, and each dependent FP64 operation costs some 80 cycles of
// latency here: five of them follow the FP32 angle.
__device__ __forceinline__ bool jacobi_rotation(double a, double b, double g, double tol, double& c,
                                                double& s) {
  if (a == 0.0 || b == 0.0) return false;
  if (!(g * g > tol * tol * a * b)) return false;
  const float fb = (float)(b - a), fg = 2.0f * (float)g;
  float tf;
  if (fabsf(fb) >= fabsf(fg)) {   // r = 2g / (b - a), |r| <= 1: t = r / (1 + sqrt(1 + r^2))
    const float r = __fdividef(fg, fb);
    tf = __fdividef(r, 1.0f + sqrtf(fmaf(r, r, 1.0f)));
  } else {                        // zeta = (b - a) / 2g, |zeta| < 1
    const float z = __fdividef(fb, fg);
    tf = __fdividef(copysignf(1.0f, z), fabsf(z) + sqrtf(fmaf(z, z, 1.0f)));
  }
  if (tf == 0.0f || !isfinite(tf)) {   // operands outside the FP32 range: the exact FP64 formula
    const double zeta = (b - a) / (2.0 * g);
    const double t = (fabs(zeta) > 1e150) ? 0.5 / zeta
                                          : copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
    c = 1.0 / sqrt(1.0 + t * t);
    s = c * t;
    return true;
  }
  const float cf = rsqrtf(fmaf(tf, tf, 1.0f));
  c = (double)cf;
  s = (double)(cf * tf);
  const double d = fma(-s, s, fma(-c, c, 1.0));
  const double f = rsqrt_corrected(1.0, d);
  c *= f;
  s *= f;
  return true;
}

__device__ __forceinline__ int rr_index(int p, int r, int nn) {
  return p == 0 ? 0 : ((p - 1 + r) % (nn - 1)) + 1;
}

// ---------------------------------------------------------------------------------------------
// Block one-sided Jacobi on a thread-block cluster of kJacobiCluster CTAs for 16 <= n <=
// kJacobiBlockMaxN: the columns (padded to P = 2C blocks of nb) are treated as P blocks paired by
// the round-robin tournament; in round r the CTA i holds the blocks rr(i, r) and rr(P-1-i, r) in its
// own shared memory and rotates all their cross pairs there (nb sub-rounds of nb disjoint pairs,
// block barrier only; the pairs inside a block are rotated in the first round of each sweep), then
// pulls the two blocks of its next pair from their holders over DSMEM into its second buffer. Every
// pair of columns is visited once per sweep, as in the scalar cyclic order, with one cluster
// barrier per round (P - 1 per sweep), and every dot product reads local memory. The sweep's
// largest cosine and sine are collected in CTA 0 after a barrier and read by every CTA, so all CTAs leave the
// loop together. Vout: the accumulated rotations.
// ---------------------------------------------------------------------------------------------
constexpr int kJacobiCluster = 8;
constexpr int kJacobiBlockMaxN = 160;

// One rotation of a column pair by a group of L lanes, with tracked squared column norms (*na, *nb): only
// the inner product is reduced; the norms follow the rotation exactly (a' = c^2 a - 2cs g + s^2 b, b' =
// s^2 a + 2cs g + c^2 b) and are recomputed from the columns once per sweep, which bounds their drift.
// The lanes' EPL elements of the four columns are loaded before anything is stored, so the loads do not
// wait for the stores. The rotation is recorded in `worst`.
//
// A rotation of (p, q) adds s |q| / |p| times the cosine of (q, r) to the cosine of (p, r). Where |q| is the larger
// norm, s |q| / |p| is about the cosine of (p, q); within a cluster of equal norms it is s, which stays large
// however small the cosines are. So a sweep whose rotations had cosines up to c and sines up to t
// leaves cosines of about n c max(c, t): where that is below the tolerance of n 2^-52 the sweep that would
// only confirm it is not run. (Stopping by c t left 4e-12 for three rows 1e6 apart in norm.)
constexpr int kNoRotation = -4096;

struct JacobiWorst {
  int cosine = kNoRotation, sine = kNoRotation;   // exponents of the largest squares
  __device__ __forceinline__ bool converged() const { return cosine + max(cosine, sine) <= -114; }
};

template <int L, int EPL>
__device__ __forceinline__ void jacobi_rotate_tracked(double* wp, double* wq, double* vp, double* vq,
                                                      double* na, double* nb, int n, double tol, int gl,
                                                      unsigned mask, JacobiWorst& worst) {
  double x[EPL], y[EPL], u[EPL], v[EPL];
  double g = 0.0;
#pragma unroll
  for (int k = 0; k < EPL; ++k) {
    const int i = gl + k * L;
    x[k] = i < n ? wp[i] : 0.0;
    y[k] = i < n ? wq[i] : 0.0;
    u[k] = i < n ? vp[i] : 0.0;
    v[k] = i < n ? vq[i] : 0.0;
    g = fma(x[k], y[k], g);
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) g += __shfl_xor_sync(mask, g, o);
  const double a = *na, b = *nb;
  double c, s;
  if (!jacobi_rotation(a, b, g, tol, c, s)) return;
#pragma unroll
  for (int k = 0; k < EPL; ++k) {
    const int i = gl + k * L;
    if (i < n) {
      wp[i] = c * x[k] - s * y[k];
      wq[i] = s * x[k] + c * y[k];
      vp[i] = c * u[k] - s * v[k];
      vq[i] = s * u[k] + c * v[k];
    }
  }
  __syncwarp(mask);   // every lane has read the norms
  if (gl == 0) {
    const double cc = c * c, ss = s * s, cs2 = 2.0 * c * s * g;
    const double a2 = cc * a - cs2 + ss * b, b2 = ss * a + cs2 + cc * b;
    *na = a2 > 0.0 ? a2 : 0.0;
    *nb = b2 > 0.0 ? b2 : 0.0;
  }
  const auto expo = [](double t) { return (__double2hiint(t) >> 20) & 0x7ff; };
  worst.cosine = max(worst.cosine, 2 * expo(g) - expo(a) - expo(b));
  worst.sine = max(worst.sine, 2 * (expo(s) - 1023));
}

// Powers of two that take a matrix whose largest entry has the high word `top` to about 1 and back: the
// products of squared norms in the rotations stay in range. 1 for a matrix that is zero, not finite or
// beyond 2^+-959.
__device__ __forceinline__ void jacobi_scale(unsigned top, double& down, double& up) {
  int e = (int)((top & 0x7fffffffu) >> 20);
  if (e < 64 || e > 1982) e = 1023;
  down = __hiloint2double((2046 - e) << 20, 0);
  up = __hiloint2double(e << 20, 0);
}

// W = R^T scaled by jacobi_scale, *up the factor back. One block.
__global__ void __launch_bounds__(1024) scaled_transpose_kernel(const double* R, int n, double* W,
                                                                double* up) {
  stream_wait();
  __shared__ unsigned top;
  if (threadIdx.x == 0) top = 0u;
  __syncthreads();
  unsigned m = 0u;
  for (int64_t t = threadIdx.x; t < (int64_t)n * n; t += blockDim.x)
    m = max(m, (unsigned)__double2hiint(R[t]) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&top, m);
  __syncthreads();
  double d, u;
  jacobi_scale(top, d, u);
  if (threadIdx.x == 0) *up = u;
  for (int64_t t = threadIdx.x; t < (int64_t)n * n; t += blockDim.x) {
    const int64_t j = t / n, i = t - j * n;
    W[t] = R[i * n + j] * d;
  }
}

// ---------------------------------------------------------------------------------------------
// One-sided (Hestenes) Jacobi of R^T (R column-major n x n, n < 16) in one warp: four lanes share a
// column pair, so a round of the round-robin tournament is one rotation step of the whole warp without
// a block barrier, and the scalars of all its rotations are computed at once (a warp per pair took 222
// us at n = 12). Un: the normalised rotated columns, Vs: the rotations, both by descending S.
// ---------------------------------------------------------------------------------------------
constexpr int kJacobiWarpMaxN = 16;

__global__ void __launch_bounds__(32) jacobi_warp_kernel(const double* R, int n, double* Un,
                                                         double* S, double* Vs, int* status) {
  stream_wait();
  constexpr int N = kJacobiWarpMaxN, ld = N + 1;
  __shared__ double W[N * ld], V[N * ld], nrm[N];
  const int lane = threadIdx.x, gid = lane / 4, gl = lane % 4;
  const unsigned mask = 0xfu << (lane & 28);
  unsigned top = 0u;
  for (int t = lane; t < n * n; t += 32) top = max(top, (unsigned)__double2hiint(R[t]) & 0x7fffffffu);
  double down, up;
  jacobi_scale(__reduce_max_sync(0xffffffffu, top), down, up);
  for (int t = lane; t < N * N; t += 32) {
    const int j = t / N, i = t % N;
    W[j * ld + i] = (i < n && j < n) ? R[(int64_t)i * n + j] * down : 0.0;
    V[j * ld + i] = i == j ? 1.0 : 0.0;
  }
  __syncwarp();
  const int nn = n + (n & 1);
  const double tol = (double)n * kEps;
  auto norms = [&]() {   // squared norms: two lanes per column
    const int c = lane / 2;
    double a = 0.0;
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
      const double w = W[c * ld + 2 * k + (lane & 1)];
      a = fma(w, w, a);
    }
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    if ((lane & 1) == 0) nrm[c] = a;
    __syncwarp();
  };
  bool converged = false;
  for (int sweep = 0; sweep < 60 && !converged; ++sweep) {
    norms();
    JacobiWorst worst;
    int u = gid, v = nn - 1 - gid;   // the pair's places in the tournament
    for (int r = 0; r < nn - 1; ++r) {
      const int p = min(u, v), q = max(u, v);
      if (gid < nn / 2 && q < n)
        jacobi_rotate_tracked<4, N / 4>(W + p * ld, W + q * ld, V + p * ld, V + q * ld, nrm + p, nrm + q, n,
                                        tol, gl, mask, worst);
      if (u != 0 && ++u == nn) u = 1;
      if (++v == nn) v = 1;
      __syncwarp();
    }
    worst.cosine = __reduce_max_sync(0xffffffffu, worst.cosine);
    worst.sine = __reduce_max_sync(0xffffffffu, worst.sine);
    converged = worst.converged();
  }
  if (!converged && lane == 0) *status = 3;
  norms();
  if (lane < n) nrm[lane] = sqrt(nrm[lane]);
  __syncwarp();
  for (int j = 0; j < n; ++j) {
    const double sj = nrm[j];
    const double si = lane < n ? nrm[lane] : -1.0;
    const int rk = __popc(__ballot_sync(0xffffffffu, lane < n && (si > sj || (si == sj && lane < j))));
    if (lane == 0) S[rk] = sj * up;
    if (lane < n) {
      Un[(int64_t)rk * n + lane] = sj > 0.0 ? W[j * ld + lane] / sj : 0.0;
      Vs[(int64_t)rk * n + lane] = V[j * ld + lane];
    }
  }
}

template <int EPL>
__global__ void __cluster_dims__(kJacobiCluster, 1, 1) __launch_bounds__(256)
    jacobi_block_kernel(const double* Win, int n, double* Wout, double* Vout, int max_sweeps,
                        int* status) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  double* sm = reinterpret_cast<double*>(sm_raw);
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int C = kJacobiCluster, P = 2 * kJacobiCluster;
  const int rank = (int)cluster.block_rank();
  const int nb = (n + P - 1) / P;
  const int64_t blk = (int64_t)nb * n;   // elements of one block of W (or of V)
  const int64_t unit = 2 * blk + nb + (nb & 1);   // W block, V block, squared column norms
  // buffer x (0/1), slot s (0/1): W block, V block, norms
  auto Wb = [&](double* base, int x, int sl) { return base + (int64_t)(x * 2 + sl) * unit; };
  auto Vb = [&](double* base, int x, int sl) { return base + (int64_t)(x * 2 + sl) * unit + blk; };
  auto Nb = [&](double* base, int x, int sl) { return base + (int64_t)(x * 2 + sl) * unit + 2 * blk; };
  __shared__ int counts[2 * kJacobiCluster];   // in CTA 0: every CTA's largest cosine and sine of a sweep
  __shared__ int local_cnt[2];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const double tol = (double)(n > 1 ? n : 1) * kEps;

  // round 0 of sweep 0: slot 0 holds block rank, slot 1 block P-1-rank
  for (int sl = 0; sl < 2; ++sl) {
    const int b = sl == 0 ? rank : P - 1 - rank;
    double* W = Wb(sm, 0, sl);
    double* V = Vb(sm, 0, sl);
    for (int64_t t = tid; t < blk; t += nt) {
      const int j = (int)(t / n), i = (int)(t - (int64_t)j * n);
      const int c = b * nb + j;
      W[t] = (c < n) ? Win[(int64_t)c * n + i] : 0.0;
      V[t] = (c < n) ? (i == c ? 1.0 : 0.0) : 0.0;
    }
  }
  int* counts0 = cluster.map_shared_rank(counts, 0);
  int x = 0, r = 0, sweep = 0;
  JacobiWorst mine;
  bool converged = false;
  if (tid < 2) local_cnt[tid] = kNoRotation;
  __syncthreads();
  while (true) {
    const int bA = rr_index(rank, r, P), bB = rr_index(P - 1 - rank, r, P);
    double* WA = Wb(sm, x, 0); double* VA = Vb(sm, x, 0); double* NA = Nb(sm, x, 0);
    double* WB = Wb(sm, x, 1); double* VB = Vb(sm, x, 1); double* NB = Nb(sm, x, 1);
    if (r == 0) {   // fresh column norms, then the pairs inside each block, once per sweep
      for (int c = warp; c < 2 * nb; c += nw) {
        const double* w = (c < nb ? WA : WB) + (int64_t)(c % nb) * n;
        double a = 0.0;
        for (int i = lane; i < n; i += 32) a = fma(w[i], w[i], a);
        a = red::warp_sum(a);
        if (lane == 0) (c < nb ? NA : NB)[c % nb] = a;
      }
      __syncthreads();
      const int m2 = nb + (nb & 1);
      for (int t = 0; t < m2 - 1; ++t) {
        for (int task = warp; task < m2; task += nw) {   // m2/2 pairs per slot, 2 slots
          const int sl = task / (m2 / 2), pi = task % (m2 / 2);
          int p = rr_index(pi, t, m2), q = rr_index(m2 - 1 - pi, t, m2);
          if (p > q) { const int u = p; p = q; q = u; }
          if (q >= nb) continue;
          double* W = sl ? WB : WA;
          double* V = sl ? VB : VA;
          double* Nm = sl ? NB : NA;
          jacobi_rotate_tracked<32, EPL>(W + (int64_t)p * n, W + (int64_t)q * n, V + (int64_t)p * n,
                                         V + (int64_t)q * n, Nm + p, Nm + q, n, tol, lane, 0xffffffffu,
                                         mine);
        }
        __syncthreads();
      }
    }
    for (int t = 0; t < nb; ++t) {   // cross pairs (j, j + t mod nb)
      for (int j = warp; j < nb; j += nw) {
        const int k = (j + t) % nb;
        const int ga = bA * nb + j, gb = bB * nb + k;
        double *wp = WA + (int64_t)j * n, *wq = WB + (int64_t)k * n;
        double *vp = VA + (int64_t)j * n, *vq = VB + (int64_t)k * n;
        double *np = NA + j, *nq = NB + k;
        if (ga > gb) {
          double* u = wp; wp = wq; wq = u; u = vp; vp = vq; vq = u; u = np; np = nq; nq = u;
        }
        jacobi_rotate_tracked<32, EPL>(wp, wq, vp, vq, np, nq, n, tol, lane, 0xffffffffu, mine);
      }
      __syncthreads();
    }
    const bool sweep_end = (r == P - 2);
    if (sweep_end) {
      if (lane == 0) {
        atomicMax(&local_cnt[0], mine.cosine);
        atomicMax(&local_cnt[1], mine.sine);
      }
      mine = JacobiWorst();
      __syncthreads();
      if (tid < 2) { counts0[2 * rank + tid] = local_cnt[tid]; local_cnt[tid] = kNoRotation; }
    }
    cluster.sync();   // every CTA finished round r (and published its count at a sweep end)
    if (sweep_end) {
      JacobiWorst all;
      for (int c = 0; c < C; ++c) {
        all.cosine = max(all.cosine, counts0[2 * c]);
        all.sine = max(all.sine, counts0[2 * c + 1]);
      }
      ++sweep;
      if (all.converged()) { converged = true; break; }
      if (sweep >= max_sweeps) break;
    }
    // pull the blocks of round r+1 into buffer 1-x from their holders' buffer x
    const int rn = (r + 1) % (P - 1);
    for (int sl = 0; sl < 2; ++sl) {
      const int b = rr_index(sl == 0 ? rank : P - 1 - rank, rn, P);
      int owner = 0, oslot = 0;
      for (int c = 0; c < C; ++c) {
        if (rr_index(c, r, P) == b) { owner = c; oslot = 0; }
        if (rr_index(P - 1 - c, r, P) == b) { owner = c; oslot = 1; }
      }
      const double* srcW = cluster.map_shared_rank(Wb(sm, x, oslot), owner);
      const double* srcV = cluster.map_shared_rank(Vb(sm, x, oslot), owner);
      const double* srcN = cluster.map_shared_rank(Nb(sm, x, oslot), owner);
      double* dW = Wb(sm, 1 - x, sl);
      double* dV = Vb(sm, 1 - x, sl);
      double* dN = Nb(sm, 1 - x, sl);
      for (int64_t t = tid; t < blk; t += nt) { dW[t] = srcW[t]; dV[t] = srcV[t]; }
      for (int t = tid; t < nb; t += nt) dN[t] = srcN[t];
    }
    __syncthreads();
    x = 1 - x;
    r = rn;
  }
  if (rank == 0 && tid == 0 && !converged && status) *status = 3;
  // buffer x holds the blocks of round r
  for (int sl = 0; sl < 2; ++sl) {
    const int b = rr_index(sl == 0 ? rank : P - 1 - rank, r, P);
    const double* W = Wb(sm, x, sl);
    const double* V = Vb(sm, x, sl);
    for (int64_t t = tid; t < blk; t += nt) {
      const int j = (int)(t / n), i = (int)(t - (int64_t)j * n);
      const int c = b * nb + j;
      if (c < n) {
        Wout[(int64_t)c * n + i] = W[t];
        Vout[(int64_t)c * n + i] = V[t];
      }
    }
  }
  cluster.sync();   // no CTA leaves while another may still read its shared memory
}

// ---------------------------------------------------------------------------------------------
// FP32 one-sided Jacobi on R^T (R column-major n x n) in one block, for a starting basis: X (column-major)
// gets the normalised columns of the rotated R^T by descending norm, i.e. R's right singular vectors to
// FP32 accuracy, sig their norms for the matrix scaled to largest entry 1, *scale the factor back,
// inv_sig the reciprocals of the unscaled norms; *bad = 1 when a norm is zero or not finite.
// The whole matrix is in shared memory and a round of the tournament one batch of pairs. The block is
// bound by its instruction issue, so 8 lanes share a pair: the scalars of a rotation are then computed
// for four pairs at once (with a warp per pair a round took 1600 cycles at n = 77). The column pitch is 8
// modulo 32, which puts the four column pairs of a warp, neighbours in the tournament, on different
// banks. A sweep stops the iteration when no cosine in it was above 1e-4: its own rotations leave about
// n times the square (*bad = 1 when 16 sweeps do not get there).
// ---------------------------------------------------------------------------------------------
constexpr int kJacobiF32MaxN = 224;

// pitch of the columns, which hold 8 EPL elements (zeros past n)
__host__ __device__ constexpr int jacobi_f32_pitch(int epl) { return (8 * epl + 23) / 32 * 32 + 8; }

template <int EPL>
__global__ void __launch_bounds__(32 * EPL) jacobi_f32_kernel(const double* R, int n, double* X,
                                                          double* sig, double* inv_sig, double* scale,
                                                          int* bad) {
  stream_wait();
  constexpr int L = 8, ld = jacobi_f32_pitch(EPL);
  extern __shared__ float wf[];
  __shared__ unsigned top, cmax;
  __shared__ float nrm[kJacobiF32MaxN];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  if (tid == 0) { top = 0u; cmax = 0u; }
  __syncthreads();
  unsigned mx = 0u;
  for (int t = tid; t < n * n; t += nt) mx = max(mx, (unsigned)__double2hiint(R[t]) & 0x7fffffffu);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) atomicMax(&top, mx);
  __syncthreads();
  const int e = (int)(top >> 20);   // exponent field of the largest entry
  if (e < 64 || e > 1982) {         // zero, not finite, or outside the scale's range
    if (tid == 0) *bad = 1;
    return;
  }
  double down, up;
  jacobi_scale(top, down, up);
  for (int t = tid; t < n * ld; t += nt) wf[t] = 0.f;
  __syncthreads();
  for (int t = tid; t < n * n; t += nt) {
    const int i = t / n, j = t - i * n;   // R[j, i] = R^T[i, j]
    wf[j * ld + i] = (float)(R[t] * down);
  }
  __syncthreads();
  const int nn = n + (n & 1), gid = tid / L, gl = tid % L;
  const unsigned mask = 0xffu << (lane & 24);
  const bool pair = gid < nn / 2;
  for (int sweep = 0; sweep < 16; ++sweep) {
    float worst = 0.f;
    // positions gid and nn - 1 - gid of the tournament: each column but 0 moves on by one per round
    int u = gid == 0 ? 0 : gid, v = nn - 1 - gid;
    for (int r = 0; r < nn - 1; ++r) {
      const int p = min(u, v), q = max(u, v);
      if (pair && q < n) {
        float* wp = wf + p * ld + gl;
        float* wq = wf + q * ld + gl;
        float x[EPL], y[EPL];
        float a = 0.f, b = 0.f, g = 0.f;
#pragma unroll
        for (int k = 0; k < EPL; ++k) {
          x[k] = wp[k * L];
          y[k] = wq[k * L];
          a = fmaf(x[k], x[k], a);
          b = fmaf(y[k], y[k], b);
          g = fmaf(x[k], y[k], g);
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
          a += __shfl_xor_sync(mask, a, o);
          b += __shfl_xor_sync(mask, b, o);
          g += __shfl_xor_sync(mask, g, o);
        }
        // the cosine, without the square of a small column's square
        const float cosine = fabsf(g) * rsqrtf(a) * rsqrtf(b);
        if (cosine > 3e-7f && a > 0.f && b > 0.f) {
          worst = fmaxf(worst, cosine);
          // t = tan of the angle = h / (d + sign(d) sqrt(d^2 + h^2)) with d = b - a, h = 2 g, scaled
          const float d = b - a, h = 2.0f * g, m = __fdividef(1.0f, fmaxf(fabsf(d), fabsf(h)));
          const float ds = d * m, hs = h * m, w = fmaf(ds, ds, hs * hs);
          const float t = __fdividef(hs, ds + copysignf(w * rsqrtf(w), ds));
          const float c = rsqrtf(fmaf(t, t, 1.0f)), s = c * t;
#pragma unroll
          for (int k = 0; k < EPL; ++k) {
            wp[k * L] = c * x[k] - s * y[k];
            wq[k * L] = s * x[k] + c * y[k];
          }
        }
      }
      if (u != 0 && ++u == nn) u = 1;
      if (++v == nn) v = 1;
      __syncthreads();
    }
    const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(worst));
    if (lane == 0) atomicMax(&cmax, w);
    __syncthreads();
    const float left = __uint_as_float(cmax);
    __syncthreads();
    if (tid == 0) {
      cmax = 0u;
      if (sweep == 15 && left > 1e-4f) *bad = 1;
    }
    if (!(left > 1e-4f)) break;
  }
  __syncthreads();
  for (int j = gid; j < n; j += nt / L) {
    float a = 0.f;
    for (int i = gl; i < n; i += L) a = fmaf(wf[j * ld + i], wf[j * ld + i], a);
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) a += __shfl_xor_sync(mask, a, o);
    if (gl == 0) nrm[j] = sqrtf(a);
  }
  __syncthreads();
  for (int j = gid; j < n; j += nt / L) {
    const float sj = nrm[j];
    int rk = 0;
    for (int i = gl; i < n; i += L) {
      const float si = nrm[i];
      rk += (si > sj) || (si == sj && i < j) ? 1 : 0;
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) rk += __shfl_xor_sync(mask, rk, o);
    const float inv = 1.0f / sj;
    if (gl == 0) {
      if (!(sj > 1e-18f) || !(sj < 1e18f)) *bad = 1;
      sig[rk] = (double)sj;
      inv_sig[rk] = 1.0 / ((double)sj * up);
      if (j == 0) *scale = up;
    }
    for (int i = gl; i < n; i += L) X[(int64_t)rk * n + i] = (double)(wf[j * ld + i] * inv);
  }
}

// E = G - I into G, both triangles, from the lower (column-major) triangle of G. One block. *bad = 1
// when ||E||_F > 2e-4 (the polar factor below is then not orthonormal to rounding).
__global__ void __launch_bounds__(1024) polar_error_kernel(double* G, int n, int* bad) {
  stream_wait();
  __shared__ float sums[32];
  float s = 0.f;
  for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
    const int j = t / n, i = t - j * n;
    if (i < j) continue;
    const double e = G[t] - (i == j ? 1.0 : 0.0);
    G[t] = e;
    if (i != j) G[(int64_t)i * n + j] = e;
    const float f = (float)e;
    s = fmaf(f, i == j ? f : 2.0f * f, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w) s += sums[w];
    if (!(s <= 4e-8f)) *bad = 1;
  }
}

// P = I - E / 2 + 3/8 F (column-major n x n)
__global__ void polar_start_kernel(const double* E, const double* F, double* P,
                                   int n) {
  stream_wait();
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * n; t += gridDim.x * blockDim.x)
    P[t] = (t / n == t % n ? 1.0 : 0.0) + fma(0.375, F[t], -0.5 * E[t]);
}

// X[:, j] *= d[j] (column-major n x n); with T: T[i, j] = X[j, i] d[i] instead
__global__ void scale_cols_kernel(double* X, const double* d, int n, double* T) {
  stream_wait();
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * n; t += gridDim.x * blockDim.x) {
    const int j = t / n, i = t - j * n;
    const double v = X[t] * d[j];
    if (T) T[i * n + j] = v;
    else X[t] = v;
  }
}

// Grid-wide block Jacobi for larger n (W, V column-major n x n in global memory, L2-resident):
// one launch per round of the P-block tournament; CTA i rotates the cross pairs of the blocks
// rr(i, r) and rr(P-1-i, r) (and, in round 0, the pairs inside both), counting its rotations.
__global__ void __launch_bounds__(256) jacobi_grid_round_kernel(double* W, double* V, int n, int nb,
                                                                int P, int r, double tol,
                                                                unsigned* count) {
  stream_wait();
  const int i = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int bA = rr_index(i, r, P), bB = rr_index(P - 1 - i, r, P);
  int mine = 0;
  auto rotate = [&](int p, int q) {
    if (p > q) { const int t = p; p = q; q = t; }
    if (q >= n) return;
    double* wp = W + (int64_t)p * n;
    double* wq = W + (int64_t)q * n;
    double a = 0.0, b = 0.0, g = 0.0;
    for (int k = lane; k < n; k += 32) {
      const double x = wp[k], y = wq[k];
      a = fma(x, x, a); b = fma(y, y, b); g = fma(x, y, g);
    }
    a = red::warp_sum(a); b = red::warp_sum(b); g = red::warp_sum(g);
    double c, sn;
    if (!jacobi_rotation(a, b, g, tol, c, sn)) return;
    double* vp = V + (int64_t)p * n;
    double* vq = V + (int64_t)q * n;
    for (int k = lane; k < n; k += 32) {
      const double x = wp[k], y = wq[k];
      wp[k] = c * x - sn * y;
      wq[k] = sn * x + c * y;
      const double u = vp[k], v = vq[k];
      vp[k] = c * u - sn * v;
      vq[k] = sn * u + c * v;
    }
    ++mine;
  };
  if (r == 0) {   // pairs inside each of the two blocks
    const int m2 = nb + (nb & 1);
    for (int t = 0; t < m2 - 1; ++t) {
      for (int task = warp; task < m2; task += nw) {
        const int sl = task / (m2 / 2), pi = task % (m2 / 2);
        const int p = rr_index(pi, t, m2), q = rr_index(m2 - 1 - pi, t, m2);
        if (p >= nb || q >= nb) continue;
        const int base = (sl ? bB : bA) * nb;
        rotate(base + p, base + q);
      }
      __syncthreads();
    }
  }
  for (int t = 0; t < nb; ++t) {
    for (int j = warp; j < nb; j += nw) rotate(bA * nb + j, bB * nb + (j + t) % nb);
    __syncthreads();
  }
  if (lane == 0 && mine) atomicAdd(count, (unsigned)mine);
}

__global__ void identity_kernel(double* V, int n) {
  stream_wait();
  const int64_t total = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    V[t] = (t % n == t / n) ? 1.0 : 0.0;
}

// From the rotated W (column-major n x n) and the rotations V: sigma_j = ||W_j||, descending order;
// Un[:, rank_j] = W_j / sigma_j, Vs[:, rank_j] = V_j, S[rank_j] = sigma_j *scale. One block.
__global__ void __launch_bounds__(1024) svd_sort_kernel(const double* W,
                                                        const double* V, int n,
                                                        double* Un, double* S, double* Vs,
                                                        double* sig, const double* scale) {
  stream_wait();
  __shared__ int rank_sh[1024];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int j = warp; j < n; j += nw) {
    double a = 0.0;
    for (int i = lane; i < n; i += 32) a = fma(W[(int64_t)j * n + i], W[(int64_t)j * n + i], a);
    a = red::warp_sum(a);
    if (lane == 0) sig[j] = sqrt(a);
  }
  __syncthreads();
  for (int j = tid; j < n; j += nt) {
    const double sj = sig[j];
    int rk = 0;
    for (int i = 0; i < n; ++i) {
      const double si = sig[i];
      rk += (si > sj) || (si == sj && i < j);
    }
    rank_sh[j] = rk;
  }
  __syncthreads();
  const double up = *scale;
  for (int j = tid; j < n; j += nt) S[rank_sh[j]] = sig[j] * up;
  for (int j = warp; j < n; j += nw) {
    const int rk = rank_sh[j];
    const double inv = sig[j] > 0.0 ? 1.0 / sig[j] : 0.0;
    for (int i = lane; i < n; i += 32) {
      Un[(int64_t)rk * n + i] = W[(int64_t)j * n + i] * inv;
      Vs[(int64_t)rk * n + i] = V[(int64_t)j * n + i];
    }
  }
}

__global__ void gemv_rm_kernel(const double* B, int64_t n, const double* x,
                               double* y) {
  stream_wait();
  const int lane = threadIdx.x & 31;
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  double s = 0.0;
  for (int64_t c = lane; c < n; c += 32) s = fma(B[row * n + c], x[c], s);
  s = red::warp_sum(s);
  if (lane == 0) y[row] = s;
}

__global__ void copy_cm_kernel(const double* A, int64_t lda, double* W, int64_t m,
                               int64_t n) {
  stream_wait();
  const int64_t total = m * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % m, j = t / m;
    W[t] = A[j * lda + i];
  }
}

void householder(const double* A, int64_t lda, int64_t m, int64_t n, double* Q, double* R,
                 LinalgWS& ws, cudaStream_t s) {
  const int64_t k = m < n ? m : n;
  const size_t smem = (size_t)(m * n + m * k + k) * sizeof(double);
  if (smem <= (size_t)kHouseholderSmemBytes) {
    smem_optin((const void*)householder_smem_kernel, kHouseholderSmemBytes);
    launch_early(householder_smem_kernel, 1, 512, smem, s, A, lda, (int)m, (int)n, Q, R);
    TTGB_CHECK_LAUNCH();
    return;
  }
  ws.d.ensure(m * n + k + 16, s);
  double* W = ws.d.p;
  double* tau = W + m * n;
  unsigned g = cdiv(m * n, 256);
  if (g > 4096) g = 4096;
  if (g == 0) g = 1;
  launch_early(copy_cm_kernel, g, 256, 0, s, A, lda, W, m, n);
  TTGB_CHECK_LAUNCH();
  launch_early(householder_kernel, 1, 512, 0, s, W, (int)m, (int)n, Q, R, tau);
  TTGB_CHECK_LAUNCH();
}

}  // namespace

void qr_r(const double* A, int64_t lda, int64_t m, int64_t n, double* R, LinalgWS& ws,
          cudaStream_t s) {
  if (m <= 0 || n <= 0) return;
  TTGB_REQUIRE(n <= 4096, "qr_r: too many columns");
  const int mb = (int)std::max<int64_t>(2 * n, 256);
  const int64_t nblk = (m + mb - 1) / mb;
  TTGB_REQUIRE(nblk < 65536, "qr_r: too many row blocks");
  const int64_t per0 = (int64_t)mb * n;
  ws.d.ensure((size_t)(per0 * nblk + 2 * n * n * ((nblk + 1) / 2) + 16), s);
  ws.e.ensure((size_t)(n * n * nblk + 16), s);
  double* W = ws.d.p;
  double* Rb = ws.e.p;
  unsigned g = cdiv(per0 * nblk, 256);
  if (g > 8192) g = 8192;
  tsqr_gather_kernel<<<g, 256, 0, s>>>(A, lda, m, (int)n, mb, (int)nblk, W);
  TTGB_CHECK_LAUNCH();
  householder_r_kernel<<<(unsigned)nblk, 512, 0, s>>>(W, per0, mb, (int)n, Rb);
  TTGB_CHECK_LAUNCH();
  int64_t cur = nblk;
  while (cur > 1) {
    const int64_t nxt = (cur + 1) / 2;
    const int64_t per = 2 * n * n;
    unsigned g2 = cdiv(per * nxt, 256);
    if (g2 > 8192) g2 = 8192;
    tsqr_stack_kernel<<<g2, 256, 0, s>>>(Rb, (int)n, (int)cur, W);
    TTGB_CHECK_LAUNCH();
    householder_r_kernel<<<(unsigned)nxt, 512, 0, s>>>(W, per, (int)(2 * n), (int)n, Rb);
    TTGB_CHECK_LAUNCH();
    cur = nxt;
  }
  copy(Rb, R, n * n, s);
}

void gemm_cm(const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
             int64_t m, int64_t n, int64_t k, double alpha, double beta, cudaStream_t s,
             bool transA, bool transB, int tri, bool c_zero) {
  ContractDesc c;
  c.M = (int)m; c.N = (int)n; c.K = (int)k;
  c.A = A;
  if (!transA) { c.am = Ax::one(1); c.ak = Ax::one(lda); }
  else { c.am = Ax::one(lda); c.ak = Ax::one(1); }
  c.B = B;
  if (!transB) { c.bk = Ax::one(1); c.bn = Ax::one(ldb); }
  else { c.bk = Ax::one(ldb); c.bn = Ax::one(1); }
  c.C = C; c.cm = Ax::one(1); c.cn = Ax::one(ldc);
  c.alpha = alpha; c.beta = beta;
  c.tri = tri;
  c.c_zero = c_zero;
  contract(c, s);
}

QRResult qr(const double* A, int64_t lda, int64_t m, int64_t n, double* Q, double* R,
            LinalgWS& ws, const RedWS& red, cudaStream_t s) {
  (void)red;
  QRResult res;
  res.k = m < n ? m : n;
  if (m <= 0 || n <= 0) return res;
  // Wide and small factors have FP64 products whatever the engine of the calling thread: the bases of the mixed
  // path's enrichment are orthonormal to rounding.
  Fp64EngineScope engine(m < n || (m < 1024 && (double)m * n * n < 4e5) ? kFp64Native : fp64_engine());
  if (m < n) {
    // Wide: a factorisation of the leading m x m block has all of Q, whatever the block's rank; the other
    // columns of R are products. Against the sweep over the whole matrix: 3 x 6 18 -> 15 us, 5 x 8 31 -> 18, 8 x 12
    // 51 -> 19, 10 x 15 66 -> 27, 16 x 24 118 -> 30, 32 x 48 307 -> 73, 48 x 64 568 -> 110.
    qr(A, lda, m, m, Q, R, ws, red, s);
    gemm_cm(Q, m, A + m * lda, lda, R + m * m, m, m, n - m, m, 1.0, 0.0, s, true, false);
    return res;
  }
  if (n > 1024) {   // beyond CholeskyQR's factor: single-block Householder
    householder(A, lda, m, n, Q, R, ws, s);
    return res;
  }
  // One block's FP64 pipe does a pass of m n^2 multiply-adds while the launches of the grid-wide passes
  // cost about 30 us a pass, so the line lies where one pass fills that.
  if (n <= kCholQrSmallN && (double)m * n * n <= 3.5e4 && cholqr_small_smem(m, n) <= kHouseholderSmemBytes) {
    smem_optin((const void*)cholqr_small_kernel, kHouseholderSmemBytes);
    launch_early(cholqr_small_kernel, 1, 512, cholqr_small_smem(m, n), s, A, lda, (int)m, (int)n, Q, R);
    TTGB_CHECK_LAUNCH();
    return res;
  }
  // CholeskyQR2, or shifted CholeskyQR3
  ws.a.ensure(5 * n * n + 16, s);
  double* Rp[3] = {ws.a.p, ws.a.p + n * n, ws.a.p + 2 * n * n};   // R of each pass (row-major)
  double* Ri = ws.a.p + 3 * n * n;   // inverse of the current factor
  double* T1 = ws.a.p + 4 * n * n;   // R_1 R_0
  if (ws.gram.p == nullptr || ws.gram.n < (size_t)(n * n)) {   // (re)allocated: clear it once
    ws.gram.ensure((size_t)(n * n), s);
    TTGB_CUDA(cudaMemsetAsync(ws.gram.p, 0, ws.gram.n * sizeof(double), s));
    ws.gram_zero = (int64_t)ws.gram.n;
  }
  double* G = ws.gram.p;             // n x n Gram matrix (row-major upper triangle)
  ws.b.ensure(m * n + 16, s);
  double* Qt = ws.b.p;
  // words of ws.status: 0 the failure, 2 whether two passes were enough
  TTGB_CUDA(cudaMemsetAsync(ws.status, 0, 3 * sizeof(int), s));
  const double* Ain = A;
  int64_t ldin = lda;
  double* outs[3] = {Qt, Q, Qt};
  const bool smem_chol = n <= kCholSmemMax;
  int passes = 0;
  while (passes < 3) {
    const int pass = passes++;
    // Gram matrix: only its lower (column-major) = upper (row-major) triangle is formed and read;
    // with the shared-memory Cholesky the buffer is already zero (cleared by the previous one)
    gemm_cm(Ain, ldin, Ain, ldin, G, n, n, n, m, 1.0, 0.0, s, true, false, kTriLowerC,
            smem_chol && ws.gram_zero >= n * n);
    if (smem_chol) {
      const size_t smem = (size_t)n * (n + 1) * sizeof(double);
      smem_optin((const void*)chol_inv_smem_kernel,
                 (int)(kCholSmemMax * (kCholSmemMax + 1) * sizeof(double)));
      launch_early(chol_inv_smem_kernel, 1, 512, smem, s, G, (int)n, m, pass, Rp[pass], Ri, ws.status,
                                                ws.status + 2);
      TTGB_CHECK_LAUNCH();
      if (ws.gram_zero < n * n) ws.gram_zero = n * n;   // the kernel cleared [0, n^2)
    } else {
      launch_early(chol_kernel, 1, 512, 0, s, G, (int)n, pass == 0 ? m : 0, pass == 2 ? 1 : 0, ws.status);
      TTGB_CHECK_LAUNCH();
      launch_early(trinv_kernel, cdiv(n, 128), 128, 0, s, G, Ri, (int)n);
      TTGB_CHECK_LAUNCH();
      copy(G, Rp[pass], n * n, s);
      ws.gram_zero = 0;   // G now holds R
    }
    // Q_next = Ain * R^{-1}   (Ri row-major == (Ri)^T column-major; R^{-1} upper triangular)
    gemm_cm(Ain, ldin, Ri, n, outs[pass], m, m, n, n, 1.0, 0.0, s, false, true, kTriUpperB);
    Ain = outs[pass];
    ldin = m;
    // After an unshifted first pass the second one's Gram matrix is near the identity, and its Q is
    // orthonormal to rounding; the third pass is for a shifted start.
    if (pass > 0 && (smem_chol || pass == 2)) {
      TTGB_CUDA(cudaMemcpyAsync(ws.h_status, ws.status, 3 * sizeof(int), cudaMemcpyDeviceToHost, s));
      TTGB_CUDA(cudaStreamSynchronize(s));
      if (ws.h_status[0] != 0) {
        householder(A, lda, m, n, Q, R, ws, s);
        return res;
      }
      if (pass == 1 && ws.h_status[2] != 0) break;
    }
  }
  // R of the passes multiplied (row-major factors; a row-major X is the column-major X^T), the last
  // product written column-major
  if (passes == 2) {
    gemm_cm(Rp[1], n, Rp[0], n, R, n, n, n, n, 1.0, 0.0, s, true, true);
  } else {
    copy(Qt, Q, m * n, s);
    gemm_cm(Rp[0], n, Rp[1], n, T1, n, n, n, n, 1.0, 0.0, s, false, false);   // T1 = R_1 R_0, row-major
    gemm_cm(Rp[2], n, T1, n, R, n, n, n, n, 1.0, 0.0, s, true, true);
  }
  return res;
}

namespace {

template <int EPL>
void launch_jacobi_block(double* W, double* V, int n, size_t smem, int* status, cudaStream_t s) {
  smem_optin((const void*)jacobi_block_kernel<EPL>, (int)smem);
  jacobi_block_kernel<EPL><<<kJacobiCluster, 256, smem, s>>>(W, n, W, V, 60, status);
  TTGB_CHECK_LAUNCH();
}

// FP64 one-sided Jacobi of the columns of W (n x n column-major, n >= 2 kJacobiCluster, rotated in
// place; V: n x n scratch): W V = Un diag(S) / *scale, S descending, the rotations in Vs.
void jacobi_columns(double* W, double* V, int64_t n, const double* scale, double* Un, double* S, double* Vs,
                    LinalgWS& ws, cudaStream_t s) {
  if (n <= kJacobiBlockMaxN) {
    const int nb = (int)((n + 2 * kJacobiCluster - 1) / (2 * kJacobiCluster));
    const int64_t unit = 2 * nb * n + nb + (nb & 1);
    const size_t smem = (size_t)4 * unit * sizeof(double);
    if (n <= 32) launch_jacobi_block<1>(W, V, (int)n, smem, ws.status, s);
    else if (n <= 64) launch_jacobi_block<2>(W, V, (int)n, smem, ws.status, s);
    else if (n <= 96) launch_jacobi_block<3>(W, V, (int)n, smem, ws.status, s);
    else launch_jacobi_block<5>(W, V, (int)n, smem, ws.status, s);
  } else {   // grid-wide block Jacobi, one launch per round
    const int sms = num_sms();
    const int nb = (int)std::max<int64_t>(1, (n + 2 * sms - 1) / (2 * sms));
    int P = (int)((n + nb - 1) / nb);
    P += P & 1;
    launch_early(identity_kernel, cdiv((int64_t)n * n, 256), 256, 0, s, V, (int)n);
    TTGB_CHECK_LAUNCH();
    DevBuf<unsigned> cnt(1, s);
    unsigned hcnt = 0;
    const double tol = std::max((double)n, 1.0) * kEps;
    int sweep = 0;
    for (; sweep < 60; ++sweep) {
      TTGB_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(unsigned), s));
      for (int r = 0; r < P - 1; ++r) {
        launch_early(jacobi_grid_round_kernel, P / 2, 256, 0, s, W, V, (int)n, nb, P, r, tol, cnt.p);
        TTGB_CHECK_LAUNCH();
      }
      TTGB_CUDA(cudaMemcpyAsync(&hcnt, cnt.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
      TTGB_CUDA(cudaStreamSynchronize(s));
      if (hcnt == 0) break;
    }
    if (sweep >= 60) TTGB_CUDA(cudaMemsetAsync(ws.status, 0x03, 1, s));
  }
  DBuf sig((size_t)n, s);
  launch_early(svd_sort_kernel, 1, 1024, 0, s, W, V, (int)n, Un, S, Vs, sig.p, scale);
  TTGB_CHECK_LAUNCH();
}

template <int EPL>
void launch_jacobi_f32(const double* R, int n, double* X, double* sig, int* bad, cudaStream_t s) {
  const int smem = 8 * EPL * jacobi_f32_pitch(EPL) * (int)sizeof(float);
  smem_optin((const void*)jacobi_f32_kernel<EPL>, smem);
  launch_early(jacobi_f32_kernel<EPL>, 1, cdiv((n + 1) / 2 * 8, 32) * 32, smem, s, R, n, X, sig, sig + n, sig + 2 * n,
                                                                           bad);
  TTGB_CHECK_LAUNCH();
}

// From here on the preconditioned route is the faster one (n = 16: 256 against 460 us).
constexpr int64_t kPreconditionMinN = 16;

// A start for the FP64 Jacobi from FP32: X (n x n, orthonormal to FP64 rounding, followed by n
// estimates of the singular values of the scaled R, the n reciprocals for R itself, and the scale) holds R's right singular vectors to FP32
// accuracy, and B = R X diag(1 / sigma), whose columns are nearly orthonormal. The QR factor L of R X is
// then so near to diagonal, whatever the grading, that Jacobi on L^T takes two or three sweeps where
// it takes nine on R^T (FP32 rotations alone leave six to ten sweeps for a graded R, whose small
// columns drown in the FP32 rounding of the large ones; the QR step removes that). Returns false
// when the FP32 sweeps cannot be used (R zero, not finite or numerically singular beyond FP32).
bool precondition(const double* R, int64_t n, DBuf& X, DBuf& B, LinalgWS& ws, const RedWS& red,
                  cudaStream_t s) {
  (void)red;
  X.reset((size_t)(n * n + 2 * n + 1), s);
  B.reset((size_t)(n * n), s);
  DBuf X0((size_t)(n * n), s), G((size_t)(n * n), s), P((size_t)(n * n), s);
  double* sig = X.p + n * n;
  double* inv = sig + n;
  int* bad = ws.status + 3;
  TTGB_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s));
  if (n <= 32) launch_jacobi_f32<4>(R, (int)n, X0.p, sig, bad, s);
  else if (n <= 64) launch_jacobi_f32<8>(R, (int)n, X0.p, sig, bad, s);
  else if (n <= 80) launch_jacobi_f32<10>(R, (int)n, X0.p, sig, bad, s);
  else if (n <= 112) launch_jacobi_f32<14>(R, (int)n, X0.p, sig, bad, s);
  else if (n <= 160) launch_jacobi_f32<20>(R, (int)n, X0.p, sig, bad, s);
  else launch_jacobi_f32<28>(R, (int)n, X0.p, sig, bad, s);
  // X = X0 (I - E/2 + 3/8 E^2 - 5/16 E^3) with E = X0^T X0 - I: the polar factor to fourth order
  gemm_cm(X0.p, n, X0.p, n, G.p, n, n, n, n, 1.0, 0.0, s, true, false, kTriLowerC);
  launch_early(polar_error_kernel, 1, 1024, 0, s, G.p, (int)n, bad);
  TTGB_CHECK_LAUNCH();
  gemm_cm(G.p, n, G.p, n, B.p, n, n, n, n, 1.0, 0.0, s);
  launch_early(polar_start_kernel, cdiv(n * n, 256), 256, 0, s, G.p, B.p, P.p, (int)n);
  TTGB_CHECK_LAUNCH();
  gemm_cm(B.p, n, G.p, n, P.p, n, n, n, n, -0.3125, 1.0, s);
  gemm_cm(X0.p, n, P.p, n, X.p, n, n, n, n, 1.0, 0.0, s);
  gemm_cm(R, n, X.p, n, B.p, n, n, n, n, 1.0, 0.0, s);
  launch_early(scale_cols_kernel, cdiv(n * n, 256), 256, 0, s, B.p, inv, (int)n, nullptr);
  TTGB_CHECK_LAUNCH();
  TTGB_CUDA(cudaMemcpyAsync(ws.h_status, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  TTGB_CUDA(cudaStreamSynchronize(s));
  return *ws.h_status == 0;
}

}  // namespace

void svd(const double* A, int64_t lda, int64_t m, int64_t n, double* U, double* S, double* Vh,
         LinalgWS& ws, const RedWS& red, cudaStream_t s) {
  if (m <= 0 || n <= 0) return;
  if (m < n) {
    // A^T = U' S V'^T  ->  A = V' S U'^T
    DBuf At((size_t)(n * m), s);
    transpose(A, lda, At.p, n, m, n, s);      // At (n x m col-major): At[j + i*n] = A[i + j*lda]
    // transpose() writes dst[r*dld + c] = src[c*sld + r] with rows=m? use explicit kernel via gemm
    DBuf Ut((size_t)(n * m), s), Vt((size_t)(m * m), s);
    svd(At.p, n, n, m, Ut.p, S, Vt.p, ws, red, s);
    // U = V' = Vt^T (m x m); Vh = U'^T (m x n)
    transpose(Vt.p, m, U, m, m, m, s);
    transpose(Ut.p, n, Vh, m, n, m, s);
    return;
  }
  // m >= n: A = Q R; one-sided Jacobi on R^T (QR-preconditioned Jacobi, Drmac & Veselic, SIAM J.
  // Matrix Anal. Appl. 29, 2008): R^T = U' S V'^T converges in far fewer sweeps than Jacobi on R.
  // Then R = V' S U'^T and A = (Q V') S U'^T.
  DBuf Qb((size_t)(m * n), s), Rb((size_t)(n * n), s);
  qr(A, lda, m, n, Qb.p, Rb.p, ws, red, s);
  TTGB_REQUIRE(n <= 1024, "SVD: too many columns");
  if (n >= kPreconditionMinN && n <= kJacobiF32MaxN) {
    DBuf X, B;
    if (precondition(Rb.p, n, X, B, ws, red, s)) {
      // R X = Q2 L with L^T = U'' S V''^T:  A = (Q Q2 V'') S (X U'')^T
      DBuf Q2((size_t)(n * n), s), T((size_t)(n * n), s), Un((size_t)(n * n), s);
      DBuf Vs((size_t)(n * n), s);
      const double* sig = X.p + n * n;
      qr(B.p, n, n, n, Q2.p, T.p, ws, red, s);
      ws.c.ensure(3 * n * n + 16, s);
      launch_early(scale_cols_kernel, cdiv(n * n, 256), 256, 0, s, T.p, sig, (int)n, ws.c.p);
      TTGB_CHECK_LAUNCH();
      jacobi_columns(ws.c.p, ws.c.p + n * n, n, sig + 2 * n, Un.p, S, Vs.p, ws, s);
      gemm_cm(Q2.p, n, Vs.p, n, T.p, n, n, n, n, 1.0, 0.0, s);
      gemm_cm(Qb.p, m, T.p, n, U, m, m, n, n, 1.0, 0.0, s);
      gemm_cm(Un.p, n, X.p, n, Vh, n, n, n, n, 1.0, 0.0, s, true, true);
      return;
    }
  }
  ws.c.ensure(3 * n * n + 16, s);
  double* Vs = ws.c.p;           // V'
  DBuf Up((size_t)(n * n), s);   // U' (normalised columns of the rotated R^T, sorted)
  if (n < kJacobiWarpMaxN) {
    launch_early(jacobi_warp_kernel, 1, 32, 0, s, Rb.p, (int)n, Up.p, S, Vs, ws.status);
    TTGB_CHECK_LAUNCH();
  } else {
    double* W = Vs + n * n;      // R^T, rotated in place
    double* scale = W + 2 * n * n;
    launch_early(scaled_transpose_kernel, 1, 1024, 0, s, Rb.p, (int)n, W, scale);
    TTGB_CHECK_LAUNCH();
    jacobi_columns(W, W + n * n, n, scale, Up.p, S, Vs, ws, s);
  }
  gemm_cm(Qb.p, m, Vs, n, U, m, m, n, n, 1.0, 0.0, s);   // U = Q V'
  transpose(Up.p, n, Vh, n, n, n, s);                    // Vh = U'^T
}

void gemv(const double* B, int64_t n, const double* x, double* y, cudaStream_t s) {
  if (n <= 0) return;
  launch_early(gemv_rm_kernel, cdiv(n * 32, 256), 256, 0, s, B, n, x, y);
  TTGB_CHECK_LAUNCH();
}

}  // namespace ttgb
