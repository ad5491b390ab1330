// FP64 dense linear algebra: shifted CholeskyQR3 with a Householder fallback, one-sided Jacobi
// thin SVD.
//
// GB300 note: FP64 runs at ~1.9 FMA/clock/SM (measured), so every O(m n^2) step is expressed as a
// GEMM on the contraction engine (spread over all SMs); only O(n^3) steps on the small n x n
// factors run on few SMs: Cholesky + triangular inverse and the Jacobi of n < 16 in one thread
// block, the block Jacobi of 16 <= n <= 160 on an 8-CTA cluster, larger ones one grid-wide round
// per launch. Small QRs (the kickrank-wide blocks) run a shared-memory Householder in one block.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "contract.cuh"
#include "linalg.cuh"

namespace cg = cooperative_groups;

namespace ttgb {

namespace {

constexpr double kEps = 2.220446049250313e-16;

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ double block_sum_d(double v, double* sh) {
  v = warp_sum_d(v);
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

// 1 / sqrt(d) for d in the FP32 range: y from FP32, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - d y^2
__device__ __forceinline__ double rsqrt_refined(double d) {
  const double y = (double)rsqrtf((float)d);
  const double e = fma(-d * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

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
    tr = warp_sum_d(tr);
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
          for (int j = 0; j < kCholNb; ++j) {
            if (i == j) {
              const double d = __shfl_sync(0xffffffffu, v, j);
              if (!(d > floor_d) || !isfinite(d)) ch.bad = 1;   // the same in every lane
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

__global__ void __launch_bounds__(512) chol_inv_smem_kernel(double* __restrict__ Gin, int n,
                                                            int64_t shift_rows, int pass, double* Rout,
                                                            double* Riout, int* status, int* done) {
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
__global__ void trinv_kernel(const double* __restrict__ R, double* Ri, int n) {
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
        w = warp_sum_d(w) + c0;
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
      w = warp_sum_d(w) + q0;
      const double tw = tj * w;
      if (lane == 0) qc[j] -= tw;
      for (int i = j + 1 + lane; i < m; i += 32) qc[i] = fma(-tw, col[i], qc[i]);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(512) householder_kernel(double* W, int m, int n, double* Q,
                                                          double* R, double* tau) {
  householder_body(W, m, n, Q, R, tau);
}

// The same factorisation with W, Q and tau in shared memory (m * n + m * k + k doubles), read
// straight from A (ld lda): every step of the column sweep is a shared-memory access instead of an
// L2 round trip, which is what bounds the small QRs of the enrichment blocks (m <= 1024, n <= 16).
constexpr int kHouseholderSmemBytes = 200 * 1024;

__global__ void __launch_bounds__(512, 1) householder_smem_kernel(const double* __restrict__ A,
                                                               int64_t lda, int m, int n,
                                                               double* Qout, double* R) {
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

__global__ void __launch_bounds__(512, 1) cholqr_small_kernel(const double* __restrict__ A, int64_t lda,
                                                              int m, int n, double* Qout, double* Rout) {
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
        w = warp_sum_d(w) + c0;
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

// ---------------------------------------------------------------------------------------------
// One-sided (Hestenes) Jacobi SVD of the n x n column-major matrix W in one thread block, with
// the round-robin parallel ordering; rotation formulas of Demmel & Veselic (SIAM J. Matrix Anal.
// Appl. 13, 1992). On exit U (n x n) holds W_j / sigma_j, V the accumulated rotations, both with
// columns sorted by descending sigma, S the sorted singular values.
// ---------------------------------------------------------------------------------------------
// Rotation (c, s) of one-sided Jacobi for a column pair with squared norms a, b and inner product
// g (Demmel-Veselic formulas): false when the pair is orthogonal to `tol`. The tangent t of the
// angle comes from FP32 arithmetic (relative error ~1e-7: the pair is left orthogonal to ~1e-7 and
// a later sweep finishes it), and c = 1/sqrt(1 + t^2) is refined from the FP32 rsqrt to full FP64
// accuracy by two Newton steps, so (c, s) is orthogonal to rounding. On GB300 an FP64 sqrt or
// division is a sequence of DFMA on a pipe that issues one warp instruction per 16 cycles; the
// exact formula costs ~4 sqrt + 3 divisions per rotation, this one ~8 DFMA.
__device__ __forceinline__ bool jacobi_rotation(double a, double b, double g, double tol, double& c,
                                                double& s) {
  if (a == 0.0 || b == 0.0) return false;
  if (!(g * g > tol * tol * a * b)) return false;
  const double bma = b - a, g2 = 2.0 * g;
  const float fb = (float)bma, fg = (float)g2;
  float tf;
  if (fabsf(fb) >= fabsf(fg)) {   // r = 2g / (b - a), |r| <= 1: t = r / (1 + sqrt(1 + r^2))
    const float r = __fdividef(fg, fb);
    tf = __fdividef(r, 1.0f + sqrtf(fmaf(r, r, 1.0f)));
  } else {                        // zeta = (b - a) / 2g, |zeta| < 1
    const float z = __fdividef(fb, fg);
    tf = __fdividef(copysignf(1.0f, z), fabsf(z) + sqrtf(fmaf(z, z, 1.0f)));
  }
  double t;
  if (tf != 0.0f && isfinite(tf)) {
    t = (double)tf;
  } else {   // operands outside the FP32 range: the exact FP64 formula
    const double zeta = bma / g2;
    t = (fabs(zeta) > 1e150) ? 0.5 / zeta
                             : copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
  }
  const double x = fma(t, t, 1.0);
  double y = (double)rsqrtf((float)x);
  y = y * fma(-0.5 * x, y * y, 1.5);
  y = y * fma(-0.5 * x, y * y, 1.5);
  c = y;
  s = y * t;
  return true;
}

__device__ __forceinline__ double warp_sum_t(double v) { return warp_sum_d(v); }

__device__ __forceinline__ int rr_index(int p, int r, int nn) {
  return p == 0 ? 0 : ((p - 1 + r) % (nn - 1)) + 1;
}

__global__ void __launch_bounds__(512) jacobi_svd_kernel(double* Wg, double* Vg, int n, double* U,
                                                         double* S, int use_smem, int max_sweeps,
                                                         int* status, const double* Vinit) {
  extern __shared__ double smem[];
  __shared__ int nrot;
  double* W = use_smem ? smem : Wg;
  double* V = use_smem ? smem + (int64_t)n * n : Vg;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  if (use_smem) {
    for (int64_t t = tid; t < (int64_t)n * n; t += nt) W[t] = Wg[t];
  }
  for (int64_t t = tid; t < (int64_t)n * n; t += nt)
    V[t] = Vinit ? Vinit[t] : (((t % n) == (t / n)) ? 1.0 : 0.0);
  __syncthreads();
  const int nn = n + (n & 1);
  const double tol = fmax((double)n, 1.0) * kEps;
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (tid == 0) nrot = 0;
    __syncthreads();
    for (int r = 0; r < nn - 1; ++r) {
      for (int pi = warp; pi < nn / 2; pi += nw) {
        int p = rr_index(pi, r, nn), q = rr_index(nn - 1 - pi, r, nn);
        if (p > q) { const int t = p; p = q; q = t; }
        if (q >= n) continue;
        double* wp = W + (int64_t)p * n;
        double* wq = W + (int64_t)q * n;
        double a = 0.0, b = 0.0, g = 0.0;
        for (int i = lane; i < n; i += 32) {
          const double x = wp[i], y = wq[i];
          a = fma(x, x, a); b = fma(y, y, b); g = fma(x, y, g);
        }
        a = warp_sum_d(a); b = warp_sum_d(b); g = warp_sum_d(g);
        double c, s;
        if (!jacobi_rotation(a, b, g, tol, c, s)) continue;
        for (int i = lane; i < n; i += 32) {
          const double x = wp[i], y = wq[i];
          wp[i] = c * x - s * y;
          wq[i] = s * x + c * y;
        }
        double* vp = V + (int64_t)p * n;
        double* vq = V + (int64_t)q * n;
        for (int i = lane; i < n; i += 32) {
          const double x = vp[i], y = vq[i];
          vp[i] = c * x - s * y;
          vq[i] = s * x + c * y;
        }
        if (lane == 0) atomicAdd(&nrot, 1);
      }
      __syncthreads();
    }
    __syncthreads();
    if (nrot == 0) break;
    __syncthreads();
  }
  if (tid == 0 && sweep >= max_sweeps) *status = 3;
  // singular values, ranks by descending value (ties by index)
  double* sig = S;  // temporary: write unsorted to S via registers below
  for (int j = warp; j < n; j += nw) {
    const double* wj = W + (int64_t)j * n;
    double a = 0.0;
    for (int i = lane; i < n; i += 32) a = fma(wj[i], wj[i], a);
    a = warp_sum_d(a);
    if (lane == 0) U[(int64_t)j] = sqrt(a);   // stash sigma_j in U's first column temporarily
  }
  __syncthreads();
  // rank computation, then write sorted S (U column 0 is rewritten afterwards)
  __shared__ int rank_sh[1024];
  for (int j = tid; j < n; j += nt) {
    const double sj = U[j];
    int rk = 0;
    for (int i = 0; i < n; ++i) {
      const double si = U[i];
      rk += (si > sj) || (si == sj && i < j);
    }
    if (j < 1024) rank_sh[j] = rk;
  }
  __syncthreads();
  for (int j = tid; j < n; j += nt) sig[rank_sh[j]] = U[j];
  __syncthreads();
  // U[:, rank_j] = W_j / sigma_j ; V columns permuted into Wg (scratch) then copied back
  for (int j = warp; j < n; j += nw) {
    const int rk = rank_sh[j];
    const double sj = sig[rk];
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    const double* wj = W + (int64_t)j * n;
    for (int i = lane; i < n; i += 32) Vg[(int64_t)n * n + (int64_t)rk * n + i] = wj[i] * inv;
  }
  __syncthreads();
  for (int64_t t = tid; t < (int64_t)n * n; t += nt) U[t] = Vg[(int64_t)n * n + t];
  __syncthreads();
  for (int j = warp; j < n; j += nw) {
    const int rk = rank_sh[j];
    const double* vj = V + (int64_t)j * n;
    for (int i = lane; i < n; i += 32) Vg[(int64_t)n * n + (int64_t)rk * n + i] = vj[i];
  }
  __syncthreads();
  for (int64_t t = tid; t < (int64_t)n * n; t += nt) Vg[t] = Vg[(int64_t)n * n + t];
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
// rotation count is summed in CTA 0 after a barrier and read by every CTA, so all CTAs leave the
// loop together. The value type T is the arithmetic of the sweeps; Vin (optional) gives starting
// rotations (identity when null), Vout the accumulated ones.
// ---------------------------------------------------------------------------------------------
constexpr int kJacobiCluster = 8;
constexpr int kJacobiBlockMaxN = 160;

// One rotation of a column pair with tracked squared column norms (*na, *nb): only the inner product is
// reduced; the norms follow the rotation exactly (a' = c^2 a - 2cs g + s^2 b, b' = s^2 a + 2cs g +
// c^2 b) and are recomputed from the columns once per sweep, which bounds their drift.
template <typename T>
__device__ __forceinline__ int jacobi_rotate_tracked(T* wp, T* wq, T* vp, T* vq, T* na, T* nb, int n,
                                                     T tol, int lane) {
  T g = T(0);
  for (int i = lane; i < n; i += 32) g = fma(wp[i], wq[i], g);
  g = warp_sum_t(g);
  const T a = *na, b = *nb;
  T c, s;
  if (!jacobi_rotation(a, b, g, tol, c, s)) return 0;
  for (int i = lane; i < n; i += 32) {
    const T x = wp[i], y = wq[i];
    wp[i] = c * x - s * y;
    wq[i] = s * x + c * y;
    const T u = vp[i], v = vq[i];
    vp[i] = c * u - s * v;
    vq[i] = s * u + c * v;
  }
  if (lane == 0) {
    const T cc = c * c, ss = s * s, cs2 = T(2) * c * s * g;
    const T a2 = cc * a - cs2 + ss * b, b2 = ss * a + cs2 + cc * b;
    *na = a2 > T(0) ? a2 : T(0);
    *nb = b2 > T(0) ? b2 : T(0);
  }
  return 1;
}

template <typename T>
__global__ void __cluster_dims__(kJacobiCluster, 1, 1) __launch_bounds__(256)
    jacobi_block_kernel(const T* __restrict__ Win, int n, T* Wout, T* Vout, int max_sweeps,
                        int* status, const T* __restrict__ Vin) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T* sm = reinterpret_cast<T*>(sm_raw);
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int C = kJacobiCluster, P = 2 * kJacobiCluster;
  const int rank = (int)cluster.block_rank();
  const int nb = (n + P - 1) / P;
  const int64_t blk = (int64_t)nb * n;   // elements of one block of W (or of V)
  const int64_t unit = 2 * blk + nb + (nb & 1);   // W block, V block, squared column norms
  // buffer x (0/1), slot s (0/1): W block, V block, norms
  auto Wb = [&](T* base, int x, int sl) { return base + (int64_t)(x * 2 + sl) * unit; };
  auto Vb = [&](T* base, int x, int sl) { return base + (int64_t)(x * 2 + sl) * unit + blk; };
  auto Nb = [&](T* base, int x, int sl) { return base + (int64_t)(x * 2 + sl) * unit + 2 * blk; };
  __shared__ int counts[kJacobiCluster];
  __shared__ int local_cnt;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const T tol = T(n > 1 ? n : 1) * (sizeof(T) == 8 ? T(kEps) : T(1.1920929e-7f));
  // round 0 of sweep 0: slot 0 holds block rank, slot 1 block P-1-rank
  for (int sl = 0; sl < 2; ++sl) {
    const int b = sl == 0 ? rank : P - 1 - rank;
    T* W = Wb(sm, 0, sl);
    T* V = Vb(sm, 0, sl);
    for (int64_t t = tid; t < blk; t += nt) {
      const int j = (int)(t / n), i = (int)(t - (int64_t)j * n);
      const int c = b * nb + j;
      W[t] = (c < n) ? Win[(int64_t)c * n + i] : T(0);
      V[t] = (c < n) ? (Vin ? Vin[(int64_t)c * n + i] : (i == c ? T(1) : T(0))) : T(0);
    }
  }
  int* counts0 = cluster.map_shared_rank(counts, 0);
  int x = 0, r = 0, sweep = 0, mine = 0;
  bool converged = false;
  if (tid == 0) local_cnt = 0;
  __syncthreads();
  while (true) {
    const int bA = rr_index(rank, r, P), bB = rr_index(P - 1 - rank, r, P);
    T* WA = Wb(sm, x, 0); T* VA = Vb(sm, x, 0); T* NA = Nb(sm, x, 0);
    T* WB = Wb(sm, x, 1); T* VB = Vb(sm, x, 1); T* NB = Nb(sm, x, 1);
    if (r == 0) {   // fresh column norms, then the pairs inside each block, once per sweep
      for (int c = warp; c < 2 * nb; c += nw) {
        const T* w = (c < nb ? WA : WB) + (int64_t)(c % nb) * n;
        T a = T(0);
        for (int i = lane; i < n; i += 32) a = fma(w[i], w[i], a);
        a = warp_sum_t(a);
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
          T* W = sl ? WB : WA;
          T* V = sl ? VB : VA;
          T* Nm = sl ? NB : NA;
          mine += jacobi_rotate_tracked(W + (int64_t)p * n, W + (int64_t)q * n, V + (int64_t)p * n,
                                        V + (int64_t)q * n, Nm + p, Nm + q, n, tol, lane);
        }
        __syncthreads();
      }
    }
    for (int t = 0; t < nb; ++t) {   // cross pairs (j, j + t mod nb)
      for (int j = warp; j < nb; j += nw) {
        const int k = (j + t) % nb;
        const int ga = bA * nb + j, gb = bB * nb + k;
        T *wp = WA + (int64_t)j * n, *wq = WB + (int64_t)k * n;
        T *vp = VA + (int64_t)j * n, *vq = VB + (int64_t)k * n;
        T *np = NA + j, *nq = NB + k;
        if (ga > gb) {
          T* u = wp; wp = wq; wq = u; u = vp; vp = vq; vq = u; u = np; np = nq; nq = u;
        }
        mine += jacobi_rotate_tracked(wp, wq, vp, vq, np, nq, n, tol, lane);
      }
      __syncthreads();
    }
    const bool sweep_end = (r == P - 2);
    if (sweep_end) {
      if (lane == 0 && mine) atomicAdd(&local_cnt, mine);
      mine = 0;
      __syncthreads();
      if (tid == 0) { counts0[rank] = local_cnt; local_cnt = 0; }
    }
    cluster.sync();   // every CTA finished round r (and published its count at a sweep end)
    if (sweep_end) {
      int total = 0;
      for (int c = 0; c < C; ++c) total += counts0[c];
      ++sweep;
      if (total == 0) { converged = true; break; }
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
      const T* srcW = cluster.map_shared_rank(Wb(sm, x, oslot), owner);
      const T* srcV = cluster.map_shared_rank(Vb(sm, x, oslot), owner);
      const T* srcN = cluster.map_shared_rank(Nb(sm, x, oslot), owner);
      T* dW = Wb(sm, 1 - x, sl);
      T* dV = Vb(sm, 1 - x, sl);
      T* dN = Nb(sm, 1 - x, sl);
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
    const T* W = Wb(sm, x, sl);
    const T* V = Vb(sm, x, sl);
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

// Grid-wide block Jacobi for larger n (W, V column-major n x n in global memory, L2-resident):
// one launch per round of the P-block tournament; CTA i rotates the cross pairs of the blocks
// rr(i, r) and rr(P-1-i, r) (and, in round 0, the pairs inside both), counting its rotations.
__global__ void __launch_bounds__(256) jacobi_grid_round_kernel(double* W, double* V, int n, int nb,
                                                                int P, int r, double tol,
                                                                unsigned* count) {
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
    a = warp_sum_d(a); b = warp_sum_d(b); g = warp_sum_d(g);
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
  const int64_t total = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    V[t] = (t % n == t / n) ? 1.0 : 0.0;
}

// From the rotated W (column-major n x n) and the rotations V: sigma_j = ||W_j||, descending order;
// Un[:, rank_j] = W_j / sigma_j, Vs[:, rank_j] = V_j, S[rank_j] = sigma_j. One block.
__global__ void __launch_bounds__(1024) svd_sort_kernel(const double* __restrict__ W,
                                                        const double* __restrict__ V, int n,
                                                        double* Un, double* S, double* Vs,
                                                        double* sig) {
  __shared__ int rank_sh[1024];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int j = warp; j < n; j += nw) {
    double a = 0.0;
    for (int i = lane; i < n; i += 32) a = fma(W[(int64_t)j * n + i], W[(int64_t)j * n + i], a);
    a = warp_sum_d(a);
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
  for (int j = tid; j < n; j += nt) S[rank_sh[j]] = sig[j];
  for (int j = warp; j < n; j += nw) {
    const int rk = rank_sh[j];
    const double inv = sig[j] > 0.0 ? 1.0 / sig[j] : 0.0;
    for (int i = lane; i < n; i += 32) {
      Un[(int64_t)rk * n + i] = W[(int64_t)j * n + i] * inv;
      Vs[(int64_t)rk * n + i] = V[(int64_t)j * n + i];
    }
  }
}

__global__ void gemv_rm_kernel(const double* __restrict__ B, int64_t n, const double* __restrict__ x,
                               double* y) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  double s = 0.0;
  for (int64_t c = lane; c < n; c += 32) s = fma(B[row * n + c], x[c], s);
  s = warp_sum_d(s);
  if (lane == 0) y[row] = s;
}

__global__ void copy_cm_kernel(const double* __restrict__ A, int64_t lda, double* W, int64_t m,
                               int64_t n) {
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
    householder_smem_kernel<<<1, 512, smem, s>>>(A, lda, (int)m, (int)n, Q, R);
    TTGB_CHECK_LAUNCH();
    return;
  }
  ws.d.ensure(m * n + k + 16, s);
  double* W = ws.d.p;
  double* tau = W + m * n;
  unsigned g = cdiv(m * n, 256);
  if (g > 4096) g = 4096;
  if (g == 0) g = 1;
  copy_cm_kernel<<<g, 256, 0, s>>>(A, lda, W, m, n);
  TTGB_CHECK_LAUNCH();
  householder_kernel<<<1, 512, 0, s>>>(W, (int)m, (int)n, Q, R, tau);
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
  if (m < n || n > 1024) {   // wide, or beyond CholeskyQR's factor: single-block Householder
    householder(A, lda, m, n, Q, R, ws, s);
    return res;
  }
  // One block's FP64 pipe does a pass of m n^2 multiply-adds while the launches of the grid-wide passes
  // cost about 30 us a pass, so the line lies where one pass fills that.
  if (n <= kCholQrSmallN && (double)m * n * n <= 3.5e4 && cholqr_small_smem(m, n) <= kHouseholderSmemBytes) {
    smem_optin((const void*)cholqr_small_kernel, kHouseholderSmemBytes);
    cholqr_small_kernel<<<1, 512, cholqr_small_smem(m, n), s>>>(A, lda, (int)m, (int)n, Q, R);
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
      chol_inv_smem_kernel<<<1, 512, smem, s>>>(G, (int)n, m, pass, Rp[pass], Ri, ws.status,
                                                ws.status + 2);
      TTGB_CHECK_LAUNCH();
      if (ws.gram_zero < n * n) ws.gram_zero = n * n;   // the kernel cleared [0, n^2)
    } else {
      chol_kernel<<<1, 512, 0, s>>>(G, (int)n, pass == 0 ? m : 0, pass == 2 ? 1 : 0, ws.status);
      TTGB_CHECK_LAUNCH();
      trinv_kernel<<<cdiv(n, 128), 128, 0, s>>>(G, Ri, (int)n);
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
  ws.c.ensure(3 * n * n + 16, s);
  double* W = ws.c.p;        // n x n: R^T, rotated in place
  double* Vw = W + n * n;    // 2 n x n: accumulated rotations V' (sorted) and scratch
  transpose(Rb.p, n, W, n, n, n, s);
  DBuf Up((size_t)(n * n), s);   // U' (normalised columns of the rotated R^T, sorted)
  if (n <= kJacobiBlockMaxN && n >= 2 * kJacobiCluster) {
    const int nb = (int)((n + 2 * kJacobiCluster - 1) / (2 * kJacobiCluster));
    const int64_t unit = 2 * nb * n + nb + (nb & 1);
    const size_t smem = (size_t)4 * unit * sizeof(double);
    smem_optin((const void*)jacobi_block_kernel<double>, (int)smem);
    jacobi_block_kernel<double><<<kJacobiCluster, 256, smem, s>>>(W, (int)n, W, Vw, 60, ws.status,
                                                                  nullptr);
    TTGB_CHECK_LAUNCH();
    DBuf sig((size_t)n, s);
    svd_sort_kernel<<<1, 1024, 0, s>>>(W, Vw, (int)n, Up.p, S, Vw + n * n, sig.p);
    TTGB_CHECK_LAUNCH();
    gemm_cm(Qb.p, m, Vw + n * n, n, U, m, m, n, n, 1.0, 0.0, s);   // U = Q V'
    transpose(Up.p, n, Vh, n, n, n, s);                            // Vh = U'^T
    return;
  }
  if (n > kJacobiBlockMaxN) {   // grid-wide block Jacobi, one launch per round
    const int sms = num_sms();
    const int nb = (int)std::max<int64_t>(1, (n + 2 * sms - 1) / (2 * sms));
    int P = (int)((n + nb - 1) / nb);
    P += P & 1;
    identity_kernel<<<cdiv((int64_t)n * n, 256), 256, 0, s>>>(Vw, (int)n);
    TTGB_CHECK_LAUNCH();
    DevBuf<unsigned> cnt(1, s);
    unsigned hcnt = 0;
    const double tol = std::max((double)n, 1.0) * kEps;
    int sweep = 0;
    for (; sweep < 60; ++sweep) {
      TTGB_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(unsigned), s));
      for (int r = 0; r < P - 1; ++r) {
        jacobi_grid_round_kernel<<<P / 2, 256, 0, s>>>(W, Vw, (int)n, nb, P, r, tol, cnt.p);
        TTGB_CHECK_LAUNCH();
      }
      TTGB_CUDA(cudaMemcpyAsync(&hcnt, cnt.p, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
      TTGB_CUDA(cudaStreamSynchronize(s));
      if (hcnt == 0) break;
    }
    if (sweep >= 60) TTGB_CUDA(cudaMemsetAsync(ws.status, 0x03, 1, s));
    DBuf sig((size_t)n, s);
    svd_sort_kernel<<<1, 1024, 0, s>>>(W, Vw, (int)n, Up.p, S, Vw + n * n, sig.p);
    TTGB_CHECK_LAUNCH();
    gemm_cm(Qb.p, m, Vw + n * n, n, U, m, m, n, n, 1.0, 0.0, s);   // U = Q V'
    transpose(Up.p, n, Vh, n, n, n, s);                            // Vh = U'^T
    return;
  }
  const size_t smem = (size_t)2 * n * n * sizeof(double);
  const int use_smem = smem <= 200 * 1024 ? 1 : 0;
  if (use_smem) smem_optin((const void*)jacobi_svd_kernel, (int)smem);
  // one warp per column pair of a round (n < 2 * kJacobiCluster here): idle warps would only
  // lengthen every block barrier of the round-robin sweep
  const int threads = (int)std::min<int64_t>(512, 32 * std::max<int64_t>(1, (n + 1) / 2));
  jacobi_svd_kernel<<<1, threads, use_smem ? smem : 0, s>>>(W, Vw, (int)n, Up.p, S, use_smem, 60,
                                                             ws.status, nullptr);
  TTGB_CHECK_LAUNCH();
  // U = Q V'
  gemm_cm(Qb.p, m, Vw, n, U, m, m, n, n, 1.0, 0.0, s);
  // Vh (n x n col-major) = U'^T
  transpose(Up.p, n, Vh, n, n, n, s);
}

void gemv(const double* B, int64_t n, const double* x, double* y, cudaStream_t s) {
  if (n <= 0) return;
  gemv_rm_kernel<<<cdiv(n * 32, 256), 256, 0, s>>>(B, n, x, y);
  TTGB_CHECK_LAUNCH();
}

}  // namespace ttgb
