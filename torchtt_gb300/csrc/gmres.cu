// Restarted GMRES on the local AMEn operator, with the Krylov basis, the Hessenberg matrix, the
// Givens rotations and the convergence test kept on the device (reference: cpp/gmres.h:34-161).
// The host reads the stop flag only from the iteration where the previous cycle's convergence rate
// predicts the stop; everything else stays device resident.
#include <cmath>

#include "gmres.cuh"
#include "reduce.cuh"
#include "rsqrt.cuh"
#include "tc_gemm.cuh"

namespace ttgb {

SplitOut LocalOperator::input_split() const {
  SplitOut o;
  if (lowp && tc && prec == kNoPrec && size() < (int64_t(1) << 31)) {
    o.hi = tc->xh.p;
    o.lo = tc->xl.p;
    o.nR = dims.n * dims.R;
    o.ld = tc->ld_r;
  }
  return o;
}

void LocalOperator::apply(const double* x, double* y, bool use_prec, cudaStream_t s,
                          bool presplit, const int* gate) const {
  const double* in = x;
  if (use_prec && prec != kNoPrec) {
    apply_prec(x, wp, s);
    in = wp;
  }
  if (lowp) {
    if (prof_lowp) prof_lowp->begin();
    if (tc) {
      tc->apply(in, y, s, presplit && prec == kNoPrec, gate);
    } else {
      cast(in, xf, size(), s);
      local_product(dims, phi_l32, A32, phi_r32, xf, yf, w1f, w2f, s, 1.0f, 0.0f, spA);
      cast(yf, y, dims.rl * dims.m * dims.RL, s);
    }
    if (prof_lowp)
      prof_lowp->end(local_product_gemm_flops(dims, spA), tc ? ((presplit && prec == kNoPrec) ? 3 : 4) : 5);
    if (count_lowp) ++*count_lowp;
    return;
  }
  Fp64EngineScope eng(fp64_engine);
  if (prof) prof->begin();
  local_product(dims, phi_l, A, phi_r, in, y, w1, w2, s, 1.0, 0.0, spA);
  if (prof) prof->end(local_product_gemm_flops(dims, spA), 3);
  if (count) ++*count;
}

void LocalOperator::apply_fp64(const double* x, double* y, cudaStream_t s) const {
  Fp64EngineScope eng(fp64_engine);
  if (prof) prof->begin();
  local_product(dims, phi_l, A, phi_r, x, y, w1, w2, s, 1.0, 0.0, spA);
  if (prof) prof->end(local_product_gemm_flops(dims, spA), 3);
  if (count) ++*count;
}


namespace {

using red::RT;
using red::block_sum;
constexpr int kMaxVec = 128;   // basis vectors a cycle may hold (RedWS::cap_vec + 1)

// scalar slots after the Hessenberg data in GmresWS::small
enum ScalSlot : int {
  kRhsNorm = 0,   // ||rhs||
  kResNorm,       // ||r|| at the start of the cycle
  kWNorm2,        // ||w||^2 of the operator output, before orthogonalisation
  kHn,            // H[k+1, k]
  kErr,           // |beta[k+1]| / ||rhs||
  kRhsInv,        // 1 / ||rhs||
  kNumScal = 12
};

struct Layout {   // GmresWS::small
  int iters;
  int64_t H, cs, sn, beta, h1, scal, total;
  explicit Layout(int it) : iters(it) {
    H = 0;
    cs = H + (int64_t)(it + 1) * it;
    sn = cs + it;
    beta = sn + it;
    h1 = beta + it + 1;
    scal = h1 + it + 1;
    total = scal + kNumScal;
  }
};

// ||x|| of the cycle's start vector (also ||rhs|| in the first cycle, where r = rhs) and the
// cycle's start state: H, the rotations and beta cleared, beta[0] = ||r||, the flag words reset.
__global__ void __launch_bounds__(RT) cycle_start_kernel(const double* x, int64_t n,
                                                          int64_t chunk, double* partial,
                                                          unsigned* counter, double* scal,
                                                          int first, int iters, double* H,
                                                          double* cs, double* sn, double* beta,
                                                          int* flag) {
  stream_wait();
  __shared__ double sh[32];
  const int64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  double s = 0.0;
  for (int64_t i = beg + threadIdx.x; i < end; i += blockDim.x) {
    const double v = x[i];
    s = fma(v, v, s);
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
  if (!red::take_last_ticket(counter)) return;
  const int tid = threadIdx.x;
  for (int i = tid; i < (iters + 1) * iters; i += blockDim.x) H[i] = 0.0;
  for (int i = tid; i < iters; i += blockDim.x) { cs[i] = 0.0; sn[i] = 0.0; }
  for (int i = tid; i < iters + 1; i += blockDim.x) beta[i] = 0.0;
  __syncthreads();
  double tot = 0.0;
  if (tid < 32) tot = red::warp_sum_partials(partial, 0, gridDim.x);
  if (tid == 0) {
    const double nr = sqrt(tot);
    if (first) {
      scal[kRhsNorm] = nr;
      scal[kRhsInv] = 1.0 / nr;
    }
    scal[kResNorm] = nr;
    beta[0] = nr;
    // 2: r == 0, nothing to do (gmres.h:56-65); 3: not finite
    flag[kGmresState] = !isfinite(nr) ? 3 : nr > 0.0 ? 0 : 2;
    flag[kGmresBreakdown] = 0;
    flag[kGmresAtIter] = -1;
    flag[kGmresReorth] = 0;
    flag[kGmresReorthVecs] = 0;
  }
  red::reset_ticket(counter);
}

// element i of the operator's next input, also written as its TF32 split when o has a target
__device__ __forceinline__ void put_split(const SplitOut& o, int64_t i, double v) {
  const float f = (float)v;
  const float h = to_tf32(f);
  // 32-bit: input_split() offers a target only for vectors below 2^31 elements
  const unsigned col = (unsigned)i / (unsigned)o.nR, row = (unsigned)i - col * (unsigned)o.nR;
  const int64_t off = (int64_t)row * o.ld + col;
  o.hi[off] = h;
  o.lo[off] = to_tf32(f - h);
}

// y = x / den (den device, y = x when den <= 0); y may alias x
__global__ void scale_by_kernel(const double* x, double* y, int64_t n, const double* den,
                                SplitOut so) {
  stream_wait();
  const double d = *den;
  const double f = (d > 0.0) ? 1.0 / d : 1.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double v = x[i] * f;
    y[i] = v;
    if (so.hi) put_split(so, i, v);
  }
}

// ---------------------------------------------------------------------------------------------
// The Arnoldi step in three launches over the basis V (kv vectors of n doubles).
//
// On GB300 a warp-wide FP64 instruction holds the SM's FP64 pipe for 16 cycles, so at these sizes
// the multiply-adds (kv n per pass) weigh less than the adds of the reductions: a butterfly per
// vector and warp costs 5 instructions for every multiply-add of a 32-element slice. The passes
// therefore deal the vectors, not the elements, to the warps of a block (warp w takes the vectors
// w, w + 8, ...; a lane accumulates E elements of each before any reduction), reduce the vectors of
// a warp together (a step halves the number of values as it halves the lanes: 9 adds for 8 vectors
// instead of 40), and leave the sum over the blocks to the blocks of the next launch, each of which
// adds the G x nv partial sums for itself, so that no pass ends in one block's serial tail.
// Measured per launch (n = 4 k to 32 k, kv up to 41): project 2.3-7 us, update 4-16 us, finish 7-14 us;
// with the elements dealt to the warps and the last block adding the partial sums 18, 31 and 13.5 us.
// ---------------------------------------------------------------------------------------------
constexpr int kWarps = RT / 32;

// Sums of NV per-lane values over the warp's 32 lanes (NV a power of two). On return the lane holds
// the sum of value j = lane / (32 / NV).
template <int NV>
__device__ __forceinline__ double warp_sums(double (&v)[NV]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int m = NV; m > 1; m >>= 1, o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < m / 2; ++j) {   // keep one half of the values, send the other
      const double send = upper ? v[j] : v[j + m / 2];
      const double keep = upper ? v[j + m / 2] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
#pragma unroll
  for (int q = 16 / NV; q > 0; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
  return s;
}

// Partial sums of the warp's vectors (acc[i]: vector warp + 8 i, nv vectors in all) into row
// blockIdx.x of part.
template <int VP>
__device__ __forceinline__ void store_partials(const double (&acc)[VP], int nv, double* part) {
  constexpr int N = VP <= 1 ? 1 : VP <= 2 ? 2 : VP <= 4 ? 4 : 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* row = part + (int64_t)blockIdx.x * nv;
#pragma unroll
  for (int g = 0; g < VP; g += N) {
    if (warp + kWarps * g >= nv) break;   // uniform in the warp
    double v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = g + j < VP ? acc[g + j < VP ? g + j : 0] : 0.0;
    const double s = warp_sums<N>(v);
    const int vec = warp + kWarps * (g + lane / (32 / N));
    if (lane % (32 / N) == 0 && vec < nv) row[vec] = s;
  }
}

// out[v] (shared, v < nv <= 128) = sum over the G rows of part of its column v, in a fixed order;
// sh holds RT doubles. Every thread of the block calls it.
__device__ __forceinline__ void reduce_partials(const double* part, int G, int nv, double* out,
                                                double* sh) {
  int width = 8;
  while (width < nv) width <<= 1;
  const int tid = threadIdx.x, lane = tid & 31;
  const int col = tid & (width - 1), first = tid / width, step = RT / width;
  double s = 0.0;
  if (col < nv) {   // four sums at once: a chain of dependent FP64 adds would take longer than the loads
    double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int g = first; g < G; g += 4 * step) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (g + q * step < G) a[q] += __ldcg(part + (int64_t)(g + q * step) * nv + col);
    }
    s = (a[0] + a[1]) + (a[2] + a[3]);
  }
  int rows = step;
  if (width < 32) {
    for (int o = width; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < width) sh[(tid >> 5) * width + lane] = s;
    rows = kWarps;
  } else {
    sh[tid] = s;
  }
  __syncthreads();
  if (tid < nv) {   // rows is a power of two, 2 to 8
    double a = 0.0, b = 0.0;
    for (int q = 0; q < rows; q += 2) {
      a += sh[q * width + tid];
      b += sh[(q + 1) * width + tid];
    }
    out[tid] = a + b;
  }
  __syncthreads();
}

// Pass 1: part[block] = partial sums of h1 = V^T w (kv values) and ||w||^2.
template <int E, int VP>
__global__ void __launch_bounds__(RT) arnoldi_project_kernel(const double* Q,
                                                              int64_t ldq, int kv,
                                                              const double* w,
                                                              int64_t n, int64_t chunk, double* part,
                                                              const int* gate) {
  stream_wait();
  if (*gate != 0) return;   // an iteration queued past the cycle's stopping point
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  double acc[VP];
#pragma unroll
  for (int i = 0; i < VP; ++i) acc[i] = 0.0;
  for (int64_t c = beg; c < end; c += 32 * E) {
    double x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int64_t i = c + e * 32 + lane;
      x[e] = i < end ? w[i] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < VP; ++i) {
      const int v = warp + kWarps * i;
      if (v > kv) break;
      const double* q = v < kv ? Q + (int64_t)v * ldq : w;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int64_t t = c + e * 32 + lane;
        acc[i] = fma(t < end ? q[t] : 0.0, x[e], acc[i]);
      }
    }
  }
  store_partials<VP>(acc, kv + 1, part);
}

// t = the block's slice of V h (h in shared memory): the warps' shares through sh (8 x 32 E doubles);
// element c of the slice is returned to thread c (0 past the slice).
template <int E, int VP>
__device__ __forceinline__ double slice_combination(const double* Q, int64_t ldq, int kv,
                                                    const double* h, int64_t c, int64_t end,
                                                    double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double t[E];
#pragma unroll
  for (int e = 0; e < E; ++e) t[e] = 0.0;
#pragma unroll
  for (int i = 0; i < VP; ++i) {
    const int v = warp + kWarps * i;
    if (v >= kv) break;
    const double hv = h[v];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int64_t j = c + e * 32 + lane;
      t[e] = fma(hv, j < end ? Q[(int64_t)v * ldq + j] : 0.0, t[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) sh[warp * 32 * E + e * 32 + lane] = t[e];
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32 * E) {   // the warps without a vector hold zeros
    const double* p = sh + threadIdx.x;
    constexpr int o = 32 * E;
    s = ((p[0] + p[o]) + (p[2 * o] + p[3 * o])) + ((p[4 * o] + p[5 * o]) + (p[6 * o] + p[7 * o]));
  }
  return s;
}

// Pass 2: w' = w - V h1, and the partial sums of h2 = V^T w' and ||w'||^2 (V's slice is read again from
// the L1 cache). Block 0 keeps h1 and ||w||^2 for the finishing pass.
template <int E, int VP>
__global__ void __launch_bounds__(RT) arnoldi_reorth_kernel(const double* Q,
                                                             int64_t ldq, int kv, double* w, int64_t n,
                                                             int64_t chunk, const double* part_in,
                                                             double* part_out, double* h1, double* scal,
                                                             const int* gate) {
  __shared__ double sums[kMaxVec];
  __shared__ double sh[kWarps * 32 * E];
  __shared__ double wn[32 * E];
  stream_wait();
  if (*gate != 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  reduce_partials(part_in, gridDim.x, kv + 1, sums, sh);
  if (blockIdx.x == 0 && tid <= kv) {
    if (tid < kv) h1[tid] = sums[tid];
    else scal[kWNorm2] = sums[kv];
  }
  const int64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  double acc[VP];
#pragma unroll
  for (int i = 0; i < VP; ++i) acc[i] = 0.0;
  for (int64_t c = beg; c < end; c += 32 * E) {
    const double s = slice_combination<E, VP>(Q, ldq, kv, sums, c, end, sh);
    if (tid < 32 * E) {
      double v = 0.0;
      if (c + tid < end) {
        v = w[c + tid] - s;
        w[c + tid] = v;
      }
      wn[tid] = v;
    }
    __syncthreads();
    double x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = wn[e * 32 + lane];
#pragma unroll
    for (int i = 0; i < VP; ++i) {
      const int v = warp + kWarps * i;
      if (v > kv) break;
      const double* q = Q + (int64_t)v * ldq;   // row kv is w itself, whose slice is in x
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int64_t t = c + e * 32 + lane;
        acc[i] = fma(v < kv ? (t < end ? q[t] : 0.0) : x[e], x[e], acc[i]);
      }
    }
  }
  store_partials<VP>(acc, kv + 1, part_out);
}

// The new Hessenberg column (h1 + h2, h2 may be null) and the cycle's rotations into shared memory.
__device__ __forceinline__ void givens_load(double* h, double* rot, const double* h1, const double* h2,
                                            int k, const double* cs, const double* sn, int tid, int nt) {
  for (int i = tid; i <= k; i += nt) h[i] = h2 ? h1[i] + h2[i] : h1[i];
  for (int i = tid; i < k; i += nt) {
    rot[2 * i] = cs[i];
    rot[2 * i + 1] = sn[i];
  }
}

// The Givens rotations of the cycle applied to the new Hessenberg column h (k + 2 values, shared
// memory), the new rotation, the residual estimate and the stop flag (apply_givens_rotation_cpu and
// the convergence test, cpp/gmres.h:20-31,105-129). One warp, after givens_load.
__device__ __forceinline__ void givens_step(double* h, const double* rot, int k, int iters, double hn,
                                            double* H, double* cs, double* sn, double* beta,
                                            double threshold, double* scal, int* flag, int reorth_vecs) {
  const int lane = threadIdx.x & 31;
  double* hc = H + (int64_t)k * (iters + 1);
  if (lane == 0) {
    double cur = h[0];
    for (int i = 0; i < k; ++i) {
      const double c = rot[2 * i], s = rot[2 * i + 1], nx = h[i + 1];
      h[i] = c * cur + s * nx;
      cur = c * nx - s * cur;
    }
    const double den2 = fma(cur, cur, hn * hn);
    double c = 1.0, s = 0.0;
    if (den2 > 0.0) {
      const double inv = rsqrt_full(den2);
      c = cur * inv;
      s = hn * inv;
    }
    h[k] = c * cur + s * hn;
    h[k + 1] = 0.0;
    cs[k] = c;
    sn[k] = s;
    const double bk = beta[k], b1 = -s * bk;
    beta[k + 1] = b1;
    beta[k] = c * bk;
    const double err = fabs(b1) * scal[kRhsInv];
    scal[kErr] = err;
    scal[kHn] = hn;
    const bool breakdown = !(hn > 0.0);
    int state = (err <= threshold || breakdown) ? 1 : 0;
    // a NaN in the column leaves the rotation the identity and err 0
    if (!isfinite(err) || !isfinite(den2)) state = 3;
    flag[kGmresBreakdown] = breakdown ? 1 : 0;
    if (state != 0) flag[kGmresAtIter] = k;
    if (reorth_vecs > 0) {
      flag[kGmresReorth] += 1;
      flag[kGmresReorthVecs] += reorth_vecs;
    }
    flag[kGmresState] = state;
  }
  __syncwarp();
  for (int i = lane; i < k + 2; i += 32) hc[i] = h[i];
}

// Pass 3. Every block adds the partial sums of pass 2 and takes the same decision (classical
// Gram-Schmidt with the reorthogonalisation criterion of Daniel, Gragg, Kaufman and Stewart, Math.
// Comp. 30 (1976), with eta = 1/sqrt(2)):
//   mode 0: ||w'||^2 >= ||w||^2 / 2, the first projection is kept, q = w' / ||w'||;
//   mode 1: w'' = w' - V h2 with ||w''||^2 = ||w'||^2 - ||h2||^2 (V orthonormal), used while the
//           difference keeps at least half of ||w'||^2 (no cancellation to speak of);
//   mode 2: w'' = w' - V h2 with its norm taken from the finished vector (near breakdown).
// b <= orth_tol^2 a (the new vector's component along the basis, |V^T w'| / |w'|, is already below the
// tolerated loss of orthogonality) also takes mode 0. With a split target, q is also written as
// the tcgen05 engine's TF32 operand, so the next operator application starts from it without a
// split launch. In mode 0, and in mode 1 without a tolerated loss of orthogonality, the norm is known and an extra
// block takes the Givens step while the others write; otherwise the last block takes it, after it has corrected the scale where the finished vector's
// norm is not 1 to rounding. Once the flag is set, later iterations leave H, beta and the flag
// alone, so iterations queued past the stopping point change nothing the solution uses.
template <int E, int VP>
__global__ void __launch_bounds__(RT) arnoldi_finish_kernel(
    const double* Q, int64_t ldq, int kv, const double* h1,
    const double* part_in, double* w, int64_t n, int64_t chunk, double* part_out, unsigned* counter,
    double* scal, int iters, double* H, double* cs, double* sn, double* beta, double threshold,
    int* flag, SplitOut so, double orth_tol2) {
  __shared__ double sums[kMaxVec];          // h2 and ||w'||^2
  __shared__ double sh[kWarps * 32 * E];
  __shared__ double hcol[kMaxVec + 1], rot[2 * kMaxVec];
  __shared__ double dec[3];                 // mode, norm, 1 / norm
  __shared__ double fac;
  stream_wait();
  // Queued past the stopping point, nothing changes. The extra block may set the flag of this very launch
  // while a block starts late: the block decides once for all its threads, or some of its warps would go
  // on without the others' sums.
  if (__syncthreads_or(flag[kGmresState] != 0)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, k = kv - 1;
  const int G = (int)gridDim.x - 1;   // slices; the block after them takes the Givens step in mode 0
  const bool extra = (int)blockIdx.x == G;
  if (extra) givens_load(hcol, rot, h1, nullptr, k, cs, sn, tid, RT);
  reduce_partials(part_in, G, kv + 1, sums, sh);
  if (warp == 0) {
    double b = 0.0;
    for (int j = lane; j < kv; j += 32) b = fma(sums[j], sums[j], b);
    b = red::warp_sum(b);
    if (lane == 0) {
      const double a = sums[kv], ww = scal[kWNorm2];
      double mode, hp, inv;
      if (!(a < 0.5 * ww) || (a > 0.0 && b <= orth_tol2 * a)) {   // NaN: the Givens step reports it
        mode = 0.0;
        inv = a > 0.0 ? rsqrt_full(a) : 1.0;
        hp = a > 0.0 && isfinite(a) ? a * inv : sqrt(a);   // sqrt: 0, infinite or NaN
      } else if (a > 0.0 && a - b >= 0.5 * a) {
        mode = 1.0;
        inv = rsqrt_full(a - b);
        hp = (a - b) * inv;
      } else {
        mode = 2.0;
        hp = 1.0;
        inv = 1.0;
      }
      dec[0] = mode;
      dec[1] = hp;
      dec[2] = inv;
    }
  }
  __syncthreads();
  const int mode = (int)dec[0];
  const double hp = dec[1], inv = dec[2];
  const int64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  if (mode == 0) {
    for (int64_t i = beg + tid; i < end; i += RT) {
      const double v = w[i] * inv;
      w[i] = v;
      if (so.hi) put_split(so, i, v);
    }
    // a block that starts after the flag is set leaves its slice of q as it is: the cycle has ended then,
    // and its solution does not use q
    if (extra && warp == 0)
      givens_step(hcol, rot, k, iters, hp, H, cs, sn, beta, threshold, scal, flag, 0);
    return;
  }
  // Without a tolerated loss of orthogonality V is orthonormal to rounding after the second projection, so in
  // mode 1 the norm is known as well: the finished vector's would be 1 to some 1e-14.
  const bool known = mode == 1 && orth_tol2 == 0.0;
  if (extra && known) {
    if (tid < kv) hcol[tid] += sums[tid];
    __syncthreads();
    if (warp == 0)
      givens_step(hcol, rot, k, iters, hp, H, cs, sn, beta, threshold, scal, flag, kv);
    return;
  }
  double ss = 0.0;
  for (int64_t c = beg; c < end; c += 32 * E) {
    const double s = slice_combination<E, VP>(Q, ldq, kv, sums, c, end, sh);
    if (tid < 32 * E && c + tid < end) {
      const double v = (w[c + tid] - s) * inv;
      w[c + tid] = v;
      if (so.hi) put_split(so, c + tid, v);
      ss = fma(v, v, ss);
    }
    __syncthreads();
  }
  if (known) return;
  ss = block_sum(ss, sh);
  if (tid == 0) part_out[blockIdx.x] = ss;
  if (!red::take_last_ticket(counter)) return;
  double tot = 0.0;
  if (warp == 0) tot = red::warp_sum_partials(part_out, 0, gridDim.x);
  if (tid == 0) {
    const double nu = sqrt(tot);
    double hn = hp, f = 1.0;
    if (mode == 2) {
      hn = nu;
      if (nu > 0.0) f = 1.0 / nu;
    } else if (nu > 0.0 && fabs(nu - 1.0) > 1e-10) {
      f = 1.0 / nu;
      hn *= nu;
    }
    fac = f;
    dec[1] = hn;
  }
  __syncthreads();
  if (warp == 0) {
    givens_load(hcol, rot, h1, sums, k, cs, sn, lane, 32);
    __syncwarp();
    givens_step(hcol, rot, k, iters, dec[1], H, cs, sn, beta, threshold, scal, flag, kv);
  }
  if (fac != 1.0) {   // rare: only when the direct norm differs from the divisor used above
    for (int64_t i = tid; i < n; i += RT) {
      const double v = w[i] * fac;
      w[i] = v;
      if (so.hi) put_split(so, i, v);
    }
  }
  red::reset_ticket(counter);
}

// sol += V[:, 0..kk] y (sol = V y when `first`, the start x0 = 0) with
// y = H[0..kk, 0..kk]^{-1} beta[0..kk] (upper triangular after the rotations; gmres.h:131-139).
// Every block solves the small triangular system itself, then adds its slice of the combination.
// The solve runs by columns in one warp: the divisions are taken at once before it, and a step is
// one broadcast and one multiply-add per 32 rows (by rows, with a sum over the warp and a division
// per step, the launch took 28-43 us; now 10-13).
__global__ void __launch_bounds__(RT) cycle_update_kernel(int kk, int iters, const double* H,
                                                           const double* beta,
                                                           const double* Q,
                                                           int64_t ldq, double* sol, int64_t n,
                                                           int first) {
  stream_wait();
  __shared__ double ys[kMaxVec];
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    double b[kMaxVec / 32], r[kMaxVec / 32];
#pragma unroll
    for (int q = 0; q < kMaxVec / 32; ++q) {
      const int i = q * 32 + lane;
      const double d = i <= kk ? H[(int64_t)i * (iters + 1) + i] : 0.0;
      b[q] = i <= kk ? beta[i] : 0.0;
      r[q] = d != 0.0 ? 1.0 / d : 0.0;
    }
#pragma unroll
    for (int q = kMaxVec / 32 - 1; q >= 0; --q) {
      for (int i = min(kk, q * 32 + 31); i >= q * 32; --i) {
        const double* col = H + (int64_t)i * (iters + 1);
        const double y = __shfl_sync(0xffffffffu, b[q] * r[q], i & 31);
        if (lane == 0) ys[i] = y;
#pragma unroll
        for (int t = 0; t <= q; ++t) {
          const int row = t * 32 + lane;
          if (row < i) b[t] = fma(-y, col[row], b[t]);
        }
      }
    }
  }
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double v = first ? 0.0 : sol[i];
    for (int j = 0; j <= kk; ++j) v = fma(ys[j], Q[(int64_t)j * ldq + i], v);
    sol[i] = v;
  }
}

unsigned elem_grid(int64_t n) {
  unsigned g = cdiv(n, 256);
  const unsigned cap = (unsigned)num_sms() * 8;
  if (g > cap) g = cap;
  if (g == 0) g = 1;
  return g;
}

// Slices of the Arnoldi passes: one block per SM at most. Blocks of 64 elements up to 64 per SM,
// then 128 and 256 (longer slices run in steps of 256): every pass adds G partial sums per vector in
// every block, so more and shorter slices would only move the work there.
struct ArnoldiGrid {
  int G, E;
  int64_t chunk;
  explicit ArnoldiGrid(int64_t n) {
    const int64_t sms = num_sms();
    E = n <= 64 * sms ? 2 : n <= 128 * sms ? 4 : 8;
    const int64_t step = 32 * E;
    chunk = step * ((n + step * sms - 1) / (step * sms));
    G = (int)((n + chunk - 1) / chunk);
  }
};

struct ArnoldiStep {
  const double* Q;
  int64_t n;
  int kv;
  double* w;
  double *part1, *part2, *h1, *scal, *H, *cs, *sn, *beta;
  unsigned* counter;
  int iters;
  double threshold, orth_tol2;
  int* flag;
  SplitOut so;
};

template <int E, int VP>
void launch_arnoldi(const ArnoldiStep& a, const ArnoldiGrid& g, cudaStream_t s) {
  int* gate = a.flag + kGmresState;
  launch_early(arnoldi_project_kernel<E, VP>, g.G, RT, 0, s, a.Q, a.n, a.kv, a.w, a.n, g.chunk, a.part1, gate);
  TTGB_CHECK_LAUNCH();
  launch_early(arnoldi_reorth_kernel<E, VP>, g.G, RT, 0, s, a.Q, a.n, a.kv, a.w, a.n, g.chunk, a.part1,
               a.part2, a.h1, a.scal, gate);
  TTGB_CHECK_LAUNCH();
  launch_early(arnoldi_finish_kernel<E, VP>, g.G + 1, RT, 0, s, a.Q, a.n, a.kv, a.h1, a.part2, a.w, a.n,
               g.chunk, a.part1, a.counter, a.scal, a.iters, a.H, a.cs, a.sn, a.beta, a.threshold, a.flag,
               a.so, a.orth_tol2);
  TTGB_CHECK_LAUNCH();
}

template <int E>
void launch_arnoldi(const ArnoldiStep& a, const ArnoldiGrid& g, cudaStream_t s) {
  const int nv = a.kv + 1;   // vectors per warp: the basis and w
  if (nv <= kWarps) launch_arnoldi<E, 1>(a, g, s);
  else if (nv <= 2 * kWarps) launch_arnoldi<E, 2>(a, g, s);
  else if (nv <= 4 * kWarps) launch_arnoldi<E, 4>(a, g, s);
  else if (nv <= 6 * kWarps) launch_arnoldi<E, 6>(a, g, s);
  else launch_arnoldi<E, kMaxVec / kWarps>(a, g, s);
}

}  // namespace

// Iterations that the convergence rate of the last converged cycle, log(threshold) / iterations, predicts
// for this threshold; 0: unknown. The flag is read from one iteration before that on. A stop earlier
// than predicted leaves the iterations queued after it, whose kernels read the flag and return at
// once; a later stop costs one more read per extra iteration.
static int predicted_iterations(const GmresWS& ws, double threshold, int iters) {
  if (!(ws.log_rate < 0.0) || !(threshold > 0.0) || !(threshold < 1.0)) return 0;
  const double need = std::log(threshold) / ws.log_rate;
  return need < (double)iters ? (int)std::ceil(need) : iters + 1;
}

GmresResult gmres(const LocalOperator& op, const double* rhs, double* sol, int iters,
                  double threshold, int resets, GmresWS& ws, const RedWS& red, cudaStream_t s,
                  double orth_tol) {
  GmresResult res;
  const int64_t n = op.size();
  TTGB_REQUIRE(iters >= 1, "gmres: local_iterations must be >= 1");
  TTGB_REQUIRE(iters + 1 <= red.cap_vec && iters + 1 <= kMaxVec,
               "gmres: local_iterations exceeds the Krylov workspace (at most 126)");
  for (cudaEvent_t& e : ws.read_done)
    if (!e) TTGB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  ws.Q.ensure((size_t)(iters + 1) * n, s);
  Layout L(iters);
  ws.small.ensure((size_t)L.total, s);
  double* Q = ws.Q.p;
  double* sm = ws.small.p;
  double* H = sm + L.H;
  double* cs = sm + L.cs;
  double* sn = sm + L.sn;
  double* beta = sm + L.beta;
  double* h1 = sm + L.h1;
  double* scal = sm + L.scal;
  int G1; int64_t ch1;
  red_launch_dims(red, n, 1, G1, ch1);
  // the kernels that write the operator's next input also write its tcgen05 operand split
  const SplitOut so = op.input_split();

  const ArnoldiGrid grid(n);
  TTGB_REQUIRE(2 * (int64_t)grid.G * kMaxVec <= (int64_t)red.cap_blocks * red.cap_vec,
               "gmres: reduction workspace too small");
  ArnoldiStep st;
  st.Q = Q; st.n = n;
  st.part1 = red.partial;
  st.part2 = red.partial + (int64_t)grid.G * kMaxVec;
  st.counter = red.counter;
  st.h1 = h1; st.scal = scal; st.H = H; st.cs = cs; st.sn = sn; st.beta = beta;
  st.iters = iters; st.threshold = threshold; st.orth_tol2 = orth_tol * orth_tol;
  st.flag = ws.d_flag; st.so = so;

  // x0 = 0: the first cycle's update writes sol, so it is not cleared beforehand
  for (int cycle = 0; cycle < resets; ++cycle) {
    // r = rhs - op(sol) into Q_0, ||r||, the cycle's start state, Q_0 = r / ||r||
    const double* r = rhs;
    if (cycle > 0) {
      op.apply(sol, Q, true, s);
      sub(rhs, Q, Q, n, s);
      r = Q;
    }
    launch_early(cycle_start_kernel, G1, RT, 0, s, r, n, ch1, red.partial, red.counter, scal, cycle == 0 ? 1 : 0,
                                         iters, H, cs, sn, beta, ws.d_flag);
    TTGB_CHECK_LAUNCH();
    launch_early(scale_by_kernel, elem_grid(n), 256, 0, s, r, Q, n, &scal[kResNorm], so);
    TTGB_CHECK_LAUNCH();
    const int predicted = predicted_iterations(ws, threshold, iters);
    const int first = predicted > 1 ? predicted - 1 : 1;
    int k = 0;
    int state = 0;
    // A read leaves the GPU without work until the host has seen the flag and launched again, some
    // 10 us. So the host first launches the next iteration (its kernels return at once when the
    // flag says stop), except where it expects the stop.
    int pending = -1;            // iteration whose flag is on its way
    const int* flag = ws.h_flag;
    const auto read = [&](int it) {
      TTGB_CUDA(cudaEventSynchronize(ws.read_done[it & 1]));
      ++res.syncs;
      flag = ws.h_flag + (it & 1) * kGmresFlagWords;
      return flag[kGmresState];
    };
    for (k = 0; k < iters; ++k) {
      const int kv = k + 1;
      double* qk = Q + (int64_t)k * n;
      double* w = Q + (int64_t)kv * n;
      // q_k's split was written with q_k; past the stopping point the product does nothing
      op.apply(qk, w, true, s, so.hi != nullptr, ws.d_flag + kGmresState);
      if (op.prof_krylov) op.prof_krylov->begin();
      st.kv = kv;
      st.w = w;
      if (grid.E == 2) launch_arnoldi<2>(st, grid, s);
      else if (grid.E == 4) launch_arnoldi<4>(st, grid, s);
      else launch_arnoldi<8>(st, grid, s);
      // bytes of the reference's MGS iteration, 8 N (2k + 3), and of the three passes here
      // without the second projection, 8 N (2k + 7); the second projection's kv reads are added
      // per cycle from the device's count
      if (op.prof_krylov)
        op.prof_krylov->end(8.0 * (double)n * (2 * k + 3), 3, 8.0 * (double)n * (2 * k + 7));
      if (k + 1 >= first || k == iters - 1) {
        if (pending >= 0) {
          state = read(pending);
          pending = -1;
          if (state != 0) break;
        }
        TTGB_CUDA(cudaMemcpyAsync(ws.h_flag + (k & 1) * kGmresFlagWords, ws.d_flag,
                                  kGmresFlagWords * sizeof(int), cudaMemcpyDeviceToHost, s));
        TTGB_CUDA(cudaEventRecord(ws.read_done[k & 1], s));
        if (k + 1 == predicted || k == iters - 1) {
          state = read(k);
          if (state != 0) break;
        } else {
          pending = k;
        }
      }
    }
    if (state == 2) {          // nothing to do in this cycle (gmres.h:56-65)
      if (cycle == 0) fill(sol, 0.0, n, s);
      res.flag = 1;
      res.overrun += (k < iters ? k : iters - 1) + 1;
      break;
    }
    if (state == 3) throw Error(kNumericalError, "GMRES: non-finite residual");
    const int kk = (state == 1) ? flag[kGmresAtIter] : iters - 1;   // gmres.h:131
    res.overrun += (k < iters ? k : iters - 1) - kk;
    res.reorth += flag[kGmresReorth];
    if (op.prof_krylov) op.prof_krylov->aux += 8.0 * (double)n * flag[kGmresReorthVecs];
    launch_early(cycle_update_kernel, elem_grid(n), RT, 0, s, kk, iters, H, beta, Q, n, sol, n,
                                                    cycle == 0 ? 1 : 0);
    TTGB_CHECK_LAUNCH();
    res.nit += kk + 1;
    if (state == 1) {
      if (threshold > 0.0 && threshold < 1.0) ws.log_rate = std::log(threshold) / (kk + 1);
      res.flag = 1;
      break;
    }
    ws.log_rate = 0.0;   // no converged cycle to predict from: read every iteration next time
  }
  return res;
}

}  // namespace ttgb
