// Direct solution of the small dense local systems (reference: at::linalg_solve,
// cpp/amen_solve.h:326).
//
// On GB300 an n = 500 FP64 factorisation is 42 M multiply-adds at 1.9 per clock and SM, so one block
// needs milliseconds however it is written. gj_solve_kernel therefore inverts the matrix in FP32 on
// one 8-CTA cluster (blocked Gauss-Jordan with partial pivoting, the matrix in distributed shared
// memory) and uses the inverse in an FP64 iterative refinement: residuals b - B x and the solution
// are FP64, so the result is as accurate as an FP64 factorisation with refinement (backward error
// at rounding level, checked). A system that this does not bring to that level (condition above
// ~1e6, entries that are not finite, a singular matrix) is left to lu_solve_kernel, the FP64 LU
// with partial pivoting, which returns at once otherwise.
//
// Measured: the systems of the d = 4, n = 16 solves (n near 500) take 184 us, 5.2 ms with the LU; those
// of a d = 5, n = 12 solve 105 us against 1.74 ms. Over 20 random 4 x 5 x 6 systems the median error of the
// solution against a dense 64-bit solve is 3e-12, 1.5e-11 with the LU.
#include <cooperative_groups.h>

#include "linalg.cuh"
#include "reduce.cuh"

namespace cg = cooperative_groups;

namespace ttgb {

namespace {

// sum over the block, valid in every thread
__device__ double block_sum_d(double v, double* sh) {
  v = red::warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  return red::warp_sum(lane < nw ? sh[lane] : 0.0);
}

constexpr int kGjCtas = 8;      // cluster size
constexpr int kGjNb = 16;       // columns per panel
constexpr int kGjMaxN = 512;    // one thread per row; 4 panels of 16 x 513 floats per CTA at most
constexpr int kGjMaxRefine = 12;

// Scratch of one solve in global memory (written and read by the CTAs of the cluster).
struct GjScratch {
  float T[2][kGjMaxN * kGjNb];        // transform of the panel, one row per matrix row
  float part[2][kGjCtas][kGjMaxN];    // each CTA's share of inverse * residual
  double r[kGjMaxN];                  // residual
  unsigned amax[kGjCtas];             // bits of the largest magnitudes
  float norm1[kGjCtas];
  int piv[kGjMaxN];                   // pivot row of each column
};

// x = B^{-1} b (B row-major n x n, n <= kGjMaxN); *fail = 0, or 1 when the refinement did not reach
// rounding level. The 16-column panels are dealt to the CTAs in turn; thread t owns row t of every
// column. A panel is factored in registers by its owner (one barrier per column: each warp offers
// its largest candidate together with that row's values), which publishes the panel's transform T
// (n x 16): every other column c becomes (row in panel ? 0 : A[row, c]) + T[row, :] A[pivots, c]. The
// owner of the next panel updates and factors that panel before its other columns, so the
// factorisation overlaps the other CTAs' updates and a panel costs one cluster barrier. Rows are
// never swapped: the inverse comes out with its rows and columns permuted by piv.
__global__ void __cluster_dims__(kGjCtas, 1, 1) __launch_bounds__(kGjMaxN, 1)
    gj_solve_kernel(const double* __restrict__ B, const double* __restrict__ b, double* x, int n,
                    GjScratch* g, int* fail) {
  extern __shared__ float A[];   // own columns, column-major with pitch ld
  __shared__ double xs[kGjMaxN], xn[kGjMaxN];
  __shared__ __align__(16) float Bs[4 * kGjNb][kGjNb];   // pivot rows of the own columns
  __shared__ __align__(16) float cand_v[2][kGjMaxN / 32][kGjNb];
  __shared__ unsigned cand_key[2][kGjMaxN / 32];
  __shared__ int cand_row[2][kGjMaxN / 32];
  __shared__ int piv_sh[kGjNb];
  __shared__ float rf[kGjMaxN];
  __shared__ double sh[32];
  __shared__ float shf[32];
  __shared__ unsigned tops[32];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int row = tid;
  const int ld = nt + 1;
  const int nblk = (n + kGjNb - 1) / kGjNb;
  const int mine = rank < nblk ? (nblk - rank + kGjCtas - 1) / kGjCtas : 0;   // own panels
  const int ncol = mine * kGjNb;                                             // own columns
  auto column = [&](int c) { return ((c / kGjNb) * kGjCtas + rank) * kGjNb + c % kGjNb; };

  // the largest magnitude sets a power-of-two scale, so that FP32 holds the scaled entries (compared as
  // integers: a NaN is above every number)
  unsigned top = 0u;
  for (int t = tid; t < n * ncol; t += nt) {
    const int i = t / ncol, j = column(t % ncol);
    if (j < n) top = max(top, __float_as_uint(fabsf((float)B[(int64_t)i * n + j])));
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) tops[warp] = top;
  __syncthreads();
  if (tid == 0) {
    for (int w = 0; w < nw; ++w) top = max(top, tops[w]);
    g->amax[rank] = top;
  }
  cluster.sync();
  top = 0u;
  for (int c = 0; c < kGjCtas; ++c) top = max(top, __ldcg(&g->amax[c]));
  const float mx = __uint_as_float(top);
  if (!(mx > 1e-30f) || !(mx < 1e30f)) {   // zero, not finite, or outside the scale's range
    if (rank == 0 && tid == 0) *fail = 1;
    return;   // the same decision in every thread of the cluster
  }
  const int e = (int)((__float_as_uint(mx) >> 23) & 0xffu) - 127;
  const double scale = __longlong_as_double((long long)(1023 - e) << 52);   // 2^-e

  for (int t = tid; t < nt * ncol; t += nt) {
    const int i = t / ncol, c = t % ncol, j = column(c);
    A[c * ld + i] = (i < n && j < n) ? (float)(B[(int64_t)i * n + j] * scale) : 0.f;
  }
  __syncthreads();
  {   // the 1-norm of the scaled matrix
    float best = 0.f;
    for (int c = warp; c < ncol; c += nw) {
      float s = 0.f;
      for (int i = lane; i < n; i += 32) s += fabsf(A[c * ld + i]);
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      best = fmaxf(best, s);
    }
    if (lane == 0) shf[warp] = best;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < nw; ++w) best = fmaxf(best, shf[w]);
      g->norm1[rank] = best;
    }
  }

  bool used = false;   // row already was a pivot
  float p[kGjNb];      // this row of the panel being factored, then of its transform
  auto factor = [&](int jb) {   // by the owner of panel jb, all threads
    const int w = min(kGjNb, n - jb * kGjNb);
    const int c0 = (jb / kGjCtas) * kGjNb;
#pragma unroll
    for (int j = 0; j < kGjNb; ++j) {
      if (j < w) {
        const unsigned key = (row < n && !used) ? __float_as_uint(fabsf(p[j])) + 1u : 0u;
        const unsigned m = __reduce_max_sync(0xffffffffu, key);
        const unsigned who = __ballot_sync(0xffffffffu, key == m);
        if (lane == __ffs(who) - 1) {
          cand_key[j & 1][warp] = m;
          cand_row[j & 1][warp] = row;
          float4* d = reinterpret_cast<float4*>(cand_v[j & 1][warp]);
#pragma unroll
          for (int q = 0; q < kGjNb / 4; ++q)
            d[q] = make_float4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
        }
        __syncthreads();
        const unsigned k2 = lane < nw ? cand_key[j & 1][lane] : 0u;
        const unsigned m2 = __reduce_max_sync(0xffffffffu, k2);
        const int ww = __ffs(__ballot_sync(0xffffffffu, k2 == m2)) - 1;
        const int pr = cand_row[j & 1][ww];
        const float* v = cand_v[j & 1][ww];
        const float inv = 1.0f / v[j];
        if (row == pr) {
          used = true;
          g->piv[jb * kGjNb + j] = row;
#pragma unroll
          for (int q = 0; q < kGjNb; ++q) p[q] = (q == j) ? inv : p[q] * inv;
        } else {
          const float f = p[j] * inv;
#pragma unroll
          for (int q = 0; q < kGjNb; ++q) p[q] = (q == j) ? -f : fmaf(-f, v[q], p[q]);
        }
      }
    }
    float4* d = reinterpret_cast<float4*>(&g->T[jb & 1][row * kGjNb]);
#pragma unroll
    for (int q = 0; q < kGjNb / 4; ++q)
      d[q] = make_float4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
#pragma unroll
    for (int q = 0; q < kGjNb; ++q) A[(c0 + q) * ld + row] = p[q];
  };

  if (rank == 0) {
#pragma unroll
    for (int q = 0; q < kGjNb; ++q) p[q] = A[q * ld + row];
    factor(0);
  }
  cluster.barrier_arrive();
  for (int jb = 0; jb < nblk; ++jb) {
    cluster.barrier_wait();   // T and the pivots of panel jb are visible
    const int w = min(kGjNb, n - jb * kGjNb);
    float t[kGjNb];
    const float4* src = reinterpret_cast<const float4*>(&g->T[jb & 1][row * kGjNb]);
#pragma unroll
    for (int q = 0; q < kGjNb / 4; ++q) {
      const float4 v = __ldcg(src + q);
      t[4 * q] = v.x; t[4 * q + 1] = v.y; t[4 * q + 2] = v.z; t[4 * q + 3] = v.w;
    }
    if (tid < kGjNb) piv_sh[tid] = tid < w ? __ldcg(&g->piv[jb * kGjNb + tid]) : -1;
    __syncthreads();
    bool in_panel = false;
#pragma unroll
    for (int q = 0; q < kGjNb; ++q) in_panel |= (piv_sh[q] == row);
    used |= in_panel;
    for (int i = tid; i < ncol * kGjNb; i += nt) {
      const int c = i / kGjNb, k = i % kGjNb;
      Bs[c][k] = k < w ? A[c * ld + piv_sh[k]] : 0.f;
    }
    __syncthreads();
    const int own = (jb % kGjCtas == rank) ? jb / kGjCtas : -1;             // this panel
    const int next = (jb + 1 < nblk && (jb + 1) % kGjCtas == rank) ? (jb + 1) / kGjCtas : -1;
    auto updated = [&](int c) {
      float v = in_panel ? 0.f : A[c * ld + row];
      const float4* bp = reinterpret_cast<const float4*>(Bs[c]);
#pragma unroll
      for (int q = 0; q < kGjNb / 4; ++q) {
        const float4 u = bp[q];
        v = fmaf(t[4 * q], u.x, v);
        v = fmaf(t[4 * q + 1], u.y, v);
        v = fmaf(t[4 * q + 2], u.z, v);
        v = fmaf(t[4 * q + 3], u.w, v);
      }
      return v;
    };
    if (next >= 0) {
#pragma unroll
      for (int q = 0; q < kGjNb; ++q) p[q] = updated(next * kGjNb + q);
      factor(jb + 1);
    }
    cluster.barrier_arrive();   // T(jb) has been read, T(jb + 1) written
    for (int lb = 0; lb < mine; ++lb) {
      if (lb == own || lb == next) continue;
#pragma unroll 4
      for (int q = 0; q < kGjNb; ++q) {
        const int c = lb * kGjNb + q;
        A[c * ld + row] = updated(c);
      }
    }
  }
  cluster.barrier_wait();

  // FP64 refinement from x = 0: d = M r with M the FP32 inverse of the scaled matrix, x += d,
  // r = b - B x; every CTA keeps the whole x and takes the same decisions.
  float a1 = 0.f;
  for (int c = 0; c < kGjCtas; ++c) a1 = fmaxf(a1, __ldcg(&g->norm1[c]));
  const int prow = row < n ? __ldcg(&g->piv[row]) : 0;
  const int per = (n + kGjCtas - 1) / kGjCtas;
  const int r0 = rank * per, r1 = min(n, r0 + per);
  if (row < n) xs[row] = 0.0;
  double ri = row < n ? b[row] : 0.0;            // residual of row
  double rp = row < n ? b[prow] : 0.0;           // residual of column row's pivot row
  double rn = block_sum_d(fabs(ri), sh);
  // b = 0 is solved by x = 0 only if the matrix is regular, which no residual would tell: left to the LU
  bool ok = isfinite(rn) && rn > 0.0;
  for (int it = 0; ok && rn > 0.0 && it < kGjMaxRefine; ++it) {
    const int ex = (int)((__double_as_longlong(rn) >> 52) & 0x7ff);
    if (ex < 64 || ex > 1982) { ok = false; break; }
    const double up = __longlong_as_double((long long)(2046 - ex) << 52);          // 2^-exponent
    const double down = __longlong_as_double((long long)ex << 52) * scale;
    __syncthreads();
    rf[row] = row < n ? (float)(rp * up) : 0.f;
    __syncthreads();
    float y0 = 0.f, y1 = 0.f;
    for (int lb = 0; lb < mine; ++lb) {
      const int j0 = (lb * kGjCtas + rank) * kGjNb;
#pragma unroll
      for (int q = 0; q < kGjNb; q += 2) {
        const int c = lb * kGjNb + q;
        y0 = fmaf(A[c * ld + row], j0 + q < n ? rf[j0 + q] : 0.f, y0);
        y1 = fmaf(A[(c + 1) * ld + row], j0 + q + 1 < n ? rf[j0 + q + 1] : 0.f, y1);
      }
    }
    g->part[it & 1][rank][row] = y0 + y1;
    cluster.sync();
    if (row < n) {
      float d = 0.f;
#pragma unroll
      for (int c = 0; c < kGjCtas; ++c) d += __ldcg(&g->part[it & 1][c][prow]);
      xn[row] = fma((double)d, down, xs[row]);
    }
    __syncthreads();
    for (int i = r0 + warp; i < r1; i += nw) {
      const double* bi = B + (int64_t)i * n;
      double s = 0.0;
      for (int j = lane; j < n; j += 32) s = fma(bi[j], xn[j], s);
      s = red::warp_sum(s);
      if (lane == 0) g->r[i] = b[i] - s;
    }
    cluster.sync();
    ri = row < n ? __ldcg(&g->r[row]) : 0.0;
    rp = row < n ? __ldcg(&g->r[prow]) : 0.0;
    const double rnew = block_sum_d(fabs(ri), sh);
    const bool better = rnew < rn;
    const bool go_on = rnew < 0.5 * rn;
    if (better) {
      if (row < n) xs[row] = xn[row];
      rn = rnew;
    }
    if (!go_on) break;
  }
  const double x1 = block_sum_d(row < n ? fabs(xs[row]) : 0.0, sh);
  // the rounding of x alone leaves about eps ||B||_1 ||x||_1
  ok = ok && isfinite(x1) && rn * scale <= 4.0 * 2.220446049250313e-16 * (double)a1 * x1;
  if (rank == 0) {
    if (row < n) x[row] = xs[row];
    if (tid == 0) *fail = ok ? 0 : 1;
  }
}

// ---------------------------------------------------------------------------------------------
// LU with partial pivoting on an n x n row-major copy of B, solving for one right-hand side, in one
// block. Does nothing when *gate is 0 (gate may be null).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) lu_solve_kernel(const double* B,
                                                        const double* b, double* LU,
                                                        double* x, int n, int* status,
                                                        const int* gate) {
  stream_wait();
  __shared__ double shv[32];
  __shared__ double piv_inv;
  __shared__ int shi[32];
  __shared__ int piv;
  if (gate != nullptr && *gate == 0) return;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  for (int64_t t = tid; t < (int64_t)n * n; t += nt) LU[t] = B[t];
  for (int t = tid; t < n; t += nt) x[t] = b[t];
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    // pivot search
    double best = -1.0;
    int bi = j;
    for (int i = j + tid; i < n; i += nt) {
      const double v = fabs(LU[(int64_t)i * n + j]);
      if (v > best) { best = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) { shv[warp] = best; shi[warp] = bi; }
    __syncthreads();
    if (tid == 0) {
      double v = -1.0; int ib = j;
      for (int w = 0; w < (nt >> 5); ++w)
        if (shv[w] > v || (shv[w] == v && shi[w] < ib)) { v = shv[w]; ib = shi[w]; }
      piv = ib;
      if (!(v > 0.0)) *status = 1;
    }
    __syncthreads();
    const int p = piv;
    if (p != j) {
      for (int c = tid; c < n; c += nt) {
        const double t = LU[(int64_t)j * n + c];
        LU[(int64_t)j * n + c] = LU[(int64_t)p * n + c];
        LU[(int64_t)p * n + c] = t;
      }
      if (tid == 0) { const double t = x[j]; x[j] = x[p]; x[p] = t; }
    }
    __syncthreads();
    if (tid == 0) piv_inv = 1.0 / LU[(int64_t)j * n + j];   // one FP64 division per step
    __syncthreads();
    const double inv = piv_inv;
    const int w = n - j - 1;
    // multipliers
    for (int i = j + 1 + tid; i < n; i += nt) LU[(int64_t)i * n + j] *= inv;
    __syncthreads();
    for (int i = j + 1 + tid; i < n; i += nt) x[i] = fma(-LU[(int64_t)i * n + j], x[j], x[i]);
    for (int64_t t = tid; t < (int64_t)w * w; t += nt) {
      const int i = j + 1 + (int)(t / w), c = j + 1 + (int)(t % w);
      LU[(int64_t)i * n + c] = fma(-LU[(int64_t)i * n + j], LU[(int64_t)j * n + c], LU[(int64_t)i * n + c]);
    }
    __syncthreads();
  }
  // back substitution
  __shared__ double shs[32];
  for (int i = n - 1; i >= 0; --i) {
    double s = 0.0;
    for (int c = i + 1 + tid; c < n; c += nt) s = fma(LU[(int64_t)i * n + c], x[c], s);
    s = red::warp_sum(s);
    if (lane == 0) shs[warp] = s;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w2 = 0; w2 < (nt >> 5); ++w2) t += shs[w2];
      x[i] = (x[i] - t) / LU[(int64_t)i * n + i];
    }
    __syncthreads();
  }
}

}  // namespace

void lu_solve(const double* B, int64_t n, const double* rhs, double* x, LinalgWS& ws,
              cudaStream_t s) {
  const size_t gj = (sizeof(GjScratch) + sizeof(double) - 1) / sizeof(double);
  ws.e.ensure((size_t)(n * n) + 16 + gj, s);
  const int* gate = nullptr;
  if (n <= kGjMaxN) {
    const int nt = (int)cdiv(n, 32) * 32;
    const int64_t panels = cdiv(n, kGjNb);
    const size_t smem = (size_t)cdiv(panels, kGjCtas) * kGjNb * (nt + 1) * sizeof(float);
    smem_optin((const void*)gj_solve_kernel, 4 * kGjNb * (kGjMaxN + 1) * (int)sizeof(float));
    gj_solve_kernel<<<kGjCtas, nt, smem, s>>>(B, rhs, x, (int)n,
                                              reinterpret_cast<GjScratch*>(ws.e.p), ws.status + 1);
    TTGB_CHECK_LAUNCH();
    gate = ws.status + 1;
  }
  launch_early(lu_solve_kernel, 1, 1024, 0, s, B, rhs, ws.e.p + gj, x, (int)n, ws.status, gate);
  TTGB_CHECK_LAUNCH();
}

}  // namespace ttgb
