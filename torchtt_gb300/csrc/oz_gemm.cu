// FP64 contraction from exact digit products on tcgen05 (see contract_emu.cuh for the splitting and
// its error). Three launches: the digits of the smaller operand Q (with the scale of every k that its
// columns give), the digits of the larger operand P, and the product.
//
// The kernel of contract_emu.cuh makes the digits of a tile where it needs them, i.e. each element once per
// tile of the other operand, and is bound by that integer work (130 us at 322 x 5024 x 161). Made once, the
// digits are a BF16 array, [row block][k / 8][digit][row][8 k]: core matrices of the unswizzled K-major
// layout, with what a stage needs in one piece, so that the digit kernels write 16 bytes per row and
// neighbouring rows side by side, and a bulk copy brings what tcgen05.mma reads. (Tensor-map copies of the
// same bytes from a row-major digit array reached 30 bytes per clock and SM.) The product is 36 BF16
// GEMMs whose accumulators, one per sum p + q of digit
// positions, share the 512 columns of tensor memory:
//
//   warp 0     producer: bulk copies of all eight digits of 16 k per stage;
//   warp 1     MMA issuer: the accumulators of kGroup neighbouring sums are one operand D of kGroup BN columns;
//              digit p of P times the digits of Q that they want, which lie side by side (with
//              blocks of zeros before the first), is one tcgen05.mma. Every D has one shape throughout,
//              which is what orders the MMAs that add to it;
//   warps 2-17 flush: after 128 k (the longest sum that stays below 2^24 in FP32) the eight accumulators of
//              an element are put together in integers, rounded once to FP64, scaled and added up in
//              registers.
//
// CTAs stay for several tiles, and two sets of accumulators let the flush of one period, and the stores of
// a finished tile, run beside the MMAs of the next.
//
// Measured (digits of Q, digits of P, product; against the kernel of contract_emu.cuh): M = 322, N = 5024, K = 161:
// 8.7 + 8.0 + 31 us against 130; 176 x 5632 x 88: 7 + 6 + 17 against 60; 60 x 13440 x 60: 7 + 7 + 16 against
// 40; 161 x 300 x 10000 in splits: 51 + 18 + 55 against 254. One tile per CTA, 48 columns wide with one set
// of accumulators, took 46 us for the first. What bounds the product is the tensor pipe (a stage 32 columns wide is 770 clocks of
// MMAs) and what waits and commits add to it, some 250 clocks per stage; the digit kernels are latency.
//
// Every wait is bounded: a CTA whose wait gives up drains its copies and MMAs (again bounded: the lane that issued
// the MMAs, which alone can ask for their completion, waits for them before it leaves), frees its tensor
// memory, writes NaN into its tiles and sets the calling thread's error word, which the entry points turn into
// a timeout. An infinity or a NaN in an operand is noted by the
// digit kernels, and the CTAs that would read it compute their tiles with FP64 multiply-adds instead.
#include <cooperative_groups.h>

#include <atomic>
#include <climits>
#include <mutex>
#include <type_traits>

#include "emu_digits.cuh"
#include "mbarrier.cuh"
#include "oz_gemm.cuh"

namespace cg = cooperative_groups;

namespace ttgb {

namespace {

constexpr int kBM = 128;              // rows of P per tile
constexpr int kBK = 16;               // k per stage: one tcgen05.mma deep
constexpr int kDig = kEmuSlices;
constexpr int kFlushWarps = 16;
constexpr int kThreads = 32 * (2 + kFlushWarps);
constexpr int kQCtas = 8;             // cluster that slices one chunk of Q
constexpr int kQCols = 64;            // columns per CTA of it
constexpr int kMaxQ = kQCtas * kQCols;
constexpr int kPRows = 32;            // rows per CTA of the P slicer

// An operand: element (row, k) of batch entry z at base[z bs + off(row) + off(k)].
struct Operand {
  const double* base;
  AxD row, k;
  int64_t bs;
  int rows, z;          // z: batch entries with digits of their own
  int blk;              // rows of a block
  __nv_bfloat16* dig;   // [z][row block][k / 8][digit][row][8]
  int* scale;           // [z][chunk][row]
  int* special;         // words of the digit kernel's CTAs
};

// digits of (row, k0) of an operand, k0 a multiple of 8; kp: K in whole stages
__device__ __forceinline__ __nv_bfloat16* digit_ptr(const Operand& o, int kp, int z, int row, int k0) {
  const int nb = (o.rows + o.blk - 1) / o.blk, rb = row / o.blk;
  return o.dig + ((((int64_t)z * nb + rb) * (kp >> 3) + (k0 >> 3)) * kDig * o.blk + (row - rb * o.blk)) * 8;
}

// 8 consecutive k of a row into the eight digits' core matrices
__device__ __forceinline__ void put8(const uint2 (&y)[8], __nv_bfloat16* p, int64_t pitch_digit) {
  unsigned lo[kDig][2], hi[kDig][2];
  const uint2 a[4] = {y[0], y[1], y[2], y[3]}, b[4] = {y[4], y[5], y[6], y[7]};
  digits4(a, lo);
  digits4(b, hi);
#pragma unroll
  for (int d = 0; d < kDig; ++d)
    *reinterpret_cast<uint4*>(p + d * pitch_digit) = make_uint4(lo[d][0], lo[d][1], hi[d][0], hi[d][1]);
}

// kPer elements of a row from k0 on, zeros past K; true when one is special
template <int PER>
__device__ __forceinline__ bool load_row(double (&v)[PER], const Operand& o, int z, int row, bool ok, int k0,
                                         int K) {
  bool special = false;
  const double* base = o.base + (int64_t)z * o.bs + (ok ? ax_off(o.row, row) : 0);
  AxWalk w(o.k, k0);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    v[i] = (ok && k0 + i < K) ? base[w.off] : 0.0;
    w.next(o.k);
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) special |= emu_special(v[i]);
  return special;
}

template <int PER>
__device__ __forceinline__ bool nonfinite(const double (&v)[PER]) {
  bool r = false;
#pragma unroll
  for (int i = 0; i < PER; ++i) r |= emu_nonfinite(v[i]);
  return r;
}

// Digits of Q, one cluster per chunk of 128 k and batch entry: thread (column, eighth of the chunk).
// Scales: Fj the column's largest exponent, kappa(k) the largest that Fj leaves in row k of Q over all
// columns (a maximum over the cluster). kappa(k) is 0 where column j has its largest element and never
// above, so nothing is left to scale in the column.
__global__ void __cluster_dims__(kQCtas, 1, 1) __launch_bounds__(kQCols * 8)
    oz_digits_q_kernel(Operand q, int K, int kp, int* kappa) {
  constexpr int kPer = kOzChunk / 8;
  __shared__ int f[kQCols], km[kOzChunk], kall[kOzChunk];
  cg::cluster_group cluster = cg::this_cluster();
  const int chunk = blockIdx.x / kQCtas, rank = blockIdx.x % kQCtas, z = blockIdx.y;
  const int nchunk = gridDim.x / kQCtas;
  const int tid = threadIdx.x, lane = tid & 31;
  const int per = (q.rows + kQCtas - 1) / kQCtas;
  const int c = tid % kQCols, part = tid / kQCols;
  const int j = rank * per + c;
  const bool ok = c < per && j < q.rows;
  const int k0 = chunk * kOzChunk + part * kPer;
  if (tid < kQCols) f[tid] = kEmuZero;
  if (tid < kOzChunk) km[tid] = kEmuZero;
  double v[kPer];
  const bool rare = __syncthreads_or(load_row(v, q, z, j, ok, k0, K) ? 1 : 0) != 0;
  const int any = rare && __syncthreads_or(nonfinite(v) ? 1 : 0);
  if (tid == 0) q.special[(z * nchunk + chunk) * kQCtas + rank] = any;
  const auto digits = [&](auto sub) {
    constexpr bool kSub = decltype(sub)::value;
    int mx = kEmuZero;
#pragma unroll
    for (int i = 0; i < kPer; ++i) mx = max(mx, emu_exponent<kSub>(v[i]));
    atomicMax(&f[c], mx);
    __syncthreads();
    const int F = f[c];
    int mine = kEmuZero;   // lane i: the maximum of k0 + i over the warp's columns
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int e = emu_exponent<kSub>(v[i]);
      const int m = __reduce_max_sync(0xffffffffu, e == kEmuZero ? kEmuZero : e - F);
      if (lane == i) mine = m;
    }
    if (lane < kPer) atomicMax(&km[part * kPer + lane], mine);
    cluster.sync();
    if (tid < kOzChunk) {
      int m = kEmuZero;
#pragma unroll
      for (int r = 0; r < kQCtas; ++r) m = max(m, cluster.map_shared_rank(km, r)[tid]);
      kall[tid] = m;
      if (rank == 0) kappa[((int64_t)z * nchunk + chunk) * kOzChunk + tid] = m;
    }
    __syncthreads();
    if (ok) {
      if (part == 0) q.scale[((int64_t)z * nchunk + chunk) * q.rows + j] = F;
      const int64_t pitch = (int64_t)q.blk * 8;
      __nv_bfloat16* p = digit_ptr(q, kp, z, j, k0);
#pragma unroll
      for (int o = 0; o < kPer / 8; ++o) {
        if (k0 >= kp) break;   // kp is a multiple of 16
        uint2 y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double x = v[8 * o + i];
          const int e = emu_exponent<kSub>(x);
          y[i] = fixed_digits<kSub>(x, e == kEmuZero ? kEmuZero : e - F - kall[part * kPer + 8 * o + i], 0);
        }
        put8(y, p + o * kDig * pitch, pitch);
      }
    }
    cluster.sync();   // no CTA leaves while another may still read its maxima
  };
  if (rare) digits(std::true_type());
  else digits(std::false_type());
}

// Digits of P: 32 rows of one chunk per CTA, thread (row, eighth of the chunk). Scale: the row's largest
// exponent after k's scale kappa(k).
__global__ void __launch_bounds__(256) oz_digits_p_kernel(Operand p, int K, int kp,
                                                          const int* kappa, int kappa_z) {
  stream_wait();
  constexpr int kPer = kOzChunk / 8;
  __shared__ int emax[kPRows], kk[kOzChunk];
  const int chunk = blockIdx.y, z = blockIdx.z, nchunk = gridDim.y;
  const int tid = threadIdx.x;
  const int c = tid % kPRows, part = tid / kPRows;
  const int i = blockIdx.x * kPRows + c;
  const bool ok = i < p.rows;
  const int k0 = chunk * kOzChunk + part * kPer;
  if (tid < kPRows) emax[tid] = kEmuZero;
  if (tid < kOzChunk) kk[tid] = kappa[((int64_t)(kappa_z > 1 ? z : 0) * nchunk + chunk) * kOzChunk + tid];
  double v[kPer];
  const bool rare = __syncthreads_or(load_row(v, p, z, i, ok, k0, K) ? 1 : 0) != 0;
  const int any = rare && __syncthreads_or(nonfinite(v) ? 1 : 0);
  if (tid == 0) p.special[((int64_t)z * nchunk + chunk) * gridDim.x + blockIdx.x] = any;
  const auto digits = [&](auto sub) {
    constexpr bool kSub = decltype(sub)::value;
    int mx = 2 * kEmuZero;
#pragma unroll
    for (int q = 0; q < kPer; ++q) mx = max(mx, emu_exponent<kSub>(v[q]) + kk[part * kPer + q]);
    atomicMax(&emax[c], mx);
    __syncthreads();
    if (!ok) return;
    const int E = emax[c];
    if (part == 0) p.scale[((int64_t)z * nchunk + chunk) * p.rows + i] = E;
    const int64_t pitch = (int64_t)p.blk * 8;
    __nv_bfloat16* d = digit_ptr(p, kp, z, i, k0);
#pragma unroll
    for (int o = 0; o < kPer / 8; ++o) {
      if (k0 >= kp) break;   // kp is a multiple of 16
      uint2 y[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        y[q] = fixed_digits<kSub>(v[8 * o + q], emu_exponent<kSub>(v[8 * o + q]) + kk[part * kPer + 8 * o + q], E);
      put8(y, d + o * kDig * pitch, pitch);
    }
  };
  if (rare) digits(std::true_type());
  else digits(std::false_type());
}

// ---- product ---------------------------------------------------------------------------------------

// Shared-memory matrix descriptor: K-major, no swizzle, core matrices of 8 rows x 16 bytes; 8-row groups
// 128 bytes apart, the next 8 k `kstep` bytes on.
__device__ __forceinline__ uint64_t desc_cores(uint32_t saddr, uint32_t kstep) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(kstep >> 4) << 16) |
         ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ void mma_bf16_ss(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const __nv_bfloat16* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

struct OzParams {
  Operand p, q;
  int K, kp, kchunk, splitk, nchunk;
  int swap;             // P is the contraction's B (its rows are the columns n of C)
  int tri;
  int tiles;
  int scale, keep;      // alpha is not 1; beta is not 0
  int* err;             // set when a wait gave up
  double* C;
  AxD cp, cq;          // C's axes along P's and Q's rows
  int64_t c_bs;
  double alpha, beta;
};

__noinline__ __device__ double emu_round_any(long long T, int E) { return emu_round(T, E); }

// The value of the eight sums over at most 128 k (weight 2^(8 (14 - d)) each) at scale exponents E, rounded
// to nearest. Sums 0 to 2 are at most 2^22 and become integers by adding 1.5 2^23 (a conversion takes eight
// issue slots); sum 7 is rounded to a multiple of 4 in the same way, 2^-64 of the scales.
__device__ __forceinline__ double oz_value(const uint32_t (&D)[8], int E) {
  constexpr unsigned kOne = 0x4b400000u, kFour = 0x4c400000u;   // 1.5 2^23, 1.5 2^25
  const auto f = [&](int d) { return __uint_as_float(D[d]); };
  const auto bits = [&](int d, unsigned magic) { return __float_as_uint(f(d) + __uint_as_float(magic)); };
  const int w0 = (int)(bits(0, kOne) * 256u + bits(1, kOne) - kOne * 257u);
  const int w1 = (int)(bits(2, kOne) * 256u + (unsigned)__float2int_rn(f(3)) - kOne * 256u);
  const int i4 = __float2int_rn(f(4)), i5 = __float2int_rn(f(5)), i6 = __float2int_rn(f(6));
  const int q7 = (int)(bits(7, kFour) - kFour);   // sum 7 in fours
  // sums 4 to 7 in units of 2^58, sums 0 to 3 (below 2^43.1) in units of 2^88
  const long long low = (long long)i4 * (1 << 22) + ((long long)i5 * (1 << 14) + (long long)(i6 * 64 + q7));
  const long long high = (long long)w0 * 65536 + w1 + (low >> 30);
  // their sum in 96 bits, its magnitude, and the leading 64 bits of that
  unsigned v0 = ((unsigned)low & 0x3fffffffu) | (unsigned)high << 30, v1 = (unsigned)(high >> 2);
  unsigned v2 = (unsigned)(high >> 34);
  const unsigned sign = (unsigned)((int)v2 >> 31);
  v0 ^= sign; v1 ^= sign; v2 ^= sign;
  asm("{\n\tadd.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, %2, 0;\n\t}\n"
      : "+r"(v0), "+r"(v1), "+r"(v2) : "r"(sign & 1u));
  int ef = E - 2110 + 1023 + 95;   // units of 2^58 at 2^(E - 2168)
  if (v2 == 0u) { v2 = v1; v1 = v0; v0 = 0u; ef -= 32; }
  if (v2 == 0u) { v2 = v1; v1 = 0u; ef -= 32; }
  if (v2 == 0u) return 0.0;
  const int lz = __clz((int)v2);
  ef -= lz;
  const unsigned mh = __funnelshift_l(v1, v2, lz), ml = __funnelshift_l(v0, v1, lz);
  if ((unsigned)(ef - 1) >= 2045u) {
    const long long T = (long long)(((unsigned long long)mh << 32 | ml) >> 2);
    return emu_round_any(sign != 0u ? -T : T, ef - 1023 - 61);
  }
  // 53 bits, the leading one adding itself to the exponent; a carry out of them does the same
  const unsigned long long frac = ((unsigned long long)(mh >> 11) << 32 | __funnelshift_r(ml, mh, 11)) +
                                  ((ml >> 10) & 1u);
  const unsigned hi = (unsigned)(frac >> 32) + ((unsigned)(ef - 1) << 20);
  return __hiloint2double((int)(hi | (sign & 0x80000000u)), (int)(unsigned)frac);
}

template <int BN>
struct OzRing {
  static constexpr int kGroup = 128 / BN;          // sums per MMA
  static constexpr int kQDig = kDig + kGroup - 1;  // digits of Q with the zeros before
  static constexpr int kP = kDig * kBM * kBK * 2, kQ = kQDig * BN * kBK * 2, kStage = kP + kQ;
  static constexpr int kBytes = kDig * (kBM + BN) * kBK * 2;   // copied per stage
  static constexpr int kStages = 4;
  static constexpr int kPart = BN / (kFlushWarps / 4);         // columns of a flush warp
  static constexpr int kTurn = kFlushWarps * 32 * (kPart + 1) * 8;
  static constexpr int kSmem = kStages * kStage + kTurn + 1024;
};

// A CTA's position in its list of tiles (row block, column block, batch entry, split), column blocks
// fastest: CTAs that run at the same time read the same rows of P.
struct OzTile {
  int r0, c0, z, zp, zq, kbeg, kend, nk;
};
template <int BN>
__device__ __forceinline__ bool oz_tile(const OzParams& P, int t, OzTile& o) {
  const int nc = (P.q.rows + BN - 1) / BN, nr = (P.p.rows + kBM - 1) / kBM;
  const int c = t % nc, rest = t / nc, r = rest % nr, zs = rest / nr;
  o.z = zs / P.splitk;
  o.r0 = r * kBM;
  o.c0 = c * BN;
  o.kbeg = (zs - o.z * P.splitk) * P.kchunk;
  o.kend = min(P.K, o.kbeg + P.kchunk);
  o.nk = (o.kend - o.kbeg + kBK - 1) / kBK;
  o.zp = P.p.z > 1 ? o.z : 0;
  o.zq = P.q.z > 1 ? o.z : 0;
  // C needed for m >= n only: is any of the tile?
  return !(P.tri & kTriLowerC) || (P.swap ? o.c0 + BN > o.r0 : o.r0 + kBM > o.c0);
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) oz_gemm_kernel(const __grid_constant__ OzParams P) {
  using Ring = OzRing<BN>;
  constexpr uint32_t kPBytes = Ring::kP, kStage = Ring::kStage;
  constexpr int kStages = Ring::kStages, kGroup = Ring::kGroup, kQDig = Ring::kQDig, kPart = Ring::kPart;
  constexpr uint32_t kPStep = kDig * kBM * 16, kQStep = kQDig * BN * 16;   // 8 k of all digits
  constexpr uint32_t kCols = 2 * 8 * BN;                                   // two sets of accumulators
  constexpr int kPeriod = kOzChunk / kBK;                                  // stages between flushes
  extern __shared__ uint8_t smraw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], accf[2], acce[2], drained;
  __shared__ uint32_t tmem_sh;
  __shared__ int abort_sh, issued_sh, consumed_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // the blocks of zeros before Q's first digit
  for (int t = tid; t < kStages * 2 * (kGroup - 1) * BN; t += kThreads) {
    const int blk = t / ((kGroup - 1) * BN), r = t - blk * ((kGroup - 1) * BN);
    *reinterpret_cast<uint4*>(ring + (size_t)(blk >> 1) * kStage + kPBytes + (blk & 1) * kQStep + r * 16) =
        make_uint4(0u, 0u, 0u, 0u);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accf[b]), 1);
      mbar_init(smem_u32(&acce[b]), kFlushWarps);
    }
    mbar_init(smem_u32(&drained), 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
    abort_sh = 0;
    issued_sh = 0;
    consumed_sh = INT_MAX;
  }
  stream_wait();   // for the digits and what an earlier kernel left in C
  // a special value in what this CTA reads
  int special = 0;
  OzTile o;
  for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
    if (!oz_tile<BN>(P, t, o)) continue;
    const int pblocks = (P.p.rows + kPRows - 1) / kPRows;
    const int ch0 = o.kbeg / kOzChunk, ch1 = (o.kend + kOzChunk - 1) / kOzChunk;
    for (int i = tid; i < (ch1 - ch0) * (kBM / kPRows); i += kThreads) {
      const int b = o.r0 / kPRows + i % (kBM / kPRows);
      if (b < pblocks)
        special |= P.p.special[((int64_t)o.zp * P.nchunk + ch0 + i / (kBM / kPRows)) * pblocks + b];
    }
    for (int i = tid; i < (ch1 - ch0) * kQCtas; i += kThreads)
      special |= P.q.special[(o.zq * P.nchunk + ch0) * kQCtas + i];
  }
  const auto put = [&](double* c, double x) {
    if (P.scale) x *= P.alpha;
    if (P.splitk > 1) atomicAdd(c, x);
    else *c = P.keep ? fma(P.beta, *c, x) : x;
  };
  special = __syncthreads_or(special);
  if (special) {   // rare: the tiles with FP64 multiply-adds
    for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
      if (!oz_tile<BN>(P, t, o)) continue;
      for (int e = tid; e < kBM * BN; e += kThreads) {
        const int i = o.r0 + e % kBM, j = o.c0 + e / kBM;
        if (i >= P.p.rows || j >= P.q.rows) continue;
        const double* a = P.p.base + (int64_t)o.z * P.p.bs + ax_off(P.p.row, i);
        const double* b = P.q.base + (int64_t)o.z * P.q.bs + ax_off(P.q.row, j);
        double s = 0.0;
        for (int k = o.kbeg; k < o.kend; ++k) s = fma(a[ax_off(P.p.k, k)], b[ax_off(P.q.k, k)], s);
        put(P.C + (int64_t)o.z * P.c_bs + ax_off(P.cp, i) + ax_off(P.cq, j), s);
      }
    }
    return;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                 "n"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_sh;

  if (warp == 0) {
    if (lane == 0) {   // ---- producer
      int g = 0;       // stages so far
      bool ok = true;
      for (int t = blockIdx.x; t < P.tiles && ok; t += gridDim.x) {
        if (!oz_tile<BN>(P, t, o)) continue;
        const __nv_bfloat16* psrc = digit_ptr(P.p, P.kp, o.zp, o.r0, o.kbeg);
        const __nv_bfloat16* qsrc = digit_ptr(P.q, P.kp, o.zq, o.c0, o.kbeg);
        for (int kc = 0; kc < o.nk; ++kc, ++g) {
          const int s = g % kStages;
          ok = mbar_wait(smem_u32(&empty[s]), ((uint32_t)(g / kStages) & 1u) ^ 1u);
          if (!ok) {
            atomicExch(&abort_sh, 1);
            break;
          }
          const uint32_t st = smem_u32(ring + (size_t)s * kStage), fb = smem_u32(&full[s]);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                       "r"((uint32_t)Ring::kBytes)
                       : "memory");
          bulk_copy(st, psrc + (int64_t)kc * (kDig * kBM * kBK), kDig * kBM * kBK * 2, fb);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            bulk_copy(st + kPBytes + h * kQStep + (kGroup - 1) * BN * 16,
                      qsrc + (int64_t)kc * (kDig * BN * kBK) + h * (kDig * BN * 8), kDig * BN * 16, fb);
          *(volatile int*)&issued_sh = g + 1;
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer; kind::f16: D = F32, A = B = BF16, K-major, M = 128. The warp stays together, so that
    // descriptors are uniform values, and one elected lane issues.
    const bool leader = elect_one();
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kBM >> 4) << 24) |
                           (uint32_t)(kGroup * BN >> 3) << 17;
    int g = 0, u = 0;   // stages and flush periods so far
    bool ok = true, ready = false;
    for (int t = blockIdx.x; t < P.tiles && ok; t += gridDim.x) {
      if (!oz_tile<BN>(P, t, o)) continue;
      for (int kc = 0; kc < o.nk; ++kc, ++g) {
        const int s = g % kStages, in_period = kc % kPeriod;
        if (in_period == 0 && u >= 2) {   // the flush of the period before last has read these accumulators
          ok = mbar_wait(smem_u32(&acce[u & 1]), ((uint32_t)(u >> 1) - 1u) & 1u);
          asm volatile("tcgen05.fence::after_thread_sync;");
        }
        ok = ok && (ready || mbar_wait(smem_u32(&full[s]), (uint32_t)(g / kStages) & 1u));
        ok = __all_sync(0xffffffffu, ok) != 0;
        if (!ok) {
          if (leader) {
            consumed_sh = g;
            atomicExch(&abort_sh, 1);
          }
          break;
        }
        // asked here, the next stage's barrier answers while the MMAs are issued
        ready = mbar_done(smem_u32(&full[(s + 1) % kStages]), (uint32_t)((g + 1) / kStages) & 1u);
        const uint32_t pa = smem_u32(ring + (size_t)s * kStage), qa = pa + kPBytes;
        const uint32_t acc = tmem + (uint32_t)((u & 1) * 8 * BN);
        const bool last = in_period == kPeriod - 1 || kc == o.nk - 1;
        if (leader) {
#pragma unroll
          for (int d = 0; d < kDig; d += kGroup) {   // sums d to d + kGroup - 1: digits p of P, d - p + .. of Q
#pragma unroll
            for (int p = 0; p < d + kGroup; ++p)
              mma_bf16_ss(acc + (uint32_t)(d * BN), desc_cores(pa + p * (kBM * 16), kPStep),
                          desc_cores(qa + (d - p + kGroup - 1) * (BN * 16), kQStep), idesc,
                          (in_period | p) != 0 ? 1u : 0u);
          }
          commit(smem_u32(&empty[s]));
          if (last) commit(smem_u32(&accf[u & 1]));
        }
        u += last ? 1 : 0;
        __syncwarp();
      }
    }
    // the MMAs issued and the arrivals of the commits above are complete when the CTA leaves, also after a
    // wait that gave up
    if (leader) {
      commit(smem_u32(&drained));
      if (!mbar_wait(smem_u32(&drained), 0u)) atomicExch(&abort_sh, 1);
    }
    __syncwarp();
  } else {   // ---- flush: the four warps of a TMEM lane quarter take a quarter of the columns each
    const int q = warp & 3;
    const int cb = (warp - 2) / 4 * kPart;
    double* turn = reinterpret_cast<double*>(ring + (size_t)kStages * kStage) + (warp - 2) * (32 * (kPart + 1));
    int u = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < P.tiles && ok; t += gridDim.x) {
      if (!oz_tile<BN>(P, t, o)) continue;
      const int row = o.r0 + q * 32 + lane, col0 = o.c0 + cb;
      const bool row_ok = row < P.p.rows;
      const int periods = (o.nk + kPeriod - 1) / kPeriod;
      double acc[kPart];
      for (int per = 0; per < periods; ++per, ++u) {
        const int chunk = o.kbeg / kOzChunk + per;
        const int E = row_ok ? P.p.scale[((int64_t)o.zp * P.nchunk + chunk) * P.p.rows + row] : kEmuZero;
        // lane i holds the scale of the warp's column i
        const int F = lane < kPart && col0 + lane < P.q.rows
                          ? P.q.scale[((int64_t)o.zq * P.nchunk + chunk) * P.q.rows + col0 + lane] : kEmuZero;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&accf[u & 1]), (uint32_t)(u >> 1) & 1u) ? 1 : 0) != 0;
        if (!ok) {
          if (lane == 0) atomicExch(&abort_sh, 1);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int c = 0; c < kPart; c += 4) {
          uint32_t v[8][4];   // [digit sum][column]
#pragma unroll
          for (int d = 0; d < 8; ++d) {
            const uint32_t taddr =
                tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((u & 1) * 8 * BN + d * BN + cb + c);
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v[d][0]), "=r"(v[d][1]), "=r"(v[d][2]), "=r"(v[d][3])
                         : "r"(taddr));
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t D[8] = {v[0][j], v[1][j], v[2][j], v[3][j], v[4][j], v[5][j], v[6][j], v[7][j]};
            const double x = oz_value(D, E + __shfl_sync(0xffffffffu, F, c + j));
            acc[c + j] = per == 0 ? x : acc[c + j] + x;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acce[u & 1])) : "memory");
      }
      if (!ok) break;
      double* C = P.C + (int64_t)o.z * P.c_bs;
      if (P.cp.s0 != 1 && P.cq.s0 == 1) {
        // neighbours in C lie along Q: the warp's part is turned through shared memory, so that a store
        // covers whole sectors
#pragma unroll
        for (int c = 0; c < kPart; ++c) turn[lane * (kPart + 1) + c] = acc[c];
        const int64_t cq = ax_off(P.cq, col0 + (lane < kPart ? lane : 0));
        const int64_t cp = ax_off(P.cp, row_ok ? row : 0);
        __syncwarp();
#pragma unroll 4
        for (int i = 0; i < kPart; ++i) {
          const int e = i * 32 + lane, r = e / kPart, c = e - r * kPart;
          const int64_t off = __shfl_sync(0xffffffffu, cp, r) + __shfl_sync(0xffffffffu, cq, c);
          if (row - lane + r < P.p.rows && col0 + c < P.q.rows) put(C + off, turn[r * (kPart + 1) + c]);
        }
        __syncwarp();
      } else if (row_ok) {
        C += ax_off(P.cp, row);
        AxWalk w(P.cq, col0);
#pragma unroll
        for (int c = 0; c < kPart; ++c) {
          if (col0 + c < P.q.rows) put(C + w.off, acc[c]);
          w.next(P.cq);
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (abort_sh) {
    if (tid == 0) {   // copies issued but not consumed (bounded; the MMAs are drained)
      const int issued = issued_sh;
      for (int g = consumed_sh; g < issued; ++g)
        mbar_wait(smem_u32(&full[g % kStages]), (uint32_t)((g / kStages) & 1));
      *(volatile int*)P.err = 1;
      __threadfence_system();
    }
    __syncthreads();
    for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
      if (!oz_tile<BN>(P, t, o)) continue;
      for (int e = tid; e < kBM * BN; e += kThreads) {
        const int i = o.r0 + e % kBM, j = o.c0 + e / kBM;
        if (i < P.p.rows && j < P.q.rows)
          P.C[(int64_t)o.z * P.c_bs + ax_off(P.cp, i) + ax_off(P.cq, j)] = __longlong_as_double(0x7ff8000000000000ll);
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kCols));
  }
}

template <int BN>
void launch_gemm(OzParams& P, int batch, cudaStream_t s) {
  smem_optin((const void*)oz_gemm_kernel<BN>, OzRing<BN>::kSmem);
  P.tiles = (int)(cdiv(P.p.rows, kBM) * cdiv(P.q.rows, BN) * batch * P.splitk);
  launch_early(oz_gemm_kernel<BN>, P.tiles < num_sms() ? P.tiles : num_sms(), kThreads, OzRing<BN>::kSmem, s, P);
  TTGB_CHECK_LAUNCH();
}

bool q_is_a(const ContractDesc& d) { return d.M <= d.N; }   // the smaller operand is Q

thread_local int* t_wait_error = nullptr;   // the thread's word, once it has one

// Tile width: the shorter time of the SM with the most tiles. A stage takes about 620 clocks 16 columns wide,
// 1020 clocks 32 wide.
int tile_width(int p_rows, int q_rows, int64_t rest) {
  const auto t = [&](int bn) {
    const int64_t tiles = (int64_t)cdiv(p_rows, kBM) * cdiv(q_rows, bn) * rest;
    return (tiles + num_sms() - 1) / num_sms() * (bn + 9);
  };
  return t(16) < t(32) ? 16 : 32;
}

}  // namespace

// One page of pinned words for the process, dealt to its threads: a word outlives its thread, as a kernel may.
int* wait_error_word() {
  constexpr unsigned kWords = 1024;
  static std::once_flag once;
  static int* page = nullptr;
  static std::atomic<unsigned> next{0};
  if (t_wait_error == nullptr) {
    std::call_once(once, [] {
      int* p = nullptr;
      TTGB_CUDA(cudaHostAlloc((void**)&p, kWords * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
      for (unsigned i = 0; i < kWords; ++i) p[i] = 0;
      page = p;
    });
    t_wait_error = page + next.fetch_add(1) % kWords;
  }
  return t_wait_error;
}

bool take_wait_error() {
  volatile int* w = t_wait_error;
  if (w == nullptr || *w == 0) return false;
  *w = 0;
  return true;
}

namespace {

int64_t align256(int64_t bytes) { return (bytes + 255) / 256 * 256; }

// Operands of d, with Q's digits in blocks of q_blk rows.
void operands(const ContractDesc& d, int q_blk, Operand& p, Operand& q) {
  const bool qa = q_is_a(d);
  Operand a, b;
  a.base = d.A; a.row = to_dev(d.am, d.M); a.k = to_dev(d.ak, d.K); a.bs = d.batch > 1 ? d.a_bs : 0; a.rows = d.M;
  b.base = d.B; b.row = to_dev(d.bn, d.N); b.k = to_dev(d.bk, d.K); b.bs = d.batch > 1 ? d.b_bs : 0; b.rows = d.N;
  p = qa ? b : a;
  q = qa ? a : b;
  // Q's scales enter P's digits, so P has digits per batch entry wherever either operand differs
  q.z = q.bs != 0 ? d.batch : 1;
  p.z = (p.bs != 0 || q.bs != 0) ? d.batch : 1;
  p.blk = kBM;
  q.blk = q_blk;
}

// Bytes of the parts of a workspace, each aligned.
struct Workspace {
  int64_t dp, dq, sp, sq, kap, fp, fq;
  Workspace(const Operand& p, const Operand& q, int K) {
    const int64_t nchunk = cdiv(K, kOzChunk), kp = cdiv(K, kBK) * kBK;
    const auto digits = [&](const Operand& o) {   // rows in whole blocks
      return align256((int64_t)o.z * cdiv(o.rows, o.blk) * o.blk * kp * kDig * 2);
    };
    dp = digits(p);
    dq = digits(q);
    sp = align256((int64_t)p.z * nchunk * p.rows * 4);
    sq = align256((int64_t)q.z * nchunk * q.rows * 4);
    kap = align256((int64_t)q.z * nchunk * kOzChunk * 4);
    fp = align256((int64_t)p.z * nchunk * cdiv(p.rows, kPRows) * 4);
    fq = align256((int64_t)q.z * nchunk * kQCtas * 4);
  }
  int64_t total() const { return dp + dq + sp + sq + kap + fp + fq; }
};

}  // namespace

// The digits take 16 bytes per element of both operands, with rows in whole blocks and k in whole stages. Where
// that padding is most of it (short rows in many batch entries), the tensor cores would multiply
// it as well; and what a solve reserves beforehand has to cover the workspace.
bool oz_takes(const ContractDesc& d) {
  const int small = d.M < d.N ? d.M : d.N, large = d.M < d.N ? d.N : d.M;
  if (small < 8 || small > kMaxQ || d.K < 16 || (d.tri & kTriUpperB) != 0 || d.batch >= 4096 ||
      (int64_t)large * d.K * d.batch >= (int64_t(1) << 25))
    return false;
  Operand p, q;
  operands(d, 32, p, q);
  return Workspace(p, q, d.K).total() <= (int64_t)oz_workspace_bound((double)large * d.K * p.z);
}

double oz_workspace_bound(double elements) {
  const double bytes = 48.0 * elements + (double)(1 << 22);
  return bytes < (double)(1 << 29) ? bytes : (double)(1 << 29);
}

int64_t oz_tiles(const ContractDesc& d) {
  const int small = d.M < d.N ? d.M : d.N, large = d.M < d.N ? d.N : d.M;
  return (int64_t)cdiv(large, kBM) * cdiv(small, 32) * d.batch;
}

bool oz_contract(const ContractDesc& d, int splitk, int kchunk, cudaStream_t s) {
  const bool qa = q_is_a(d);
  OzParams P;
  operands(d, tile_width(qa ? d.N : d.M, qa ? d.M : d.N, (int64_t)d.batch * splitk), P.p, P.q);
  const int nchunk = (int)cdiv(d.K, kOzChunk);
  const int kp = (d.K + kBK - 1) / kBK * kBK;   // whole stages
  const int pblocks = (int)cdiv(P.p.rows, kPRows);
  const Workspace size(P.p, P.q, d.K);
  DevBuf<unsigned char> ws;
  ws.s = s;
  if (cudaMallocAsync((void**)&ws.p, (size_t)size.total(), s) != cudaSuccess) {
    cudaGetLastError();   // no memory for the digits: the caller has kernels that need none
    ws.p = nullptr;
    return false;
  }
  unsigned char* w = ws.p;
  P.p.dig = reinterpret_cast<__nv_bfloat16*>(w); w += size.dp;
  P.q.dig = reinterpret_cast<__nv_bfloat16*>(w); w += size.dq;
  P.p.scale = reinterpret_cast<int*>(w); w += size.sp;
  P.q.scale = reinterpret_cast<int*>(w); w += size.sq;
  int* kappa = reinterpret_cast<int*>(w); w += size.kap;
  P.p.special = reinterpret_cast<int*>(w); w += size.fp;
  P.q.special = reinterpret_cast<int*>(w);
  oz_digits_q_kernel<<<dim3((unsigned)(nchunk * kQCtas), (unsigned)P.q.z), kQCols * 8, 0, s>>>(P.q, d.K, kp,
                                                                                                     kappa);
  TTGB_CHECK_LAUNCH();
  launch_early(oz_digits_p_kernel, dim3((unsigned)pblocks, (unsigned)nchunk, (unsigned)P.p.z), 256, 0, s, P.p, d.K,
               kp, kappa, P.q.z);
  TTGB_CHECK_LAUNCH();
  P.err = wait_error_word();
  P.K = d.K; P.kp = kp; P.kchunk = splitk > 1 ? kchunk : d.K; P.splitk = splitk; P.nchunk = nchunk;
  P.swap = qa ? 1 : 0;
  P.tri = d.tri;
  P.C = d.C;
  const AxD cm = to_dev(d.cm, d.M), cn = to_dev(d.cn, d.N);
  P.cp = qa ? cn : cm;
  P.cq = qa ? cm : cn;
  P.c_bs = d.c_bs;
  P.alpha = d.alpha; P.beta = d.beta;
  P.scale = d.alpha != 1.0; P.keep = d.beta != 0.0;
  if (P.q.blk == 32) launch_gemm<32>(P, d.batch, s);
  else launch_gemm<16>(P, d.batch, s);
  return true;
}

}  // namespace ttgb
