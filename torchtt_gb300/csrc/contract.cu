// FP64 contraction engine and the AMEn contraction recipes built on it.
//
// Every operand index of the GEMM kernels here may be a pair of tensor indices with their own strides
// (struct Ax), so the reference's tensordot permutes (cpp/amen_solve.h:17-98) cost no copies.
// contract_kernel multiplies shared-memory tiles in the operand type (BK = 16, 256 threads, each thread
// a (BM/16) x (BN/16) register tile), contract_small_kernel FP64 in 8 x 8 tiles; contract_emu_kernel
// and, from some 3e7 multiply-adds, oz_gemm.cu take the large FP64 products on the tensor cores;
// contract_df_kernel runs in double-float arithmetic on the FP32 pipe where the caller takes
// that accuracy. Which kernel, tile shape and split-K (atomic FP64 adds) a launch gets comes from the
// tile autotuner's record for its shape class, or from an occupancy heuristic.
#include <climits>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <mutex>
#include <shared_mutex>
#include <type_traits>
#include <unordered_map>

#include "contract.cuh"
#include "df.cuh"
#include "emu_digits.cuh"
#include "oz_gemm.cuh"

namespace ttgb {

namespace {

template <typename T>
struct KParams {
  int M, N, K, batch, splitk, kchunk;
  const T* A;
  AxD am, ak;
  int64_t a_bs;
  const T* B;
  AxD bk, bn;
  int64_t b_bs;
  T* C;
  AxD cm, cn;
  int64_t c_bs;
  T alpha, beta;
  int scale, keep;   // alpha is not 1, beta not 0: comparing in FP64 costs as much as a multiply-add
  int tri;
  int tall;   // the tiles' rows run along the grid's first dimension, the only one with more than 65535 blocks
};

// Row and column of the block's tile among the tiles of C.
template <typename T>
__device__ __forceinline__ int2 tile_of(const KParams<T>& p) {
  return p.tall ? make_int2((int)blockIdx.x, (int)blockIdx.y) : make_int2((int)blockIdx.y, (int)blockIdx.x);
}

constexpr int BK = 16;
constexpr int NT = 256;

template <typename T, int BM, int BN>
__global__ void __launch_bounds__(NT) contract_kernel(KParams<T> p) {
  constexpr int TM = BM / 16, TN = BN / 16;
  __shared__ T As[BK][BM + 1];
  __shared__ T Bs[BK][BN + 1];

  const int tid = threadIdx.x;
  const int bz = blockIdx.z;
  const int bidx = bz / p.splitk;
  const int ks = bz - bidx * p.splitk;
  const int kbeg = ks * p.kchunk;
  int kend = min(p.K, kbeg + p.kchunk);
  const int2 tile = tile_of(p);
  const int m0 = tile.x * BM, n0 = tile.y * BN;
  if ((p.tri & kTriLowerC) && m0 + BM <= n0) {   // tile strictly above the diagonal
    stream_wait();
    return;
  }
  if (p.tri & kTriUpperB) kend = min(kend, n0 + BN);   // B(k, n) = 0 for k > n

  const T* A = p.A + (int64_t)bidx * p.a_bs;
  const T* B = p.B + (int64_t)bidx * p.b_bs;

  // loader mapping: A tile BM x BK, B tile BK x BN, NT threads
  constexpr int A_ROWS_PER_PASS = NT / BK;   // threads cover (row, k) with k = tid % BK
  constexpr int B_COLS_PER_PASS = NT / BK;
  const int lk = tid % BK;
  const int lr = tid / BK;   // 0..15

  int64_t a_moff[BM / A_ROWS_PER_PASS];
  bool a_mok[BM / A_ROWS_PER_PASS];
#pragma unroll
  for (int i = 0; i < BM / A_ROWS_PER_PASS; ++i) {
    int m = m0 + lr + i * A_ROWS_PER_PASS;
    a_mok[i] = m < p.M;
    a_moff[i] = a_mok[i] ? ax_off(p.am, m) : 0;
  }
  int64_t b_noff[BN / B_COLS_PER_PASS];
  bool b_nok[BN / B_COLS_PER_PASS];
#pragma unroll
  for (int i = 0; i < BN / B_COLS_PER_PASS; ++i) {
    int n = n0 + lr + i * B_COLS_PER_PASS;
    b_nok[i] = n < p.N;
    b_noff[i] = b_nok[i] ? ax_off(p.bn, n) : 0;
  }

  const int ty = tid / 16, tx = tid % 16;
  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = T(0);

  stream_wait();
  // next K tile's operands in registers while the current one is multiplied (same sum order)
  T ra[BM / A_ROWS_PER_PASS], rb[BN / B_COLS_PER_PASS];
  auto load_tile = [&](int k0) {
    const int k = k0 + lk;
    const bool kok = k < kend;
    const int64_t a_koff = kok ? ax_off(p.ak, k) : 0;
    const int64_t b_koff = kok ? ax_off(p.bk, k) : 0;
#pragma unroll
    for (int i = 0; i < BM / A_ROWS_PER_PASS; ++i)
      ra[i] = (kok && a_mok[i]) ? A[a_moff[i] + a_koff] : T(0);
#pragma unroll
    for (int i = 0; i < BN / B_COLS_PER_PASS; ++i)
      rb[i] = (kok && b_nok[i]) ? B[b_noff[i] + b_koff] : T(0);
  };
  if (kbeg < kend) load_tile(kbeg);
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
    for (int i = 0; i < BM / A_ROWS_PER_PASS; ++i) As[lk][lr + i * A_ROWS_PER_PASS] = ra[i];
#pragma unroll
    for (int i = 0; i < BN / B_COLS_PER_PASS; ++i) Bs[lk][lr + i * B_COLS_PER_PASS] = rb[i];
    __syncthreads();
    if (k0 + BK < kend) load_tile(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      T a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }

  T* C = p.C + (int64_t)bidx * p.c_bs;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + 16 * i;
    if (m >= p.M) continue;
    const int64_t cmo = ax_off(p.cm, m);
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= p.N) continue;
      T* c = C + cmo + ax_off(p.cn, n);
      const T v = p.scale ? p.alpha * acc[i][j] : acc[i][j];
      if (p.splitk > 1) {
        atomicAdd(c, v);
      } else {
        *c = p.keep ? fma(p.beta, *c, v) : v;
      }
    }
  }
}

// FP64 in 8 x 8 tiles: the eight warps split a chunk of 32 k in four slices (two warps hold a tile's sums), added at the end. A
// product of 40 x 240 x 20 has 45 tiles of 16 x 16, whose SMs do 2.2 k clocks of FP64 per 16 k while the
// other 107 have nothing; in 150 tiles of 8 x 8 the same work takes a quarter of that on every SM.
__global__ void __launch_bounds__(NT) contract_small_kernel(KParams<double> p) {
  constexpr int BS = 8, CK = 32, kSlices = 4;
  __shared__ double As[CK][BS + 1], Bs[CK][BS + 1], part[kSlices - 1][BS * BS];
  const int tid = threadIdx.x;
  const int bz = blockIdx.z;
  const int bidx = bz / p.splitk;
  const int ks = bz - bidx * p.splitk;
  const int kbeg = ks * p.kchunk;
  int kend = min(p.K, kbeg + p.kchunk);
  const int2 tile = tile_of(p);
  const int m0 = tile.x * BS, n0 = tile.y * BS;
  if (p.tri & kTriUpperB) kend = min(kend, n0 + BS);   // B(k, n) = 0 for k > n
  const bool skip = (p.tri & kTriLowerC) && m0 + BS <= n0;   // tile strictly above the diagonal
  // loader: thread (row or column, k) of the chunk
  const int lk = tid % CK, lr = tid / CK;
  const bool mok = m0 + lr < p.M, nok = n0 + lr < p.N;
  const double* A = p.A + (int64_t)bidx * p.a_bs + (mok ? ax_off(p.am, m0 + lr) : 0);
  const double* B = p.B + (int64_t)bidx * p.b_bs + (nok ? ax_off(p.bn, n0 + lr) : 0);
  const int slice = tid / (BS * BS), ty = tid / BS % BS, tx = tid % BS;
  const int m = m0 + ty, n = n0 + tx;
  const bool own = slice == 0 && m < p.M && n < p.N;
  double* c = p.C + (int64_t)bidx * p.c_bs + (own ? ax_off(p.cm, m) + ax_off(p.cn, n) : 0);
  stream_wait();
  if (skip) return;
  double ra = 0.0, rb = 0.0, acc = 0.0;
  const auto load = [&](int k) {
    const bool kok = k < kend;
    ra = kok && mok ? A[ax_off(p.ak, k)] : 0.0;
    rb = kok && nok ? B[ax_off(p.bk, k)] : 0.0;
  };
  if (kbeg < kend) load(kbeg + lk);
  for (int k0 = kbeg; k0 < kend; k0 += CK) {
    As[lk][lr] = ra;
    Bs[lk][lr] = rb;
    __syncthreads();
    if (k0 + CK < kend) load(k0 + CK + lk);
    const int k1 = slice * (CK / kSlices);
    if (k0 + k1 < kend) {   // zeros past the end: a slice without any is left out
#pragma unroll
      for (int kk = 0; kk < CK / kSlices; ++kk) acc = fma(As[k1 + kk][ty], Bs[k1 + kk][tx], acc);
    }
    __syncthreads();
  }
  if (slice > 0) part[slice - 1][tid % (BS * BS)] = acc;
  __syncthreads();
  if (!own) return;
  acc = ((acc + part[0][tid]) + part[1][tid]) + part[2][tid];   // in the order of k
  if (p.scale) acc *= p.alpha;
  if (p.splitk > 1) atomicAdd(c, acc);
  else *c = p.keep ? fma(p.beta, *c, acc) : acc;
}

// The same contraction in double-float arithmetic on the FP32 pipe: every FP64 operand is split
// into hi + lo FP32 parts (x = hi + lo to ~2^-48), a product is formed error-free from the FMA
// residual of hi*hi plus the cross terms, and the sum is kept as an unnormalised (hi, lo) FP32 pair
// with an error-free two-sum per step. About 10 FP32 operations per multiply-add: on GB300, where
// the FP32 pipe is ~60x the FP64 pipe, this is several times the FP64 rate at ~1e-13 relative
// accuracy (operands within the FP32 exponent range).
//
// The FP64 -> (hi, lo) split is df_split (df.cuh).
template <int BM, int BN>
__global__ void __launch_bounds__(NT) contract_df_kernel(KParams<double> p) {
  stream_wait();
  constexpr int TM = BM / 16, TN = BN / 16;
  __shared__ float Ah[BK][BM + 1], Al[BK][BM + 1];
  __shared__ float Bh[BK][BN + 1], Bl[BK][BN + 1];

  const int tid = threadIdx.x;
  const int bz = blockIdx.z;
  const int bidx = bz / p.splitk;
  const int ks = bz - bidx * p.splitk;
  const int kbeg = ks * p.kchunk;
  int kend = min(p.K, kbeg + p.kchunk);
  const int2 tile = tile_of(p);
  const int m0 = tile.x * BM, n0 = tile.y * BN;
  if ((p.tri & kTriLowerC) && m0 + BM <= n0) return;
  if (p.tri & kTriUpperB) kend = min(kend, n0 + BN);

  const double* A = p.A + (int64_t)bidx * p.a_bs;
  const double* B = p.B + (int64_t)bidx * p.b_bs;
  constexpr int ROWS_PER_PASS = NT / BK;
  const int lk = tid % BK;
  const int lr = tid / BK;
  int64_t a_moff[BM / ROWS_PER_PASS];
  bool a_mok[BM / ROWS_PER_PASS];
#pragma unroll
  for (int i = 0; i < BM / ROWS_PER_PASS; ++i) {
    const int m = m0 + lr + i * ROWS_PER_PASS;
    a_mok[i] = m < p.M;
    a_moff[i] = a_mok[i] ? ax_off(p.am, m) : 0;
  }
  int64_t b_noff[BN / ROWS_PER_PASS];
  bool b_nok[BN / ROWS_PER_PASS];
#pragma unroll
  for (int i = 0; i < BN / ROWS_PER_PASS; ++i) {
    const int n = n0 + lr + i * ROWS_PER_PASS;
    b_nok[i] = n < p.N;
    b_noff[i] = b_nok[i] ? ax_off(p.bn, n) : 0;
  }
  const int ty = tid / 16, tx = tid % 16;
  float ch[TM][TN], cl[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) { ch[i][j] = 0.f; cl[i][j] = 0.f; }

  // The operands of the next K tile are loaded into registers while the current tile is
  // multiplied (the global-load latency overlaps the arithmetic); the order of the sums is the
  // same as with a load per tile.
  double ra[BM / ROWS_PER_PASS], rb[BN / ROWS_PER_PASS];
  auto load_tile = [&](int k0) {
    const int k = k0 + lk;
    const bool kok = k < kend;
    const int64_t a_koff = kok ? ax_off(p.ak, k) : 0;
    const int64_t b_koff = kok ? ax_off(p.bk, k) : 0;
#pragma unroll
    for (int i = 0; i < BM / ROWS_PER_PASS; ++i)
      ra[i] = (kok && a_mok[i]) ? A[a_moff[i] + a_koff] : 0.0;
#pragma unroll
    for (int i = 0; i < BN / ROWS_PER_PASS; ++i)
      rb[i] = (kok && b_nok[i]) ? B[b_noff[i] + b_koff] : 0.0;
  };
  if (kbeg < kend) load_tile(kbeg);
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
    for (int i = 0; i < BM / ROWS_PER_PASS; ++i) {
      float h, l;
      df_split(ra[i], h, l);
      Ah[lk][lr + i * ROWS_PER_PASS] = h;
      Al[lk][lr + i * ROWS_PER_PASS] = l;
    }
#pragma unroll
    for (int i = 0; i < BN / ROWS_PER_PASS; ++i) {
      float h, l;
      df_split(rb[i], h, l);
      Bh[lk][lr + i * ROWS_PER_PASS] = h;
      Bl[lk][lr + i * ROWS_PER_PASS] = l;
    }
    __syncthreads();
    if (k0 + BK < kend) load_tile(k0 + BK);
#pragma unroll 4
    for (int kk = 0; kk < BK; ++kk) {
      float ah[TM], al[TM], bh[TN], bl[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) { ah[i] = Ah[kk][ty + 16 * i]; al[i] = Al[kk][ty + 16 * i]; }
#pragma unroll
      for (int j = 0; j < TN; ++j) { bh[j] = Bh[kk][tx + 16 * j]; bl[j] = Bl[kk][tx + 16 * j]; }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float pr = ah[i] * bh[j];
          float e = fmaf(ah[i], bh[j], -pr);        // exact residual of the leading product
          e = fmaf(ah[i], bl[j], e);
          e = fmaf(al[i], bh[j], e);
          const float s = ch[i][j] + pr;            // two-sum of the running high part and pr
          const float bb = s - ch[i][j];
          const float err = (ch[i][j] - (s - bb)) + (pr - bb);
          ch[i][j] = s;
          cl[i][j] += err + e;
        }
    }
    // renormalise the pair once per K tile (two-sum of high and low part): the low part is summed
    // in plain FP32, so left to grow over a long K its own rounding would set the accuracy
    // (a 4928-long Gram sum: 2e-12 relative without, 3e-13 with this step)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float s = ch[i][j] + cl[i][j];
        const float bb = s - ch[i][j];
        cl[i][j] = (ch[i][j] - (s - bb)) + (cl[i][j] - bb);
        ch[i][j] = s;
      }
    __syncthreads();
  }

  double* C = p.C + (int64_t)bidx * p.c_bs;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + 16 * i;
    if (m >= p.M) continue;
    const int64_t cmo = ax_off(p.cm, m);
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= p.N) continue;
      double* c = C + cmo + ax_off(p.cn, n);
      const double v = p.alpha * ((double)ch[i][j] + (double)cl[i][j]);
      if (p.splitk > 1) atomicAdd(c, v);
      else *c = p.keep ? fma(p.beta, *c, v) : v;
    }
  }
}

#include "contract_emu.cuh"

// C <- beta * C over the (batched, strided) output index space
template <typename T>
__global__ void scale_output_kernel(T* C, int M, int N, int batch, AxD cm, AxD cn, int64_t c_bs,
                                    T beta) {
  stream_wait();
  const int64_t total = (int64_t)M * N * batch;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int b = (int)(t / ((int64_t)M * N));
    int rem = (int)(t - (int64_t)b * M * N);
    int m = rem / N, n = rem - (rem / N) * N;
    T* c = C + (int64_t)b * c_bs + ax_off(cm, m) + ax_off(cn, n);
    *c = (beta == T(0)) ? T(0) : beta * *c;
  }
}

thread_local int t_fp64_engine = kFp64Native;
thread_local bool t_no_digits = false;   // set by NoDigitsScope and set_no_digits

// ---------------------------------------------------------------------------------------------
// Tile autotuner. A launch is described by its shape class: the engine (FP64, double-float,
// FP32), power-of-two buckets of M, N, K and the batch, the triangular flags and which operand
// strides are unit, and the device. The first launch of a class with beta == 0 (the output is
// overwritten, so running it several times is harmless) and no overlap between C and its inputs
// times every candidate of its engine (the lists below) with CUDA events on the caller's stream, the
// second of two runs in a row, and records the fastest; later launches of the class
// use the record. Launches that cannot be tuned (beta != 0, aliasing, a capturing stream, a
// deterministic request) and classes being tuned by another thread use the occupancy heuristic.
// ---------------------------------------------------------------------------------------------
// Multiply-adds up to which a product takes the heuristic tile: it is as fast as the one chosen by time (4x5x6 solve 5.0
// and 5.1 ms, d = 5, n = 12 Laplacian 57 and 57 ms, 58 us of a small local product both ways), and a choice
// by time only makes the rounding, and with it the trajectory of a small solve, differ from run to run.
constexpr double kTuneWork = 1e5;
enum TileKind : int {
  kFma = 0,   // multiply-adds in the operand type
  kEmu = 1,   // FP64 from BF16 digits on the tensor cores (contract_emu.cuh)
  kDf = 2,    // double-float on the FP32 pipe
  kOz = 3     // FP64 from digits made beforehand, on tcgen05 (oz_gemm.cu); allocates a workspace
};
struct TileCfg {
  int bm, bn, split;   // split: 0 no split-K, 1 split-K sized to fill the GPU
  TileKind kind = kFma;
};
// FP64: on the FP64 pipe the work per SM sets the time, so the smallest tiles win below about 4 M
// multiply-adds (32 x 32 tiles took 11 us where 16 x 16 take 4-5) and the tensor-core kernel above.
constexpr TileCfg kCandidates64[] = {
    {16, 16, 0}, {16, 32, 0}, {32, 16, 0}, {32, 32, 0}, {16, 16, 1}, {32, 32, 1},
    {64, 32, 0, kEmu}, {32, 64, 0, kEmu}, {64, 16, 0, kEmu}, {16, 64, 0, kEmu},
    {64, 32, 1, kEmu}, {32, 64, 1, kEmu}, {64, 16, 1, kEmu}, {16, 64, 1, kEmu},
    {128, 32, 0, kOz}, {128, 32, 1, kOz}, {8, 8, 0}};
// where the caller takes double-float accuracy
constexpr TileCfg kCandidatesDf[] = {
    {16, 16, 0}, {16, 16, 1}, {32, 32, 0, kDf}, {64, 32, 0, kDf}, {32, 64, 0, kDf},
    {32, 32, 1, kDf}, {64, 32, 1, kDf}, {32, 64, 1, kDf},
    {64, 32, 0, kEmu}, {32, 64, 0, kEmu}, {64, 32, 1, kEmu}, {32, 64, 1, kEmu},
    {128, 32, 0, kOz}, {128, 32, 1, kOz}, {8, 8, 0}};
constexpr TileCfg kCandidates32[] = {{64, 64, 0}, {64, 32, 0}, {32, 64, 0}, {32, 32, 0},
                                     {64, 64, 1}, {64, 32, 1}, {32, 64, 1}, {32, 32, 1}};
struct CandidateList {
  const TileCfg* t;
  int n;
};
// the calling thread's candidates for a contraction of type T
template <typename T>
CandidateList candidates() {
  if (!std::is_same<T, double>::value)
    return {kCandidates32, (int)(sizeof(kCandidates32) / sizeof(TileCfg))};
  if (t_fp64_engine == kFp64DoubleFloat)
    return {kCandidatesDf, (int)(sizeof(kCandidatesDf) / sizeof(TileCfg))};
  return {kCandidates64, (int)(sizeof(kCandidates64) / sizeof(TileCfg))};
}

std::atomic<int> g_autotune{-1};   // -1: not read yet from TTGB_AUTOTUNE
std::shared_mutex g_tune_mu;   // readers: every launch of a recorded class; writers: tuning
std::unordered_map<uint64_t, int> g_tune_table;   // class -> candidate index (-1: being tuned)
std::atomic<int64_t> g_tune_runs{0};
std::once_flag g_table_once;
std::string g_table_path;   // TTGB_AUTOTUNE_TABLE: records read at first use, new ones appended

// Reads "class candidate" lines (hex, decimal) of a previous process into the table.
void load_table() {
  const char* e = std::getenv("TTGB_AUTOTUNE_TABLE");
  if (!e || !*e) return;
  std::unique_lock<std::shared_mutex> g(g_tune_mu);
  g_table_path = e;
  FILE* f = std::fopen(e, "r");
  if (!f) return;
  unsigned long long k = 0;
  int c = 0;
  while (std::fscanf(f, "%llx %d", &k, &c) == 2)
    if (c >= 0) g_tune_table[(uint64_t)k] = c;
  std::fclose(f);
}

void append_record(uint64_t key, int c) {   // caller holds the unique lock
  if (g_table_path.empty() || c < 0) return;
  FILE* f = std::fopen(g_table_path.c_str(), "a");
  if (!f) return;
  std::fprintf(f, "%llx %d\n", (unsigned long long)key, c);
  std::fclose(f);
}

thread_local bool t_no_tuning_runs = false;   // set by NoTuningScope

bool autotune_on() {
  int v = g_autotune.load();
  if (v < 0) {
    const char* e = std::getenv("TTGB_AUTOTUNE");
    v = (e && e[0] == '0') ? 0 : 1;
    g_autotune.store(v);
  }
  return v == 1;
}

int log2_bucket(int64_t v) {
  int b = 0;
  while ((int64_t(1) << b) < v && b < 40) ++b;
  return b;
}

// largest address offset of an index of the given extent
int64_t ax_span(const Ax& a, int64_t extent) {
  if (extent <= 0) return 0;
  if (a.e0 >= extent) return (extent - 1) * a.s0;
  return (a.e0 - 1) * a.s0 + ((extent - 1) / a.e0) * a.s1;
}

template <typename T>
bool overlaps(const T* x, int64_t xs, const T* y, int64_t ys) {
  return x < y + ys + 1 && y < x + xs + 1;
}

// CTAs a split-K launch aims at, in multiples of the SM count (TTGB_SPLIT_TARGET, default 2)
double split_target() {
  static const double v = [] {
    const char* e = std::getenv("TTGB_SPLIT_TARGET");
    const double x = e ? std::atof(e) : 2.0;
    return (x > 0.0 && x <= 16.0) ? x : 2.0;
  }();
  return v;
}

template <typename T>
int heuristic_split(const ContractDescT<T>& d, int bm, int bn, int sms, bool force) {
  const int64_t t = (int64_t)cdiv(d.M, bm) * cdiv(d.N, bn) * d.batch;
  const int64_t target = (int64_t)(split_target() * sms);
  if (!force && !(t < sms && d.K >= 128)) return 1;
  int splitk = (int)((target + t - 1) / t);
  const int maxsplit = d.K / 64;
  if (splitk > maxsplit) splitk = maxsplit;
  return splitk < 1 ? 1 : splitk;
}

// A triangular right factor is an inverse R factor: its columns are graded, and the product has to be
// accurate relative to each element's own terms (the tensor-core kernel's bound is per row and
// column: with it a CholeskyQR of a matrix of condition 1e12 left a residual of 2e-13, not 7e-16).
template <typename T>
bool componentwise(const ContractDescT<T>& d) {
  return (d.tri & kTriUpperB) != 0;
}

// Whether d may be a digit product.
template <typename T>
bool digits_allowed(const ContractDescT<T>& d) {
  return std::is_same<T, double>::value && !t_no_digits && !componentwise(d);
}

// Whether candidate t may run d: no workspace for a caller that must not allocate or whose stream is being
// captured.
template <typename T>
bool usable(const TileCfg& t, const ContractDescT<T>& d, cudaStream_t stream) {
  if ((t.kind == kEmu || t.kind == kOz) && !digits_allowed(d)) return false;
  if (t.kind != kOz && std::min(cdiv(d.M, t.bm), cdiv(d.N, t.bn)) >= 65536) return false;   // tiles in the grid
  if constexpr (std::is_same<T, double>::value) {
    if (t.kind == kOz) {
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
      return !t_no_tuning_runs && oz_takes(d) && cudaStreamIsCapturing(stream, &cap) == cudaSuccess &&
             cap == cudaStreamCaptureStatusNone;
    }
  }
  return true;
}

// split-K of candidate t
template <typename T>
int tile_split(const TileCfg& t, const ContractDescT<T>& d, int sms) {
  if constexpr (std::is_same<T, double>::value) {
    if (t.kind == kOz) {   // one tile per SM at most: a tile takes the SM's tensor memory
      const int64_t tiles = oz_tiles(d);
      const int s = (int)std::min<int64_t>(sms / std::max<int64_t>(1, tiles), d.K / kOzChunk);
      return s < 1 ? 1 : s;
    }
  }
  return heuristic_split(d, t.bm, t.bn, sms, true);
}

template <int BM, int BN>
void launch_emu(const KParams<double>& p, dim3 grid, cudaStream_t stream) {
  using Tile = EmuTile<BM, BN>;
  smem_optin((const void*)contract_emu_kernel<BM, BN>, (int)Tile::kSmem);
  launch_early(contract_emu_kernel<BM, BN>, grid, Tile::kThreads, Tile::kSmem, stream, p);
  TTGB_CHECK_LAUNCH();
}

template <typename T>
void launch_tiles(const ContractDescT<T>& d, KParams<T> p, TileCfg t, int splitk, cudaStream_t stream) {
  int kchunk = d.K;
  if (splitk > 1) {
    const int unit = t.kind == kOz ? kOzChunk : t.kind == kEmu ? kEmuK : BK;
    kchunk = (int)cdiv(cdiv(d.K, splitk), unit) * unit;
    splitk = (int)cdiv(d.K, kchunk);
  }
  p.splitk = splitk;
  p.kchunk = kchunk;
  if (splitk > 1 && !(d.c_zero && d.beta == T(0))) {
    int64_t total = (int64_t)d.M * d.N * d.batch;
    unsigned g = cdiv(total, 256);
    if (g > 8192) g = 8192;
    launch_early(scale_output_kernel<T>, g, 256, 0, stream, p.C, p.M, p.N, p.batch, p.cm, p.cn, p.c_bs, p.beta);
    TTGB_CHECK_LAUNCH();
  }
  if constexpr (std::is_same<T, double>::value) {
    if (t.kind == kOz) {
      if (oz_contract(d, splitk, kchunk, stream)) return;
      t = d.M >= d.N ? TileCfg{64, 32, 0, kEmu} : TileCfg{32, 64, 0, kEmu};   // digits made per tile
    }
  }
  const int bm = t.bm, bn = t.bn;
  dim3 grid(cdiv(d.N, bn), cdiv(d.M, bm), (unsigned)(d.batch * splitk));
  p.tall = grid.y >= 65536;
  if (p.tall) std::swap(grid.x, grid.y);
  TTGB_REQUIRE(grid.y < 65536 && grid.z < 65536, "contraction grid too large");
  if constexpr (std::is_same<T, double>::value) {
    if (t.kind == kEmu) {
      if (bm == 64 && bn == 32) launch_emu<64, 32>(p, grid, stream);
      else if (bm == 32 && bn == 64) launch_emu<32, 64>(p, grid, stream);
      else if (bm == 64 && bn == 16) launch_emu<64, 16>(p, grid, stream);
      else launch_emu<16, 64>(p, grid, stream);
      return;
    }
    if (t.kind == kDf) {
      if (bm == 64 && bn == 32) launch_early(contract_df_kernel<64, 32>, grid, NT, 0, stream, p);
      else if (bm == 32 && bn == 64) launch_early(contract_df_kernel<32, 64>, grid, NT, 0, stream, p);
      else launch_early(contract_df_kernel<32, 32>, grid, NT, 0, stream, p);
    } else if (bm == 8) launch_early(contract_small_kernel, grid, NT, 0, stream, p);
    else if (bm == 16 && bn == 16) launch_early(contract_kernel<T, 16, 16>, grid, NT, 0, stream, p);
    else if (bm == 16 && bn == 32) launch_early(contract_kernel<T, 16, 32>, grid, NT, 0, stream, p);
    else if (bm == 32 && bn == 16) launch_early(contract_kernel<T, 32, 16>, grid, NT, 0, stream, p);
    else launch_early(contract_kernel<T, 32, 32>, grid, NT, 0, stream, p);
  } else {
    if (bm == 64 && bn == 64) launch_early(contract_kernel<T, 64, 64>, grid, NT, 0, stream, p);
    else if (bm == 64 && bn == 32) launch_early(contract_kernel<T, 64, 32>, grid, NT, 0, stream, p);
    else if (bm == 32 && bn == 64) launch_early(contract_kernel<T, 32, 64>, grid, NT, 0, stream, p);
    else launch_early(contract_kernel<T, 32, 32>, grid, NT, 0, stream, p);
  }
  TTGB_CHECK_LAUNCH();
}

template <typename T>
uint64_t tune_key(const ContractDescT<T>& d) {
  const int eng = std::is_same<T, float>::value ? 2
                  : (t_fp64_engine == kFp64DoubleFloat ? 4 : 3) + (t_no_digits ? 2 : 0);
  const int units = (d.am.s0 == 1) | ((d.ak.s0 == 1) << 1) | ((d.bk.s0 == 1) << 2) |
                    ((d.bn.s0 == 1) << 3) | ((d.cm.s0 == 1) << 4);
  uint64_t k = (uint64_t)eng;
  k = k * 64 + (uint64_t)log2_bucket(d.M);
  k = k * 64 + (uint64_t)log2_bucket(d.N);
  k = k * 64 + (uint64_t)log2_bucket(d.K);
  k = k * 64 + (uint64_t)log2_bucket(d.batch);
  k = k * 4 + (uint64_t)(d.tri & 3);
  k = k * 32 + (uint64_t)units;
  k = k * 1024 + (uint64_t)(num_sms() & 1023);   // the GPU model, through its SM count
  return k;
}

// Returns the candidate index to use, tuning the class first when this launch may be repeated (a record of a file
// that names no candidate counts as none).
// -1: use the heuristic. A tuned launch has already written C (tuned = true).
template <typename T>
int tuned_choice(const ContractDescT<T>& d, const KParams<T>& p, cudaStream_t stream,
                 bool& tuned) {
  tuned = false;
  if (d.beta != T(0)) return -1;
  const int64_t sa = (d.batch - 1) * d.a_bs + ax_span(d.am, d.M) + ax_span(d.ak, d.K);
  const int64_t sb = (d.batch - 1) * d.b_bs + ax_span(d.bk, d.K) + ax_span(d.bn, d.N);
  const int64_t sc = (d.batch - 1) * d.c_bs + ax_span(d.cm, d.M) + ax_span(d.cn, d.N);
  if (overlaps<T>(d.C, sc, d.A, sa) || overlaps<T>(d.C, sc, d.B, sb)) return -1;
  std::call_once(g_table_once, load_table);
  const CandidateList cand = candidates<T>();
  const uint64_t key = tune_key(d);
  {
    std::shared_lock<std::shared_mutex> g(g_tune_mu);
    auto it = g_tune_table.find(key);
    if (it != g_tune_table.end() && it->second < cand.n) return it->second;
  }
  {
    std::unique_lock<std::shared_mutex> g(g_tune_mu);
    auto it = g_tune_table.find(key);
    if (it != g_tune_table.end() && it->second < cand.n) return it->second;
    if (t_no_tuning_runs) return -1;   // a caller that must not block: heuristic tile
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
      return -1;
    g_tune_table[key] = -1;   // being tuned: other threads use the heuristic meanwhile
  }
  const int sms = num_sms();
  struct Events {   // destroyed on every exit, also when a launch check throws
    cudaEvent_t e[2] = {nullptr, nullptr};
    ~Events() {
      if (e[0]) cudaEventDestroy(e[0]);
      if (e[1]) cudaEventDestroy(e[1]);
    }
  } evs;
  struct Claim {   // a class whose tuning throws is tuned by a later launch
    uint64_t key;
    bool kept = false;
    ~Claim() {
      if (kept) return;
      std::unique_lock<std::shared_mutex> g(g_tune_mu);
      g_tune_table.erase(key);
    }
  } claim{key};
  cudaEvent_t* ev = evs.e;
  TTGB_CUDA(cudaEventCreate(&ev[0]));
  TTGB_CUDA(cudaEventCreate(&ev[1]));
  int best = -1;
  float best_ms = 0.f;
  for (int c = 0; c < cand.n; ++c) {
    const TileCfg& t = cand.t[c];
    if (!usable(t, d, stream)) continue;
    const int split = t.split ? tile_split(t, d, sms) : 1;
    if (t.split && split == 1) continue;   // the same launch as the unsplit candidate
    // The first run loads the code and keeps the GPU busy while the second one is enqueued: timed from an
    // idle stream, a candidate of several launches is charged for the host's time between them.
    launch_tiles(d, p, t, split, stream);
    TTGB_CUDA(cudaEventRecord(ev[0], stream));
    launch_tiles(d, p, t, split, stream);
    TTGB_CUDA(cudaEventRecord(ev[1], stream));
    TTGB_CUDA(cudaEventSynchronize(ev[1]));
    float ms = 0.f;
    TTGB_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
    if (best < 0 || ms < best_ms) { best = c; best_ms = ms; }
  }
  g_tune_runs.fetch_add(1);
  {
    std::unique_lock<std::shared_mutex> g(g_tune_mu);
    g_tune_table[key] = best;
    append_record(key, best);
    claim.kept = true;
  }
  tuned = true;
  return best;
}

template <typename T>
void launch_contract(const ContractDescT<T>& d, cudaStream_t stream, bool deterministic) {
  if (d.M <= 0 || d.N <= 0 || d.batch <= 0) return;
  // the tuning runs write C before the chosen tile runs again: those launches may not assume C = 0
  ContractDescT<T> dz = d;
  dz.c_zero = false;
  KParams<T> p;
  p.M = d.M; p.N = d.N; p.K = d.K; p.batch = d.batch;
  p.A = d.A; p.am = to_dev(d.am, d.M); p.ak = to_dev(d.ak, d.K); p.a_bs = d.a_bs;
  p.B = d.B; p.bk = to_dev(d.bk, d.K); p.bn = to_dev(d.bn, d.N); p.b_bs = d.b_bs;
  p.C = d.C; p.cm = to_dev(d.cm, d.M); p.cn = to_dev(d.cn, d.N); p.c_bs = d.c_bs;
  p.alpha = d.alpha; p.beta = d.beta;
  p.scale = d.alpha != T(1); p.keep = d.beta != T(0);
  p.tri = d.tri;
  if (d.K <= 0) {  // empty sum: C = beta * C
    launch_early(scale_output_kernel<T>, std::min(cdiv((int64_t)d.M * d.N * d.batch, 256), 4096u), 256, 0, stream,
        p.C, p.M, p.N, p.batch, p.cm, p.cn, p.c_bs, p.beta);
    TTGB_CHECK_LAUNCH();
    return;
  }
  const int sms = num_sms();
  const double work = (double)d.M * d.N * d.K * d.batch;
  if (!deterministic && autotune_on() && work > kTuneWork) {
    bool tuned = false;
    const int c = tuned_choice(dz, p, stream, tuned);
    // after tuning, C holds the last candidate's result: the chosen tile runs once more, so the
    // first launch of a class gives what every later launch of the class computes
    if (c >= 0 && usable(candidates<T>().t[c], d, stream)) {
      const TileCfg& t = candidates<T>().t[c];
      launch_tiles(tuned ? dz : d, p, t,
                   t.split ? tile_split(t, d, sms) : 1, stream);
      return;
    }
  }
  // occupancy heuristic: the largest tile whose grid still gives two CTAs per SM, split-K when
  // even the smallest tiles leave SMs idle
  auto tiles = [&](int bm, int bn) { return (int64_t)cdiv(d.M, bm) * cdiv(d.N, bn) * d.batch; };
  const int64_t target = 2 * (int64_t)sms;
  TileCfg t{64, 64, 0};
  if (std::is_same<T, double>::value) {
    if (!digits_allowed(d)) t.kind = t_fp64_engine == kFp64DoubleFloat ? kDf : kFma;
    else if (work > 4e6) t.kind = kEmu;
    t.bm = t.bn = 32;
    // 200 x 300 x 100 (6 M): 22 us either way; 60 x 13440 x 60 (48 M): 40 us with digits made per tile, 29 us
    // with digits made beforehand; 176 x 5632 x 88 (87 M): 60 and 31 us
    const TileCfg oz{128, 32, 1, kOz};
    if (t.kind == kEmu && work > 3e7 && usable(oz, d, stream)) {
      launch_tiles(d, p, oz, deterministic ? 1 : tile_split(oz, d, sms), stream);
      return;
    }
    if (t.kind == kEmu) {
      if (d.N <= 16) { t.bm = 64; t.bn = 16; }
      else if (d.M <= 16) { t.bm = 16; t.bn = 64; }
      else if (d.M >= d.N) t.bm = 64;
      else t.bn = 64;
    } else if (t.kind == kFma && tiles(32, 32) < target) {
      // 8 x 8 where 16 x 16 would leave half of the SMs without a tile
      t.bm = t.bn = 2 * tiles(16, 16) <= sms ? 8 : 16;
    }
  } else if (tiles(64, 64) < target) {
    if (d.M >= d.N) { t.bm = 64; t.bn = 32; } else { t.bm = 32; t.bn = 64; }
    if (tiles(t.bm, t.bn) < target) { t.bm = 32; t.bn = 32; }
  }
  launch_tiles(d, p, t, deterministic ? 1 : heuristic_split(d, t.bm, t.bn, sms, false), stream);
}

}  // namespace

int set_autotune(int mode) {
  const int prev = autotune_on() ? 1 : 0;
  if (mode == 0 || mode == 1) g_autotune.store(mode);
  return prev;
}

int64_t autotune_classes() {
  std::shared_lock<std::shared_mutex> g(g_tune_mu);
  return (int64_t)g_tune_table.size();
}

NoTuningScope::NoTuningScope() : prev_(t_no_tuning_runs) { t_no_tuning_runs = true; }
NoTuningScope::~NoTuningScope() { t_no_tuning_runs = prev_; }

NoDigitsScope::NoDigitsScope(bool on) : prev_(t_no_digits) { t_no_digits = t_no_digits || on; }
NoDigitsScope::~NoDigitsScope() { t_no_digits = prev_; }

int set_no_digits(int mode) {
  const int prev = t_no_digits ? 1 : 0;
  if (mode == 0 || mode == 1) t_no_digits = mode == 1;
  return prev;
}

int fp64_engine() { return t_fp64_engine; }
Fp64EngineScope::Fp64EngineScope(int engine) : prev_(t_fp64_engine) { t_fp64_engine = engine; }
Fp64EngineScope::~Fp64EngineScope() { t_fp64_engine = prev_; }

void contract(const ContractDesc& d, cudaStream_t stream, bool deterministic) {
  launch_contract<double>(d, stream, deterministic);
}

void contract(const ContractDescF& d, cudaStream_t stream, bool deterministic) {
  launch_contract<float>(d, stream, deterministic);
}

// --------------------------------------------------------------------------------------------
// AMEn contraction recipes
// --------------------------------------------------------------------------------------------

template <typename T>
static void local_product_t(const LocalOpDims& d, const T* phi_l, const T* A, const T* phi_r,
                            const T* x, T* y, T* w1, T* w2, cudaStream_t stream, T alpha, T beta,
                            const SparseCore* sp) {
  // step 1: W[(l,s),(n,R)] = sum_r Phi_l[(l,s), r] X[r, (n,R)]
  {
    ContractDescT<T> c;
    c.M = (int)(d.rl * d.s); c.N = (int)(d.n * d.R); c.K = (int)d.r;
    c.A = phi_l; c.am = Ax::one(d.r); c.ak = Ax::one(1);
    c.B = x; c.bk = Ax::one(d.n * d.R); c.bn = Ax::one(1);
    c.C = w1; c.cm = Ax::one(d.n * d.R); c.cn = Ax::one(1);
    contract(c, stream);
  }
  // step 2 (batched over l): Y2_l[(m,S), R] = sum_{(s,n)} A[s,m,n,S] W_l[(s,n), R]
  if (sp && sp->use) {
    // from the nonzeros: Y2[l,(m,S),R] = sum A[s,m,n,S] W[l,s,n,R]
    const StageDims g{d.rl, d.R, d.s * d.n * d.R, d.m * d.S * d.R, d.R, d.n * d.R, d.R};
    sparse_stage(sp->lp, w1, w2, g, stream);
  } else {
    ContractDescT<T> c;
    c.M = (int)(d.m * d.S); c.N = (int)d.R; c.K = (int)(d.s * d.n); c.batch = (int)d.rl;
    c.A = A; c.am = Ax::two(d.S, d.n * d.S, 1); c.ak = Ax::two(d.n, d.m * d.n * d.S, d.S);
    c.B = w1; c.bk = Ax::one(d.R); c.bn = Ax::one(1); c.b_bs = d.s * d.n * d.R;
    c.C = w2; c.cm = Ax::one(d.R); c.cn = Ax::one(1); c.c_bs = d.m * d.S * d.R;
    contract(c, stream);
  }
  // step 3: y[(l,m), L] = alpha * sum_{(S,R)} Y2[(l,m),(S,R)] Phi_r[L,(S,R)] + beta * y
  {
    ContractDescT<T> c;
    c.M = (int)(d.rl * d.m); c.N = (int)d.RL; c.K = (int)(d.S * d.R);
    c.A = w2; c.am = Ax::one(d.S * d.R); c.ak = Ax::one(1);
    c.B = phi_r; c.bk = Ax::one(1); c.bn = Ax::one(d.S * d.R);
    c.C = y; c.cm = Ax::one(d.RL); c.cn = Ax::one(1);
    c.alpha = alpha; c.beta = beta;
    contract(c, stream);
  }
}

void local_product(const LocalOpDims& d, const double* phi_l, const double* A, const double* phi_r,
                   const double* x, double* y, double* w1, double* w2, cudaStream_t stream,
                   double alpha, double beta, const SparseCore* sp) {
  local_product_t<double>(d, phi_l, A, phi_r, x, y, w1, w2, stream, alpha, beta, sp);
}

void local_product(const LocalOpDims& d, const float* phi_l, const float* A, const float* phi_r,
                   const float* x, float* y, float* w1, float* w2, cudaStream_t stream,
                   float alpha, float beta, const SparseCore* sp) {
  local_product_t<float>(d, phi_l, A, phi_r, x, y, w1, w2, stream, alpha, beta, sp);
}

size_t phi_A_workspace(const PhiDims& d) {
  size_t fwd = size_t(d.s * d.r * d.M * d.L + d.r * d.L * d.N * d.S);
  size_t bck = size_t(d.l * d.M * d.S * d.R + d.l * d.s * d.N * d.R);
  return fwd > bck ? fwd : bck;
}

void phi_fwd_A(const PhiDims& d, const double* phi, const double* left, const double* A,
               const double* right, double* out, double* work, cudaStream_t stream,
               const SparseCore* sp) {
  double* T1 = work;                              // [s, r, M, L]
  double* T2 = work + d.s * d.r * d.M * d.L;      // [r, L, N, S]
  {  // T1[(s,r),(M,L)] = sum_l Phi[l,(s,r)] left[l,(M,L)]
    ContractDesc c;
    c.M = (int)(d.s * d.r); c.N = (int)(d.M * d.L); c.K = (int)d.l;
    c.A = phi; c.am = Ax::one(1); c.ak = Ax::one(d.s * d.r);
    c.B = left; c.bk = Ax::one(d.M * d.L); c.bn = Ax::one(1);
    c.C = T1; c.cm = Ax::one(d.M * d.L); c.cn = Ax::one(1);
    contract(c, stream);
  }
  if (sp && sp->use) {
    // from the nonzeros, into the key-major layout T2'[N,S,r,L]
    const StageDims g{d.r, d.L, d.M * d.L, d.L, d.r * d.L, d.r * d.M * d.L, d.L};
    sparse_stage(sp->fw, T1, T2, g, stream);
    // out[L,S,R] = sum_{(r,N)} T2'[N,S,r,L] right[r,N,R]   (batched over S)
    ContractDesc c;
    c.M = (int)d.L; c.N = (int)d.R; c.K = (int)(d.r * d.N); c.batch = (int)d.S;
    c.A = T2; c.am = Ax::one(1); c.ak = Ax::two(d.N, d.L, d.S * d.r * d.L); c.a_bs = d.r * d.L;
    c.B = right; c.bk = Ax::one(d.R); c.bn = Ax::one(1);
    c.C = out; c.cm = Ax::one(d.S * d.R); c.cn = Ax::one(1); c.c_bs = d.R;
    contract(c, stream);
    return;
  }
  {  // T2[(r,L),(N,S)] = sum_{(s,M)} T1[s,r,M,L] A[s,M,N,S]
    ContractDesc c;
    c.M = (int)(d.r * d.L); c.N = (int)(d.N * d.S); c.K = (int)(d.s * d.M);
    c.A = T1; c.am = Ax::two(d.L, d.M * d.L, 1); c.ak = Ax::two(d.M, d.r * d.M * d.L, d.L);
    c.B = A; c.bk = Ax::two(d.M, d.M * d.N * d.S, d.N * d.S); c.bn = Ax::one(1);
    c.C = T2; c.cm = Ax::one(d.N * d.S); c.cn = Ax::one(1);
    contract(c, stream);
  }
  {  // out[L,S,R] = sum_{(r,N)} T2[r,L,N,S] right[r,N,R]   (batched over S)
    ContractDesc c;
    c.M = (int)d.L; c.N = (int)d.R; c.K = (int)(d.r * d.N); c.batch = (int)d.S;
    c.A = T2; c.am = Ax::one(d.N * d.S); c.ak = Ax::two(d.N, d.L * d.N * d.S, d.S); c.a_bs = 1;
    c.B = right; c.bk = Ax::one(d.R); c.bn = Ax::one(1);
    c.C = out; c.cm = Ax::one(d.S * d.R); c.cn = Ax::one(1); c.c_bs = d.R;
    contract(c, stream);
  }
}

void phi_bck_A(const PhiDims& d, const double* phi, const double* left, const double* A,
               const double* right, double* out, double* work, cudaStream_t stream,
               const SparseCore* sp) {
  double* T1 = work;                              // [l, M, S, R]
  double* T2 = work + d.l * d.M * d.S * d.R;      // [l, s, N, R]
  {  // T1[(l,M),(S,R)] = sum_L left[(l,M), L] Phi[L,(S,R)]
    ContractDesc c;
    c.M = (int)(d.l * d.M); c.N = (int)(d.S * d.R); c.K = (int)d.L;
    c.A = left; c.am = Ax::one(d.L); c.ak = Ax::one(1);
    c.B = phi; c.bk = Ax::one(d.S * d.R); c.bn = Ax::one(1);
    c.C = T1; c.cm = Ax::one(d.S * d.R); c.cn = Ax::one(1);
    contract(c, stream);
  }
  if (sp && sp->use) {   // from the nonzeros: key (s,N), free (l, R)
    const StageDims g{d.l, d.R, d.M * d.S * d.R, d.s * d.N * d.R, d.R, d.S * d.R, d.R};
    sparse_stage(sp->bk, T1, T2, g, stream);
  } else {  // T2[l,s,N,R] = sum_{(M,S)} T1[l,M,S,R] A[s,M,N,S]; rows (l,R), cols (s,N)
    ContractDesc c;
    c.M = (int)(d.l * d.R); c.N = (int)(d.s * d.N); c.K = (int)(d.M * d.S);
    c.A = T1; c.am = Ax::two(d.R, d.M * d.S * d.R, 1); c.ak = Ax::two(d.S, d.S * d.R, d.R);
    c.B = A; c.bk = Ax::two(d.S, d.N * d.S, 1); c.bn = Ax::two(d.N, d.M * d.N * d.S, d.S);
    c.C = T2; c.cm = Ax::two(d.R, d.s * d.N * d.R, 1); c.cn = Ax::two(d.N, d.N * d.R, d.R);
    contract(c, stream);
  }
  {  // out[(l,s), r] = sum_{(N,R)} T2[(l,s),(N,R)] right[r,(N,R)]
    ContractDesc c;
    c.M = (int)(d.l * d.s); c.N = (int)d.r; c.K = (int)(d.N * d.R);
    c.A = T2; c.am = Ax::one(d.N * d.R); c.ak = Ax::one(1);
    c.B = right; c.bk = Ax::one(1); c.bn = Ax::one(d.N * d.R);
    c.C = out; c.cm = Ax::one(d.r); c.cn = Ax::one(1);
    contract(c, stream);
  }
}

size_t phi_rhs_workspace(const PhiRhsDims& d) {
  size_t f = size_t(d.n * d.B * d.r), b = size_t(d.b * d.n * d.R);
  return f > b ? f : b;
}

void phi_fwd_rhs(const PhiRhsDims& d, const double* phi, const double* core_b, const double* core,
                 double* out, double* work, cudaStream_t stream) {
  {  // T[(n,B), r] = sum_b core_b[b,(n,B)] Phi[b, r]
    ContractDesc c;
    c.M = (int)(d.n * d.B); c.N = (int)d.r; c.K = (int)d.b;
    c.A = core_b; c.am = Ax::one(1); c.ak = Ax::one(d.n * d.B);
    c.B = phi; c.bk = Ax::one(d.r); c.bn = Ax::one(1);
    c.C = work; c.cm = Ax::one(d.r); c.cn = Ax::one(1);
    contract(c, stream);
  }
  {  // out[B, R] = sum_{(r,n)} T[n,B,r] core[r,n,R]
    ContractDesc c;
    c.M = (int)d.B; c.N = (int)d.R; c.K = (int)(d.r * d.n);
    c.A = work; c.am = Ax::one(d.r); c.ak = Ax::two(d.n, 1, d.B * d.r);
    c.B = core; c.bk = Ax::one(d.R); c.bn = Ax::one(1);
    c.C = out; c.cm = Ax::one(d.R); c.cn = Ax::one(1);
    contract(c, stream);
  }
}

void phi_bck_rhs(const PhiRhsDims& d, const double* phi, const double* core_b, const double* core,
                 double* out, double* work, cudaStream_t stream) {
  {  // T[(b,n), R] = sum_B core_b[(b,n), B] Phi[B, R]
    ContractDesc c;
    c.M = (int)(d.b * d.n); c.N = (int)d.R; c.K = (int)d.B;
    c.A = core_b; c.am = Ax::one(d.B); c.ak = Ax::one(1);
    c.B = phi; c.bk = Ax::one(d.R); c.bn = Ax::one(1);
    c.C = work; c.cm = Ax::one(d.R); c.cn = Ax::one(1);
    contract(c, stream);
  }
  {  // out[b, r] = sum_{(n,R)} T[b,(n,R)] core[r,(n,R)]
    ContractDesc c;
    c.M = (int)d.b; c.N = (int)d.r; c.K = (int)(d.n * d.R);
    c.A = work; c.am = Ax::one(d.n * d.R); c.ak = Ax::one(1);
    c.B = core; c.bk = Ax::one(1); c.bn = Ax::one(d.n * d.R);
    c.C = out; c.cm = Ax::one(d.r); c.cn = Ax::one(1);
    contract(c, stream);
  }
}

size_t local_rhs_workspace(int64_t b, int64_t n, int64_t B, int64_t r, int64_t R) {
  (void)B; (void)r;
  return size_t(b * n * R);
}

void local_rhs(int64_t b, int64_t n, int64_t B, int64_t r, int64_t R, const double* phi_l,
               const double* core_b, const double* phi_r, double alpha, double* out, double* work,
               cudaStream_t stream) {
  {  // T[(b,n), R] = sum_B core_b[(b,n),B] Phi_r[B,R]
    ContractDesc c;
    c.M = (int)(b * n); c.N = (int)R; c.K = (int)B;
    c.A = core_b; c.am = Ax::one(B); c.ak = Ax::one(1);
    c.B = phi_r; c.bk = Ax::one(R); c.bn = Ax::one(1);
    c.C = work; c.cm = Ax::one(R); c.cn = Ax::one(1);
    contract(c, stream);
  }
  {  // out[r, (n,R)] = alpha * sum_b Phi_l[b, r] T[b, (n,R)]
    ContractDesc c;
    c.M = (int)r; c.N = (int)(n * R); c.K = (int)b;
    c.A = phi_l; c.am = Ax::one(1); c.ak = Ax::one(r);
    c.B = work; c.bk = Ax::one(n * R); c.bn = Ax::one(1);
    c.C = out; c.cm = Ax::one(n * R); c.cn = Ax::one(1);
    c.alpha = alpha;
    contract(c, stream);
  }
}

}  // namespace ttgb
