// Structure-aware A-core stage (see sparse_a.cuh).
#include <algorithm>

#include "reduce.cuh"
#include "sparse_a.cuh"
#include "tc_gemm.cuh"

namespace ttgb {

namespace {

constexpr int kThreads = 256;

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(kThreads)
sparse_stage_kernel(const int* rp, const int* ja, const int* jb, const T* val, const T* in, T* out,
                    float* out_lo, StageDims g) {
  __shared__ T sv[SparseCore::kMaxRow];
  __shared__ int64_t soff[SparseCore::kMaxRow];
  stream_wait();
  if (g.gate != nullptr && *g.gate != 0) return;
  const int key = blockIdx.x;
  const int beg = rp[key];
  const int cnt = rp[key + 1] - beg;
  for (int j = threadIdx.x; j < cnt; j += blockDim.x) {
    sv[j] = val[beg + j];
    soff[j] = (int64_t)ja[beg + j] * g.pa + (int64_t)jb[beg + j] * g.pb;
  }
  __syncthreads();
  const int64_t total = g.O1 * g.O2;
  const int64_t koff = g.ke0 > 0 ? (key % g.ke0) * g.sk + (key / g.ke0) * g.sk1 : (int64_t)key * g.sk;
  T* ob = out + koff;
  for (int64_t t = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.y * blockDim.x) {
    const int64_t o1 = t / g.O2, o2 = t - o1 * g.O2;
    const T* ib = in + o1 * g.si1 + o2;
    T acc = T(0);
    for (int j = 0; j < cnt; ++j) acc = fma(sv[j], ib[soff[j]], acc);
    const int64_t o = o1 * g.so1 + o2;
    if constexpr (SPLIT) {
      const float h = to_tf32((float)acc);
      ob[o] = h;
      out_lo[koff + o] = to_tf32((float)acc - h);
    } else {
      ob[o] = acc;
    }
  }
}

template <typename T, bool SPLIT>
void launch_stage(const SparseCsr& c, const T* val, const T* in, T* out, float* lo,
                  const StageDims& g, cudaStream_t s) {
  if (c.keys <= 0 || g.O1 <= 0 || g.O2 <= 0) return;
  TTGB_REQUIRE(c.keys < (int64_t(1) << 31) && c.rp != nullptr, "sparse stage: grouping not built");
  const int64_t total = g.O1 * g.O2;
  int64_t gy = (int64_t)cdiv(total, kThreads);
  const int64_t want = std::max<int64_t>(1, (int64_t)8 * num_sms() / c.keys);
  gy = std::max<int64_t>(1, std::min<int64_t>({gy, want, 65535}));
  dim3 grid((unsigned)c.keys, (unsigned)gy);
  launch_early(sparse_stage_kernel<T, SPLIT>, grid, kThreads, 0, s, c.rp, c.a, c.b, val, in, out, lo, g);
  TTGB_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------------------------
// The four groupings of a core's nonzeros, built on the device: one warp per key walks the key's
// candidates in (a, b) order. The first launch counts them (all groupings, and the last block turns
// the counts into row pointers and reports the totals to pinned host memory), the second writes the
// entries at the positions that the ballots give. Measured for a 3 x 64 x 64 x 3 core: the copy of the
// core to the host, the scan there and 20 uploads took about 190 us, the two launches and the wait
// between them 25 us.
// ---------------------------------------------------------------------------------------------
struct Grouping {
  int64_t keys;       // rows of the CSR
  int64_t cand;       // candidates per key: c -> (a, b) = (c / cb, c % cb)
  int64_t cb;
  int64_t kb;         // key -> (k1, k0) = (key / kb, key % kb)
  int64_t o1, o0;     // element offset: k1 o1 + k0 o0 + a oa + b ob
  int64_t oa, ob;
};

struct Groupings {
  Grouping g[SparseCore::kGroupings];
};

Groupings groupings(int64_t s, int64_t M, int64_t N, int64_t S) {
  const int64_t os = M * N * S, om = N * S, on = S;   // strides of A[s, m, n, S]
  Groupings r;
  r.g[0] = {M * S, s * N, N, S, om, 1, os, on};   // lp: key (m, S), pairs (s, n)
  r.g[1] = {N * S, s * M, M, S, on, 1, os, om};   // fw: key (n, S), pairs (s, m)
  r.g[2] = {s * N, M * S, S, N, os, on, om, 1};   // bk: key (s, n), pairs (m, S)
  r.g[3] = {s * M, N * S, S, M, os, om, on, 1};   // rh: key (s, m), pairs (n, S)
  return r;
}

__device__ __forceinline__ double candidate(const Grouping& g, const double* A, int64_t key, int64_t c) {
  return A[(key / g.kb) * g.o1 + (key % g.kb) * g.o0 + (c / g.cb) * g.oa + (c % g.cb) * g.ob];
}

// rp (kGroupings arrays of keys + 1 row pointers, one after the other), info: {nonzeros, longest row
// over all groupings}
__global__ void __launch_bounds__(kThreads) sparse_count_kernel(const double* A, Groupings gs,
                                                                int* rp, unsigned* counter, int64_t* info) {
  stream_wait();
  __shared__ int longest;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t key = (int64_t)blockIdx.x * (kThreads / 32) + warp;
  int64_t off = 0;
#pragma unroll
  for (int q = 0; q < SparseCore::kGroupings; ++q) {
    const Grouping& g = gs.g[q];
    if (key >= 0 && key < g.keys) {
      int n = 0;
      for (int64_t c = lane; c < g.cand; c += 32) n += candidate(g, A, key, c) != 0.0 ? 1 : 0;
      n = __reduce_add_sync(0xffffffffu, n);
      if (lane == 0) rp[off + key + 1] = n;
    }
    key -= g.keys;
    off += g.keys + 1;
  }
  if (!red::take_last_ticket(counter)) return;
  if (threadIdx.x == 0) longest = 0;
  __syncthreads();
  if (warp < SparseCore::kGroupings) {   // one warp per grouping: inclusive sums in place, 32 keys at a time
    int* p = rp;
    for (int q = 0; q < warp; ++q) p += gs.g[q].keys + 1;
    const int64_t keys = gs.g[warp].keys;
    long long carry = 0;
    int most = 0;
    for (int64_t k0 = 0; k0 < keys; k0 += 32) {
      const int64_t k = k0 + lane;
      int v = k < keys ? __ldcg(p + k + 1) : 0;
      most = max(most, v);
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
      }
      if (k < keys) p[k + 1] = (int)(carry + v);
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) {
      p[0] = 0;
      atomicMax(&longest, most);
      if (warp == 0) info[0] = carry;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) info[1] = longest;
  red::reset_ticket(counter);
}

__global__ void __launch_bounds__(kThreads) sparse_fill_kernel(const double* A, Grouping g,
                                                               const int* rp, int* ja, int* jb,
                                                               double* val, float* val32) {
  stream_wait();
  const int lane = threadIdx.x & 31;
  const int64_t key = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (key >= g.keys) return;
  int at = rp[key];
  for (int64_t c0 = 0; c0 < g.cand; c0 += 32) {
    const int64_t c = c0 + lane;
    const double v = c < g.cand ? candidate(g, A, key, c) : 0.0;
    const unsigned hit = __ballot_sync(0xffffffffu, v != 0.0);
    if (v != 0.0) {
      const int i = at + __popc(hit & ((1u << lane) - 1u));
      ja[i] = (int)(c / g.cb);
      jb[i] = (int)(c % g.cb);
      val[i] = v;
      val32[i] = (float)v;
    }
    at += __popc(hit);
  }
}

// a few words of pinned host memory per host thread, kept for the thread's lifetime
int64_t* pinned_info() {
  struct Holder {
    int64_t* p = nullptr;
    ~Holder() { if (p) cudaFreeHost(p); }
  };
  static thread_local Holder h;
  if (!h.p) TTGB_CUDA(cudaMallocHost((void**)&h.p, 64));
  return h.p;
}

}  // namespace

void SparseCore::build(const double* A, int64_t s_, int64_t M_, int64_t N_, int64_t S_,
                       cudaStream_t st, unsigned which) {
  s = s_; M = M_; N = N_; S = S_;
  use = false;
  const int64_t ne = s * M * N * S;
  if (ne <= 0 || s * N >= (int64_t(1) << 31) || M * S >= (int64_t(1) << 31)) return;
  const Groupings gs = groupings(s, M, N, S);
  int64_t keys = 0;
  for (const Grouping& g : gs.g) keys += g.keys;
  int groups = 0;
  for (int q = 0; q < kGroupings; ++q) groups += (which >> q) & 1u;
  // Row pointers, ticket counter, and the entries: allocated for the most nonzeros that a core in
  // use can have where that is small, so that nothing is allocated between the count and the fill.
  const int64_t most = ne / 4;
  const bool early = most * groups <= (int64_t(1) << 16);
  const size_t head = ((size_t)(keys + kGroupings + 1) + 3) / 4 * 4;   // ints, to 16 bytes
  const auto entry_bytes = [&](int64_t n) { return (size_t)groups * (size_t)n * 20; };   // 8 + 3 x 4
  head_.reset(head * 4 + (early ? entry_bytes(most) : 0), st);
  int* row_ptr = reinterpret_cast<int*>(head_.p);
  unsigned* counter = reinterpret_cast<unsigned*>(row_ptr + keys + kGroupings);
  TTGB_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), st));
  int64_t* info = pinned_info();
  launch_early(sparse_count_kernel, cdiv(keys, kThreads / 32), kThreads, 0, st, A, gs, row_ptr, counter, info);
  TTGB_CHECK_LAUNCH();
  TTGB_CUDA(cudaStreamSynchronize(st));
  const int64_t nnz = info[0];
  if (4 * nnz >= ne || info[1] > kMaxRow) return;   // dense enough for the GEMM path
  SparseCsr* csr[kGroupings] = {&lp, &fw, &bk, &rh};
  if (!early) entries_.reset(entry_bytes(nnz), st);
  const int64_t per = early ? most : nnz;
  double* val = reinterpret_cast<double*>(early ? head_.p + head * 4 : entries_.p);
  float* val32 = reinterpret_cast<float*>(val + groups * per);
  int* ja = reinterpret_cast<int*>(val32 + groups * per);
  int* rp = row_ptr;
  for (int q = 0; q < kGroupings; ++q) {
    SparseCsr& c = *csr[q];
    c = SparseCsr();
    c.keys = gs.g[q].keys;
    const int* rows = rp;
    rp += c.keys + 1;
    if (!((which >> q) & 1u)) continue;   // its rp stays null: a stage refuses it
    c.rp = rows; c.a = ja; c.b = ja + per; c.val = val; c.val32 = val32;
    launch_early(sparse_fill_kernel, cdiv(c.keys, kThreads / 32), kThreads, 0, st, A, gs.g[q], c.rp, ja, ja + per, val,
                                                                      val32);
    TTGB_CHECK_LAUNCH();
    ja += 2 * per;
    val += per;
    val32 += per;
  }
  use = true;
}

void sparse_stage(const SparseCsr& c, const double* in, double* out, const StageDims& g,
                  cudaStream_t s) {
  launch_stage<double, false>(c, c.val, in, out, nullptr, g, s);
}

void sparse_stage(const SparseCsr& c, const float* in, float* out, const StageDims& g,
                  cudaStream_t s) {
  launch_stage<float, false>(c, c.val32, in, out, nullptr, g, s);
}

void sparse_stage_split(const SparseCsr& c, const float* in, float* hi, float* lo,
                        const StageDims& g, cudaStream_t s) {
  launch_stage<float, true>(c, c.val32, in, hi, lo, g, s);
}

}  // namespace ttgb
