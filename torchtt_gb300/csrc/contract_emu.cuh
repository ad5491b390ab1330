// FP64 contraction on the tensor cores: C = alpha A B + beta C for FP64 operands, computed from exact
// products of 8-bit slices (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59 (2012)). Included by contract.cu inside its anonymous namespace.
//
// Why: GB300's FP64 pipe does 1.9 multiply-adds per clock and SM, mma.sync with BF16 operands about a
// thousand, and 36 slice products replace one FP64 product.
//
// A tile's K chunk of 64 is brought to a common fixed point: column j of B by its largest exponent
// Fj; then row k of B by the largest exponent kb(k) that this leaves in it, which is folded into A's
// column k (their product does not change); then row i of A by Ei = max_k exponent(a_ik) + kb(k), and
// column j of B once more by Ec = max_k exponent(b_kj) - Fj - kb(k). An element becomes a signed 62-bit integer, cut into 8 balanced 8-bit digits, which BF16 holds
// exactly. The products of digits p and q with p + q = d (0 is the leading digit) share one FP32
// accumulator: at most 8 x 64 products of at most 2^14, below 2^24, so every sum is exact. The digits
// with p + q <= 7 are used. The eight sums are put together as a 64-bit integer and rounded once to FP64 by
// integer operations; several chunks (and splits) are added in FP64.
//
// Error of an element: per k up to 2^-57 of 2^(Ei + Fj + Ec) is left out (seven products of 2^14 at weight 2^48 for
// p + q = 8; some 2^-60 of it as a rule), and its own rounding. The folded scales follow a grading of
// rows, of columns and of k, but they are the scales of a whole row and column: where an element's own terms lie
// far below them it keeps fewer digits than multiply-adds give it. For a row (1, e) of A and columns (e, 1) and
// (1, e) of B, e = 2^-50, every scale is 1 and the element 2 e keeps some 8 bits. NoDigitsScope is for callers
// whom that concerns.
//
// Relative error (2-norm) of random products with K = 30 to 130: 4e-17 to 1e-16, FP64 multiply-adds
// 1.9e-16 to 3.7e-16; graded rows, columns and opposite gradings of both alike. Local products of Kronecker sums,
// whose interfaces have rows with one nonzero: 0.9e-16 to 1.0e-16 in norm, multiply-adds 1.2e-16 to 4.8e-16; per
// element and sum of its terms 0.45 to 0.74 u on average, multiply-adds 0.5 to 1.0 u (39 u and 14 u at most). A chunk with an
// infinity or a NaN is computed with FP64 multiply-adds, so these go through; subnormal numbers have digits as
// any others.
//
// Measured (M = 322, N = 5024, K = 161): 130 us against 513 us for FP64 multiply-adds in 32 x 32 tiles, which
// ran at 80% of the FP64 pipe. The tensor pipe is 25% busy; what bounds the kernel is the integer work of
// making digits (each element once per tile that reads it) and of putting the sums together. From some
// 3e7 multiply-adds on, oz_gemm.cu makes the digits once per element: 48 us for the same product.

constexpr int kEmuK = 64;                    // K chunk
constexpr int kEmuPitch = kEmuK + 8;         // BF16 per shared-memory row: conflict-free ldmatrix

// 4 consecutive k of one row, all digits, into s[digit][row][k]
__device__ __forceinline__ void store_digits(const uint2 (&y)[4], __nv_bfloat16* s, int rows) {
  unsigned v[kEmuSlices][2];
  digits4(y, v);
#pragma unroll
  for (int p = 0; p < kEmuSlices; ++p)
    *reinterpret_cast<uint2*>(s + (size_t)p * rows * kEmuPitch) = make_uint2(v[p][0], v[p][1]);
}

__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0,
                                         unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, "
               "{%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The value of the eight exact sums D (weight 2^(8 (14 - d)) each) at scale exponents E, rounded to
// nearest. Neighbouring sums fit one 32-bit integer: |D[d]| < 2^22.9, 2^20 for d = 0.
__device__ __forceinline__ double emu_value(const float (&D)[8], int E) {
  int w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = __float2int_rn(D[2 * i]) * 256 + __float2int_rn(D[2 * i + 1]);
  const long long H = (long long)w[0] * 65536 + w[1], L = (long long)w[2] * 65536 + w[3];
  // H in units of 2^88, |H| < 2^42.1, L in units of 2^56: as T 2^sh to 62 bits or all there are, so that what an
  // element has far below the scales of its row and column stays in T
  const long long hi = H + (L >> 32);
  const int sh = max(0, 34 - __clzll(hi < 0 ? ~hi : hi));
  const unsigned long long lo = ((unsigned long long)(unsigned)L + ((1u << sh) >> 1)) >> sh;
  const long long T = (long long)(((unsigned long long)hi << (32 - sh)) + lo);
  return emu_round(T, E - 2112 + sh);   // T 2^(56 + sh) 2^(E - 2168)
}

// One operand's share of a thread: row `row` of the tile, quads of 4 consecutive k.
template <int ROWS, int NTH>
struct EmuLoader {
  static constexpr int kPer = NTH / ROWS;                 // threads per row
  static constexpr int kQuads = kEmuK / 4 / kPer;         // quads per thread
  static_assert(kPer * ROWS == NTH && kQuads >= 1, "tile and block sizes");
  double v[kQuads][4];
  int row, part;
  bool ok;
  int64_t off;
  __device__ __forceinline__ void init(int tid, int r0, int extent, const AxD& ax) {
    row = tid % ROWS;
    part = tid / ROWS;
    ok = r0 + row < extent;
    off = ok ? ax_off(ax, r0 + row) : 0;
  }
  __device__ __forceinline__ bool nonfinite() const {
    bool r = false;
#pragma unroll
    for (int q = 0; q < kQuads; ++q)
#pragma unroll
      for (int i = 0; i < 4; ++i) r |= emu_nonfinite(v[q][i]);
    return r;
  }
  __device__ __forceinline__ int k(int q) const { return (part + q * kPer) * 4; }
  // Loads the chunk of len elements at k0; true when an element is special.
  __device__ __forceinline__ bool load(const double* base, const AxD& ak, int k0, int len) {
    bool special = false;
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int kk = k(q);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[q][i] = 0.0;
      if (ok && kk < len) {
        if (ak.e0 == INT_MAX) {
          const double* p = base + off + (int64_t)(k0 + kk) * ak.s0;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (kk + i < len) v[q][i] = p[i * ak.s0];
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (kk + i < len) v[q][i] = base[off + ax_off(ak, k0 + kk + i)];
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) special |= emu_special(v[q][i]);
    }
    return special;
  }
};

// BM x BN tile, one warp per 16 x 16 of it. MINB: blocks per SM that the registers have to leave room
// for (as many as the shared memory does).
template <int BM, int BN>
struct EmuTile {
  static constexpr int kWarpsN = BN / 16;
  static constexpr int kThreads = 32 * (BM / 16) * kWarpsN;
  static constexpr size_t kSmem = (size_t)kEmuSlices * (BM + BN) * kEmuPitch * sizeof(__nv_bfloat16);
  static constexpr int kMinBlocks = (int)(220 * 1024 / kSmem);
};

template <int BM, int BN>
__global__ void __launch_bounds__(EmuTile<BM, BN>::kThreads, EmuTile<BM, BN>::kMinBlocks)
    contract_emu_kernel(KParams<double> p) {
  stream_wait();
  using Tile = EmuTile<BM, BN>;
  constexpr int NTH = Tile::kThreads;
  extern __shared__ __align__(16) unsigned char emu_sm[];
  __nv_bfloat16* As = reinterpret_cast<__nv_bfloat16*>(emu_sm);
  __nv_bfloat16* Bs = As + (size_t)kEmuSlices * BM * kEmuPitch;
  // scales of a chunk, by the parity of the chunk: kb(k), Ei, Fj, Ec
  __shared__ __align__(16) int kmax[2][kEmuK];
  __shared__ int emax_a[2][BM], fmax_b[2][BN], emax_b[2][BN];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bz = blockIdx.z;
  const int bidx = bz / p.splitk;
  const int ks = bz - bidx * p.splitk;
  const int kbeg = ks * p.kchunk;
  const int kend = min(p.K, kbeg + p.kchunk);
  const int2 tile = tile_of(p);
  const int m0 = tile.x * BM, n0 = tile.y * BN;
  if ((p.tri & kTriLowerC) && m0 + BM <= n0) return;   // tile strictly above the diagonal
  const double* A = p.A + (int64_t)bidx * p.a_bs;
  const double* B = p.B + (int64_t)bidx * p.b_bs;

  EmuLoader<BM, NTH> la;
  EmuLoader<BN, NTH> lb;
  la.init(tid, m0, p.M, p.am);
  lb.init(tid, n0, p.N, p.bn);
  const int wm = (warp / Tile::kWarpsN) * 16, wn = (warp % Tile::kWarpsN) * 16;
  const int g = lane >> 2, t2 = (lane & 3) * 2;   // fragment row and column of the accumulators
  const bool work = m0 + wm < p.M && n0 + wn < p.N;   // the warp's part of the tile is not empty

  double acc[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[j][r] = 0.0;

  int par = 0;
  for (int k0 = kbeg; k0 < kend; k0 += kEmuK, par ^= 1) {
    const int len = min(kend - k0, kEmuK);
    const int steps = (len + 15) / 16, len16 = steps * 16;   // digits are made up to len16
    const bool special = la.load(A, p.ak, k0, len) | lb.load(B, p.bk, k0, len);
    for (int i = tid; i < kEmuK; i += NTH) kmax[par][i] = kEmuZero;
    for (int i = tid; i < BM; i += NTH) emax_a[par][i] = kEmuZero;
    for (int i = tid; i < BN; i += NTH) { fmax_b[par][i] = kEmuZero; emax_b[par][i] = kEmuZero; }
    // the previous chunk's digits have been read, this chunk's scales are cleared
    const bool rare = __syncthreads_or(special ? 1 : 0) != 0;   // infinities, NaN or subnormals in the chunk
    if (rare && __syncthreads_or(la.nonfinite() | lb.nonfinite() ? 1 : 0)) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int m = m0 + wm + g + 8 * (r >> 1), n = n0 + wn + 8 * j + t2 + (r & 1);
          if (m >= p.M || n >= p.N) continue;
          const int64_t mo = ax_off(p.am, m), no = ax_off(p.bn, n);
          double s = acc[j][r];
          for (int k = k0; k < k0 + len; ++k)
            s = fma(A[mo + ax_off(p.ak, k)], B[no + ax_off(p.bk, k)], s);
          acc[j][r] = s;
        }
      continue;
    }
    const auto make_digits = [&](auto sub) {
      constexpr bool kSub = decltype(sub)::value;
      int mb = kEmuZero;
#pragma unroll
      for (int q = 0; q < lb.kQuads; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) mb = max(mb, emu_exponent<kSub>(lb.v[q][i]));
      atomicMax(&fmax_b[par][lb.row], mb);
      __syncthreads();
      const int F = fmax_b[par][lb.row];
#pragma unroll
      for (int q = 0; q < lb.kQuads; ++q) {
        if (q * lb.kPer * 4 >= len) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          constexpr bool kHalf = BN < 32;   // lanes of a half warp share k
          const int e = emu_exponent<kSub>(lb.v[q][i]);
          const int m = __reduce_max_sync(kHalf ? 0xffffu << (lane & 16) : 0xffffffffu,
                                          e == kEmuZero ? kEmuZero : e - F);
          if ((lane & (kHalf ? 15 : 31)) == 0) atomicMax(&kmax[par][lb.k(q) + i], m);
        }
      }
      __syncthreads();
      auto kb = [&](int k, int (&out)[4]) {
        const int4 m = *reinterpret_cast<const int4*>(&kmax[par][k]);
        out[0] = m.x; out[1] = m.y; out[2] = m.z; out[3] = m.w;
      };
      // a row k of B that is zero (kb = kEmuZero) takes column k of A out of the scale; a zero of A or
      // B stays more than 2^11 below any other exponent
      int ma = 2 * kEmuZero;
      mb = kEmuZero;
#pragma unroll
      for (int q = 0; q < la.kQuads; ++q) {
        if (q * la.kPer * 4 >= len) break;
        int b[4];
        kb(la.k(q), b);
#pragma unroll
        for (int i = 0; i < 4; ++i) ma = max(ma, emu_exponent<kSub>(la.v[q][i]) + b[i]);
      }
#pragma unroll
      for (int q = 0; q < lb.kQuads; ++q) {
        if (q * lb.kPer * 4 >= len) break;
        int b[4];
        kb(lb.k(q), b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int e = emu_exponent<kSub>(lb.v[q][i]);
          mb = max(mb, e == kEmuZero ? kEmuZero : e - F - b[i]);
        }
      }
      atomicMax(&emax_a[par][la.row], ma);
      atomicMax(&emax_b[par][lb.row], mb);
      __syncthreads();
      {
        const int E = emax_a[par][la.row];
#pragma unroll
        for (int q = 0; q < la.kQuads; ++q) {
          if (q * la.kPer * 4 >= len16) break;
          int b[4];
          uint2 y[4];
          kb(la.k(q), b);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            y[i] = fixed_digits<kSub>(la.v[q][i], emu_exponent<kSub>(la.v[q][i]) + b[i], E);
          store_digits(y, As + (size_t)la.row * kEmuPitch + la.k(q), BM);
        }
        const int G = emax_b[par][lb.row];
#pragma unroll
        for (int q = 0; q < lb.kQuads; ++q) {
          if (q * lb.kPer * 4 >= len16) break;
          int b[4];
          uint2 y[4];
          kb(lb.k(q), b);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int e = emu_exponent<kSub>(lb.v[q][i]);
            y[i] = fixed_digits<kSub>(lb.v[q][i], e == kEmuZero ? kEmuZero : e - F - b[i], G);
          }
          store_digits(y, Bs + (size_t)lb.row * kEmuPitch + lb.k(q), BN);
        }
      }
      __syncthreads();
    };
    if (rare) make_digits(std::true_type());
    else make_digits(std::false_type());
    if (!work) continue;
    // one n8 half of the warp's tile at a time: its eight accumulators and B digits stay in registers
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float d[kEmuSlices][4];
#pragma unroll
      for (int s = 0; s < kEmuSlices; ++s)
#pragma unroll
        for (int r = 0; r < 4; ++r) d[s][r] = 0.f;
      for (int kk = 0; kk < steps; ++kk) {
        // four slices' digits of n8 x k16 per two loads (lanes 0-15: slice s, 16-31: slice s + 1)
        unsigned b[kEmuSlices / 2][4];
        const __nv_bfloat16* bp = Bs + (size_t)((lane >> 4) * BN + wn + 8 * j + (lane & 7)) * kEmuPitch +
                                  kk * 16 + (((lane >> 3) & 1) << 3);
#pragma unroll
        for (int q = 0; q < kEmuSlices / 2; ++q) ldmatrix_x4(b[q], bp + (size_t)(2 * q) * BN * kEmuPitch);
        const __nv_bfloat16* ap = As + (size_t)(wm + (lane & 15)) * kEmuPitch + kk * 16 +
                                  ((lane >> 4) << 3);
#pragma unroll
        for (int s = 0; s < kEmuSlices; ++s) {
          unsigned a[4];
          ldmatrix_x4(a, ap + (size_t)s * BM * kEmuPitch);
#pragma unroll
          for (int q = 0; q < kEmuSlices - s; ++q)
            mma_bf16(d[s + q], a, b[q / 2][2 * (q & 1)], b[q / 2][2 * (q & 1) + 1]);
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float D[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) D[s] = d[s][r];
        const int n = wn + 8 * j + t2 + (r & 1);
        const double v =
            emu_value(D, emax_a[par][wm + g + 8 * (r >> 1)] + fmax_b[par][n] + emax_b[par][n]);
        acc[j][r] = k0 == kbeg ? v : acc[j][r] + v;
      }
    }
  }

  double* C = p.C + (int64_t)bidx * p.c_bs;
#pragma unroll
  for (int r = 0; r < 4; r += 2) {
    const int m = m0 + wm + g + 8 * (r >> 1);
    if (m >= p.M) continue;
    const int64_t cmo = ax_off(p.cm, m);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = n0 + wn + 8 * j + t2 + h;
        if (n >= p.N) continue;
        double* c = C + cmo + ax_off(p.cn, n);
        const double v = p.scale ? p.alpha * acc[j][r + h] : acc[j][r + h];
        if (p.splitk > 1) atomicAdd(c, v);
        else *c = p.keep ? fma(p.beta, *c, v) : v;
      }
  }
}
