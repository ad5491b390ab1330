// The digits of the error-free splitting of FP64 operands (see contract_emu.cuh) and the rounding of their
// product's sums, shared by the two kernels that multiply them.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace ttgb {

constexpr int kEmuSlices = 8;
constexpr int kEmuZero = -20000;             // exponent of a zero: far below any other

// Exponent field of x, kEmuZero for a zero. With SUB, which the digit kernels take where they have found a subnormal
// number (some 10% slower: zeros take the same branches), continued below 1 for these, to -51.
template <bool SUB>
__device__ __forceinline__ int emu_exponent(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  if (!SUB) return e == 0 ? kEmuZero : e;
  if (e != 0) return e;
  const long long m = __double_as_longlong(x) & 0xfffffffffffffll;
  return m == 0 ? kEmuZero : 12 - __clzll(m);
}

// whether x is an infinity, a NaN or subnormal
__device__ __forceinline__ bool emu_special(double x) {
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  return h >= 0x7ff00000u || (h < 0x00100000u && (h | (unsigned)__double2loint(x)) != 0u);
}

// whether x is an infinity or a NaN
__device__ __forceinline__ bool emu_nonfinite(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) == 0x7ff00000u;
}

// x in fixed point, 2^(E - e) below the leading position of a 62-bit integer, plus the 0x80 of every
// byte that makes the bytes of the sum the balanced digits + 128
template <bool SUB>
__device__ __forceinline__ uint2 fixed_digits(double x, int e, int E) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  unsigned hi = ((h & 0xfffffu) | 0x100000u) << 9 | l >> 23, lo = l << 9;   // 53 bits at 2^61
  if (SUB && (h & 0x7ff00000u) == 0u) {   // subnormal: its leading bit to 2^61
    const unsigned long long m = (unsigned long long)(h & 0xfffffu) << 32 | l;
    const unsigned long long y = m << ((__clzll((long long)m) - 2) & 63);
    hi = (unsigned)(y >> 32);
    lo = (unsigned)y;
  }
  int sh = E - e;
  if (sh >= 32) { lo = hi; hi = 0u; sh -= 32; }
  sh = min(sh, 32);   // a zero, whose exponent is far below E, leaves no bits
  lo = __funnelshift_rc(lo, hi, sh);
  hi = sh < 32 ? hi >> sh : 0u;
  const unsigned neg = (unsigned)((int)h >> 31);
  const unsigned long long y = ((unsigned long long)(hi ^ neg) << 32 | (lo ^ neg)) +
                               (0x8080808080808080ull - (unsigned long long)(long long)(int)neg);
  return make_uint2((unsigned)y, (unsigned)(y >> 32));
}

// The digits of 4 consecutive k as BF16 pairs, v[digit][pair]. With a byte b the digit is b - 128, the
// difference of the BF16 values 128 + (b mod 128) and 256 - 128 (b div 128), whose bits are b's own.
__device__ __forceinline__ void digits4(const uint2 (&y)[4], unsigned (&v)[kEmuSlices][2]) {
#pragma unroll
  for (int p = 0; p < kEmuSlices; ++p) {
    const int byte = 7 - p;
    const unsigned sel = (unsigned)(byte & 3) | (unsigned)(4 + (byte & 3)) << 8;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const unsigned w = byte >= 4 ? __byte_perm(y[2 * i].y, y[2 * i + 1].y, sel | sel << 4)
                                   : __byte_perm(y[2 * i].x, y[2 * i + 1].x, sel | sel << 4);
      const unsigned a = (w & 0x007f007fu) | 0x43004300u, b = (w & 0x00800080u) ^ 0x43804380u;
      asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(v[p][i]) : "r"(a), "r"(b));
    }
  }
}

// T 2^E rounded to nearest even (E below -17000: of a row or column of zeros, whose digits mean nothing).
__device__ __forceinline__ double emu_round(long long T, int E) {
  if (T == 0 || E < -17000) return 0.0;
  unsigned long long m = (unsigned long long)(T < 0 ? -T : T);
  const int lz = __clzll((long long)m);
  int ef = 63 - lz + E + 1023;
  m <<= lz;
  const unsigned long long r = m + 0x3ffull + ((m >> 11) & 1ull);   // to 53 bits, ties to even
  ef += r < m ? 1 : 0;                                              // carried out of the top bit
  const unsigned long long frac = r < m ? 0ull : (r >> 11) & 0xfffffffffffffull;
  const unsigned long long sign = T < 0 ? 1ull << 63 : 0ull;
  if (ef >= 1 && ef <= 2046)
    return __longlong_as_double((long long)(sign | ((unsigned long long)ef << 52) | frac));
  const double v = scalbn(__longlong_as_double((long long)((1023ull << 52) | frac)), ef - 1023);
  return T < 0 ? -v : v;   // subnormal or infinite
}

}  // namespace ttgb
