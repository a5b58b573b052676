// st3d_f64.cuh -- the FP64 sums of the wave update in integer arithmetic.
//
// GB300 issues FP64 at 1/64 of its integer rate (two lanes a clock and SM), and
// the wave update is bound by it: of its 3 NP + 4 FP64 operations a point, 2 NP
// are the two sums of each neighbour pair,
//     t = rn(a + b),   d = rn(t - 2u)
// (rn: round to nearest even, 53 bits).  Both are formed here exactly as the
// FP64 unit forms them, bit for bit, from the operands' bits: the three
// significands are aligned as 64-bit integers (8 guard bits, so exponents may
// differ by 8), summed exactly, rounded to 53 bits where t and d are, and d is
// packed again.  The integer instructions run beside the FP64 unit's
// multiply-adds; shifts and logic (half rate) bound them, so what can be a
// multiply-add is one.
// Operands further apart, zeros, subnormals, infinities, NaN and results near
// the ends of the exponent range take the FP64 unit: the two functions say so.
// Measured (wave, 25 points, 512^3): 10437 us a step with all sums on the FP64
// unit, 6040 on uniform random fields (a fifth of the warps meets a pair that
// does not fit), 5683 on smooth ones; 7 points 256^3 474 -> 308.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define ST3D_HD __host__ __device__ __forceinline__
#else
#define ST3D_HD inline
#endif

namespace st3d {

struct Bits64 {
  uint32_t hi, lo;
};

ST3D_HD Bits64 bits_of(double x) {
#ifdef __CUDA_ARCH__
  return {(uint32_t)__double2hiint(x), (uint32_t)__double2loint(x)};
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return {(uint32_t)(b >> 32), (uint32_t)b};
#endif
}

ST3D_HD double double_of(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}

// position of the highest set bit, -1 for 0
ST3D_HD int top_bit(uint32_t x) {
#ifdef __CUDA_ARCH__
  return 31 - __clz((int)x);
#else
  return x ? 31 - __builtin_clz(x) : -1;
#endif
}

ST3D_HD uint64_t join(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// acc + (hi:lo) * p, modulo 2^64; ph is p's sign extension.  Alignment, sign
// and sum in three multiply-adds, which run on another pipe than the shifts
// and logic that bound this path.
ST3D_HD uint64_t add_scaled(uint64_t acc, uint32_t hi, uint32_t lo, uint32_t p, uint32_t ph) {
  const uint64_t w = (uint64_t)lo * p + acc;
  return join((uint32_t)(w >> 32) + hi * p + lo * ph, (uint32_t)w);
}

constexpr uint32_t kExpMask = 0x7ff00000u;  // exponents stay where they are, in bits 20..30
constexpr uint32_t kExpOne = 1u << 20;
constexpr uint32_t kExpInfinite = 2047u * kExpOne;
constexpr uint32_t kGuard = 8;  // 3 * 2^(53 + kGuard) < 2^63

// The centre's -2u as the sums take it.
struct Twice {
  uint32_t e;        // exponent bits of 2u, kExpInfinite and above where 2u is not finite
  uint32_t hi, lo;   // significand with its leading bit
  uint32_t neg;      // all ones where -2u is negative
};

ST3D_HD Twice twice_of(double u) {
  const Bits64 b = bits_of(u);
  Twice t;
  const uint32_t e = b.hi & kExpMask;
  t.e = e ? e + kExpOne : 0u;  // zero and subnormal u fail the range check
  t.hi = (b.hi & 0xfffffu) | 0x100000u;
  t.lo = b.lo;
  t.neg = ~(uint32_t)((int32_t)b.hi >> 31);
  return t;
}

// Whether the integer path serves this pair; the exponents' top in *E.
ST3D_HD bool pair_fits(const Bits64& a, const Bits64& b, const Twice& u, uint32_t* E) {
  const uint32_t ea = a.hi & kExpMask, eb = b.hi & kExpMask;
  const uint32_t top = ea > eb ? (ea > u.e ? ea : u.e) : (eb > u.e ? eb : u.e);
  const uint32_t low = ea < eb ? (ea < u.e ? ea : u.e) : (eb < u.e ? eb : u.e);
  *E = top;
  // 64 <= low and top <= 2044 hold together where low lies in 64 .. 2036
  return top - low <= kGuard * kExpOne && low - 64u * kExpOne <= 1972u * kExpOne;
}

// rn(rn(a + b) - 2u) for operands that fit, in *d; false where the difference
// cancels below 2^32 of its 61-bit scale and the FP64 unit has to form it.
ST3D_HD bool pair_diff_bits(const Bits64& a, const Bits64& b, const Twice& u, uint32_t E, double* out) {
  const uint32_t base = E - kGuard * kExpOne;
  const uint32_t sa = (uint32_t)((int32_t)a.hi >> 31), sb = (uint32_t)((int32_t)b.hi >> 31);
  const uint32_t pa = (sa | 1u) << (((a.hi & kExpMask) - base) >> 20);
  const uint32_t pb = (sb | 1u) << (((b.hi & kExpMask) - base) >> 20);
  const uint32_t pu = (u.neg | 1u) << ((u.e - base) >> 20);
  uint64_t t = add_scaled(0, (a.hi & 0xfffffu) | 0x100000u, a.lo, pa, sa);
  t = add_scaled(t, (b.hi & 0xfffffu) | 0x100000u, b.lo, pb, sb);
  // t to 53 bits: k low bits go, to nearest, ties to even (k <= 9; on two's
  // complement the same as on the magnitude)
  {
    const uint32_t th = (uint32_t)(t >> 32), tl = (uint32_t)t;
    const int pos = top_bit(th ^ (uint32_t)((int32_t)th >> 31)) - 20;
    const int k = pos > 0 ? pos : 0;
    const uint32_t r = (1u << k) - 1u;
    t += (r >> 1) + ((tl >> k) & r & 1u);
    t = join((uint32_t)(t >> 32), (uint32_t)t & ~r);
  }
  const uint64_t d = add_scaled(t, u.hi, u.lo, pu, u.neg);
  // pack: magnitude, leading bit to bit 62, round at bit 10
  const uint32_t dh = (uint32_t)(d >> 32), sd = (uint32_t)((int32_t)dh >> 31);
  const uint64_t m = add_scaled(0, dh, (uint32_t)d, sd | 1u, sd);
  const uint32_t mh = (uint32_t)(m >> 32);
  const int z = 30 - top_bit(mh);
  uint64_t n = m * (uint64_t)(1u << (z & 31));
  n += 0x1ffu + (((uint32_t)n >> 10) & 1u);
  const uint32_t hi = (uint32_t)(n >> 42) + E + kExpOne - (uint32_t)z * kExpOne;
  *out = double_of(hi + (sd << 31), (uint32_t)(n >> 10));
  return mh != 0;
}

}  // namespace st3d
