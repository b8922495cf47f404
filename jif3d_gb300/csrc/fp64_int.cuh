// fp64_int.cuh -- correctly rounded FP64 square roots, quotients and sums on the
// integer pipes, bit for bit what the FP64 instructions round to.
//
// The GB300 starts an FP64 instruction every 16 cycles per SM.  A square root or
// a quotient takes five to ten of them and 50 integer instructions here; a sum
// takes 65 integer instructions, about 20 cycles of the SM's integer pipe, so
// moving a part of the sums of a kernel bound by FP64 uses both pipes.  Roots and
// quotients go from an FP32 estimate and one Newton step of 32 bits to a result
// within one unit, and an exact remainder decides the last bit.
#pragma once
#include "node_fixed.cuh"

namespace j3g {

constexpr uint64_t kIntFrac = 0xfffffffffffffull, kIntOne = 0x10000000000000ull;

J3G_FX int int_clz64(uint64_t v) {
  return fx_hi(v) ? fx_clz(fx_hi(v)) : 32 + fx_clz(fx_lo(v));
}

// v 2^-scale exactly, |v| up to 2^53.
J3G_FX double int_to_double(int64_t v, int scale) {
  if (v == 0) return 0.0;
  const uint32_t neg = (uint32_t)(v >> 63);
  const uint64_t a = (uint64_t)(v < 0 ? -v : v);
  const int n = int_clz64(a);
  const uint64_t m = (a << n) >> 11;
  return fx_double(fx_pair(fx_hi(m) + ((uint32_t)(1085 - scale - n) << 20) | neg << 31, fx_lo(m)));
}

// The operands that int_add leaves to the FP64 instruction.  Out of line: a
// predicated FP64 instruction takes its slot of the pipe in every lane's absence.
#ifdef __CUDACC__
static __device__ __noinline__ double int_add_rare(double a, double b) { return __dadd_rn(a, b); }
J3G_FX uint64_t int_shl(uint64_t v, int n) {  // zero for n of 64 and more
  uint64_t r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
  return r;
}
#else
J3G_FX double int_add_rare(double a, double b) { return a + b; }
J3G_FX uint64_t int_shl(uint64_t v, int n) { return (uint32_t)n > 63u ? 0 : v << n; }
#endif

J3G_FX double int_neg(double a) { return fx_double(fx_bits(a) ^ 1ull << 63); }

// a + b
J3G_FX double int_add(double a, double b) {
  const uint64_t A = fx_bits(a), B = fx_bits(b), kAbs = 0x7fffffffffffffffull;
  const bool swap = (A & kAbs) < (B & kAbs);
  const uint64_t x = swap ? B : A, y = swap ? A : B;
  const uint32_t xh = fx_hi(x), yh = fx_hi(y);
  const uint32_t ex = xh >> 20 & 0x7ffu, ey = yh >> 20 & 0x7ffu;
  // ten bits below the larger operand's last one, the rest of the smaller as a
  // sticky bit: it is only ever set where at most one bit cancels
  const uint64_t my = ((y & kIntFrac) | kIntOne) << 10;
  const int d = (int)(ex - ey);
  uint64_t s = fx_shr(my, d);
  s |= int_shl(s, d) != my;
  const uint64_t neg = (uint64_t)(int64_t)((int32_t)(xh ^ yh) >> 31);
  const uint64_t m = (((x & kIntFrac) | kIntOne) << 10) + ((s ^ neg) - neg);
  // zeros, subnormals, ends of the range, and 30 bits and more cancelled
  if (ey == 0 || ex - 64u >= 0x7feu - 64u || fx_hi(m) == 0) return int_add_rare(a, b);
  const int n = fx_clz(fx_hi(m));
  const uint64_t t = m << n;
  uint64_t r = t >> 11;
  r += (fx_lo(t) & 0x7ffu) + (fx_lo(r) & 1u) > 0x400u;  // a carry out raises the exponent
  return fx_double(fx_pair(fx_hi(r) + (ex - (uint32_t)n << 20) | (xh & 0x80000000u), fx_lo(r)));
}

// sqrt of a positive normal x: with X = x 4^-h in [1, 4) the 53-bit integer z
// nearest to sqrt(X) 2^52.
J3G_FX double int_sqrt(double x) {
  const uint64_t b = fx_bits(x);
  const uint32_t e = fx_hi(b) >> 20;
  const int odd = (int)(~e & 1u);  // an odd power of two
  const uint64_t m = (b & kIntFrac) | kIntOne, s = m << (9 + odd);  // X 2^61
  const float inv = fx_rsqrt(fx_float((uint32_t)(127 + odd) << 23 | (uint32_t)(b >> 29 & 0x7fffffu)));
  // 1 / sqrt(X) to 2^-20, a little low, then to 2^-29, scale 2^30
  const int32_t y0 = (int32_t)fx_f2u(inv * 1073741824.0f) - 1024;
  const uint32_t yy = (uint32_t)((uint64_t)((int64_t)y0 * y0) >> 28);
  const int64_t d = (int64_t)((1ull << 61) - fx_mul32(s, yy));
  const uint32_t y = (uint32_t)(y0 + (int32_t)((int64_t)y0 * (int32_t)(d >> 13) >> 49));
  // sqrt(X) 2^59 and its correction by half of 1 - X y^2
  const uint64_t p = fx_mul32(s, y);
  const int32_t t = (int32_t)((1ull << 57) - fx_mul32(p, y));
  const uint64_t R = p + (uint64_t)((int64_t)(int32_t)(p >> 30) * t >> 28);
  uint64_t z = (R + 64) >> 7;
  // X 2^104 - z^2 beyond -z and z: the root is beyond the half
  const int64_t rem = (int64_t)((m << (52 + odd)) - z * z);
  z += rem > (int64_t)z;
  z -= rem <= -(int64_t)z;
  const uint32_t h = (e - 1023u - (uint32_t)odd) >> 1;  // wraps below zero: 11 bits are kept
  return fx_double(z + ((uint64_t)((h + 1022u) & 0x7ffu) << 52));
}

// num / den for mantissas num, den in [2^52, 2^53): z 2^-52 (down = 0) or
// z 2^-53 (down = 1), z in [2^52, 2^53], rounded to nearest.
J3G_FX uint64_t int_quotient(uint64_t num, uint64_t den, int &down) {
  down = num < den;
  // 2^84 / den to 2^-30
  const uint32_t dh = (uint32_t)(den >> 21);
  const float inv = fx_rcp(fx_float(127u << 23 | (uint32_t)(den >> 29 & 0x7fffffu)));
  const uint32_t y0 = fx_f2u(inv * 2147483648.0f) * 2 - 1024;  // 2^63 / dh, a little low
  const int64_t d = (int64_t)((1ull << 63) - (uint64_t)dh * y0);
  const uint32_t y = y0 + (uint32_t)((int64_t)(int32_t)(y0 >> 1) * (int32_t)(d >> 12) >> 50);
  // num 2^53 / den in two digits of 31 and 22 bits
  const uint32_t q1 = fx_mulhi((uint32_t)(num >> 21), y);
  const int64_t r1 = (int64_t)((num << 31) - (uint64_t)q1 * den);
  const int64_t q2 = (int64_t)(int32_t)(r1 >> 25) * (int32_t)(y >> 1) >> 36;
  const uint64_t q = ((uint64_t)q1 << 22) + (uint64_t)q2;
  uint64_t z = down ? q : (q + 1) >> 1;
  const int64_t rem = (int64_t)((num << (52 + down)) - z * den);  // never +-den / 2
  z += 2 * rem > (int64_t)den;
  z -= 2 * rem < -(int64_t)den;
  return z;
}

}  // namespace j3g
