// node_fixed.cuh -- the node terms of prism_math.cuh (node_terms) on the
// integer and FP32 pipes, for kernels that evaluate very many of them.
//
// The GB300 retires 2 FP64 operations per clock and SM against 64 integer
// multiply-adds and 128 FP32 operations, so the FP64 form of a joint node
// (about 140 FP64 instructions) is bound by that pipe alone.  Here every
// quantity with more than 24 bits is a 64-bit integer with a power-of-two
// scale; FP32 only gives starting values (relative error about 2^-19) and
// table indices, and the few FP64 operations left are the products with the
// model or the weights.  Truncation keeps each logarithm and angle within
// about 2^-55 and the square root within about 2^-57 relative, below the
// rounding of the FP64 form; the results are rounded to FP64 once.
//
//   offsets   |d| = m 2^e, m a 64-bit integer with its top bit set, and d^2
//   r         Newton's iteration for 1/sqrt(s) from an FP32 start, then one
//             correction of r = s / sqrt(s)
//   log       m G_j - 1 = z, |z| < 2^-10, G_j a table of short reciprocals;
//             log = k log 2 - log G_j + z - z^2/2 + z^3 (1/3 - z/4 + z^2/5)
//   angles    with a >= b >= c the sorted |dx|, |dy|, |dz| the three angles
//             atan(bc / ar), atan(ac / br), atan(ab / cr) add up to pi/2 (the
//             corner's solid angle), so the two smaller ones, both <= pi/4,
//             are evaluated and the third is their complement.
//             atan(N/D) = atan(j/1024) + atan(d), d = (N - jD/1024) / (D + jN/1024),
//             |d| <= 2^-11, by two digits of long division with a Newton
//             reciprocal, atan d = d - d^3/3 + d^5/5; small angles keep a scale of
//             their own, so that each has at least 53 bits.  (With 512 steps at
//             scale 2^61 angles below 2^-9 were up to 13 units off in the last
//             place, four on average, the cubic term's 32 bits being worth 2^-51 of
//             them; 1024 steps at 2^63 and the term's shift after its product leave
//             less than FP64's own error, for 4 KB more of tables.)
//
// Mantissas have their top bit at 2^62, so that the cross products of a 64 x 64
// bit multiplication add up without a carry (three multiply-adds).
//
// Offsets beyond 2^+-40 and dz and another offset both exactly zero are left to
// node_terms (fx_node returns false).
// The same code compiles for the host, where its accuracy is tested.
#pragma once
#include <cstdint>
#include <cstring>

#include "node_tables.h"

#ifdef __CUDACC__
#define J3G_FX __device__ __forceinline__
#define J3G_FX_MEMBER __device__ __forceinline__
#else
#include <cmath>
#define J3G_FX static inline
#define J3G_FX_MEMBER inline
#endif

namespace j3g {

#ifdef __CUDACC__
J3G_FX uint32_t fx_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
J3G_FX int32_t fx_mulhi_s(int32_t a, int32_t b) { return __mulhi(a, b); }
J3G_FX int fx_clz(uint32_t a) { return __clz((int)a); }
J3G_FX float fx_rsqrt(float a) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
J3G_FX float fx_rcp(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
J3G_FX uint32_t fx_f2u(float a) {
  uint32_t r;
  asm("cvt.rzi.ftz.u32.f32 %0, %1;" : "=r"(r) : "f"(a));
  return r;
}
// v >> n, zero for n of 64 and more (n unsigned)
J3G_FX uint64_t fx_shr(uint64_t v, int n) {
  uint64_t r;
  asm("shr.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
  return r;
}
// (hi:lo) >> n, low word, n below 32
J3G_FX uint32_t fx_funnel(uint32_t lo, uint32_t hi, int n) { return __funnelshift_r(lo, hi, n); }
J3G_FX uint32_t fx_bits(float a) { return __float_as_uint(a); }
J3G_FX float fx_float(uint32_t a) { return __uint_as_float(a); }
// The bits of a double and back, opaque: where the compiler sees the double
// behind a mask or a flip of the sign bit it makes them an FP64 absolute value or
// negation, each of which takes a slot of that pipe.
J3G_FX uint64_t fx_bits(double a) {
  uint64_t r;
  asm("mov.b64 %0, %1;" : "=l"(r) : "d"(a));
  return r;
}
J3G_FX double fx_double(uint64_t a) {
  double r;
  asm("mov.b64 %0, %1;" : "=d"(r) : "l"(a));
  return r;
}
J3G_FX float fx_fmaf(float a, float b, float c) { return __fmaf_rn(a, b, c); }
#else
J3G_FX uint32_t fx_mulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
J3G_FX int32_t fx_mulhi_s(int32_t a, int32_t b) { return (int32_t)((int64_t)a * b >> 32); }
J3G_FX int fx_clz(uint32_t a) { return a ? __builtin_clz(a) : 32; }
J3G_FX float fx_rsqrt(float a) { return 1.0f / sqrtf(a); }
J3G_FX float fx_rcp(float a) { return 1.0f / a; }
J3G_FX uint32_t fx_f2u(float a) { return a > 0.0f ? (uint32_t)a : 0u; }
J3G_FX uint64_t fx_shr(uint64_t v, int n) { return (uint32_t)n > 63u ? 0 : v >> n; }
J3G_FX uint32_t fx_funnel(uint32_t lo, uint32_t hi, int n) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (n & 31));
}
J3G_FX uint32_t fx_bits(float a) { uint32_t u; memcpy(&u, &a, 4); return u; }
J3G_FX float fx_float(uint32_t a) { float f; memcpy(&f, &a, 4); return f; }
J3G_FX uint64_t fx_bits(double a) { uint64_t u; memcpy(&u, &a, 8); return u; }
J3G_FX double fx_double(uint64_t a) { double d; memcpy(&d, &a, 8); return d; }
J3G_FX float fx_fmaf(float a, float b, float c) { return std::fma(a, b, c); }
#endif

J3G_FX uint32_t fx_hi(uint64_t v) { return (uint32_t)(v >> 32); }
J3G_FX uint32_t fx_lo(uint64_t v) { return (uint32_t)v; }
J3G_FX uint64_t fx_pair(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
J3G_FX int fx_max(int a, int b) { return a > b ? a : b; }
J3G_FX int fx_min(int a, int b) { return a < b ? a : b; }
// floor(x y / 2^64) up to two units for x, y below 2^63 (without the product
// of the low words)
J3G_FX uint64_t fx_mul64(uint64_t x, uint64_t y) {
  const uint64_t t = (uint64_t)fx_lo(x) * fx_hi(y) + (uint64_t)fx_hi(x) * fx_lo(y);
  return (uint64_t)fx_hi(x) * fx_hi(y) + fx_hi(t);
}
// floor(x y / 2^32) for a 32-bit y, up to one unit (x y below 2^96)
J3G_FX uint64_t fx_mul32(uint64_t x, uint32_t y) {
  return (uint64_t)fx_hi(x) * y + fx_mulhi(fx_lo(x), y);
}

// The tables as the kernels keep them in shared memory: -log G_j and G_j side
// by side (one 16-byte lookup), k log 2 for k = -kLogBias .. kLogBias - 1.
struct FxTables {
  struct alignas(16) Log {
    uint64_t l;
    uint32_t g, pad;
  };
  Log log[nodetab::kLogN];
  uint64_t atan[nodetab::kAtanN + 1];
  uint64_t klog[2 * nodetab::kLogBias];
  J3G_FX_MEMBER void set(int thread, int threads) {
    for (int i = thread; i < nodetab::kLogN; i += threads) {
      log[i].l = nodetab::kLogL[i];
      log[i].g = nodetab::kLogG[i];
    }
    for (int i = thread; i <= nodetab::kAtanN; i += threads) atan[i] = nodetab::kAtan[i];
    for (int i = thread; i < 2 * nodetab::kLogBias; i += threads)
      klog[i] = (uint64_t)(i - nodetab::kLogBias) * nodetab::kLn2 +
                (uint64_t)((int64_t)(i - nodetab::kLogBias) * (int64_t)nodetab::kLn2Low >> 32);
  }
};

// log(DBL_EPSILON) = -52 log 2, scale 2^57
constexpr int64_t kFxLogEps =
    -52 * (int64_t)nodetab::kLn2 - (int64_t)((52ull * nodetab::kLn2Low) >> 32);
constexpr int kFxZeroExp = -4096;  // exponent of a zero offset: shifted out of every sum

// One offset |d| = m 2^e (m = 0 or in [2^62, 2^63)), d^2 = q 2^qe with q in
// [2^60, 2^62) and qe even, and FP32 values |d|, d^2 and 2^62 / m.
struct FxAxis {
  uint64_t m, q;
  int e, qe;
  float f, f2, im;
  uint32_t neg;  // 1 for a negative offset
  uint32_t bad;  // 1: outside 2^+-40 (and not zero), infinite or NaN
};

J3G_FX FxAxis fx_axis(double d) {
  FxAxis a;
  const uint64_t b = fx_bits(d);
  const uint32_t eb = fx_hi(b) >> 20 & 0x7ffu;
  a.neg = fx_hi(b) >> 31;
  const bool zero = (b << 1) == 0;
  a.bad = !zero && (eb < 1023u - 40u || eb > 1023u + 40u);
  a.m = zero ? 0 : ((b << 10) & 0x3fffffffffffffffull) | 0x4000000000000000ull;
  a.e = zero ? kFxZeroExp : (int)eb - 1023 - 62;
  // the leading 24 bits as a float: 2^(eb - 1023) [1, 2)
  const uint32_t frac = fx_hi(a.m) >> 7 & 0x7fffffu;
  a.f = zero || a.bad ? 0.0f : fx_float((eb - 1023u + 127u) << 23 | frac);
  a.f2 = a.f * a.f;
  a.im = fx_rcp(fx_float(127u << 23 | frac));
  a.q = fx_mul64(a.m, a.m);
  a.qe = zero ? kFxZeroExp : 2 * a.e + 64;
  return a;
}

// q 2^qe of two sums of squares, aligned at the larger exponent.
J3G_FX void fx_add_sq(uint64_t qa, int ea, uint64_t qb, int eb, uint64_t &s, int &es) {
  es = fx_max(ea, eb);
  s = fx_shr(qa, es - ea) + fx_shr(qb, es - eb);
}

// The offsets of one node column (fixed x and y, all z) from one station:
// the larger (hi) and the smaller (lo) of |dx| and |dy|, and dx^2 + dy^2.
struct FxColumn {
  uint64_t mx, my, mhi, mlo, p;
  int64_t logp;  // log(dx^2 + dy^2), scale 2^57 (where Uxy is wanted)
  int ex, ey, ehi, elo, pe;
  float fhi, flo, imhi, imlo, ifhi, pf;
  uint32_t negx, negy, neghi, neglo;
  bool yhi;    // |dy| > |dx|
  bool axial;  // dx = dy = 0: the station is above or below the column
  bool bad;
};

// r = R 2^e with R in [2^58, 2^59.8); 2^88 / R, r and 1/r as floats.
struct FxRadius {
  uint64_t R;
  int e;
  float ys, f, inv;
};

J3G_FX FxRadius fx_radius(uint64_t p, int pe, float pf, const FxAxis &z) {
  uint64_t s;
  int es;
  fx_add_sq(p, pe, z.q, z.qe, s, es);  // [2^60, 2^63.6), es even
  FxRadius r;
  const float sf = pf + z.f2;
  r.inv = fx_rsqrt(sf);
  r.f = sf * r.inv;
  const int h = es >> 1;
  r.ys = r.inv * fx_float((uint32_t)(127 + 60 + h) << 23);  // 2^60 / sqrt(s)
  // a little low, so that its square stays within 32 bits: (2^28.2, 2^30)
  const int32_t y0 = (int32_t)fx_f2u(r.ys) - 1024;
  const uint32_t yy = (uint32_t)((uint64_t)((int64_t)y0 * y0) >> 28);  // 2^92 / s
  const int64_t d = (int64_t)((1ull << 60) - fx_mul32(s, yy));
  const uint32_t y = (uint32_t)(y0 + (int32_t)((int64_t)y0 * (int32_t)(d >> 13) >> 48));
  const uint64_t p1 = fx_mul32(s, y);  // sqrt(s) 2^28
  const int32_t t = (int32_t)((1ull << 56) - fx_mul32(p1, y));
  r.R = p1 + (uint64_t)((int64_t)(int32_t)(p1 >> 29) * t >> 28);
  r.e = h - 28;
  return r;
}

// log(u 2^e) at scale 2^57 for u in [2^32, 2^64).
J3G_FX int64_t fx_log(uint64_t u, int e, const FxTables &T) {
  const int n = fx_clz(fx_hi(u));
  const uint64_t m = u << n;
  const FxTables::Log g = T.log[fx_hi(m) >> 22 & 511u];
  const int64_t z = (int64_t)(fx_mul32(m, g.g) << 9);  // z 2^72 (the leading one shifts out)
  const int32_t zh = (int32_t)(z >> 32);               // z 2^40
  const int32_t zl = (int32_t)(fx_lo(z) >> 1);
  const int64_t zz = (int64_t)zh * zh + (fx_mulhi_s(zh * 2, zl) * 2);  // z^2 2^80
  const int32_t zc = zh >> 8;                                         // z 2^32
  const int32_t c = 1431655765 - fx_mulhi_s(zc, 1073741824 - fx_mulhi_s(zc, 858993459));
  const int32_t z3 = (int32_t)((int64_t)(int32_t)(zz >> 32) * zh >> 27);  // z^3 2^61
  const int64_t t = (z >> 15) - (zz >> 24) + (fx_mulhi_s(z3, c) >> 4);
  return (int64_t)(T.klog[(e + 63 - n + nodetab::kLogBias) & (2 * nodetab::kLogBias - 1)] + g.l) +
         t;
}

template <int MASK>
J3G_FX FxColumn fx_column(const FxAxis &x, const FxAxis &y, const FxTables &T) {
  FxColumn c;
  c.yhi = y.f > x.f;  // equal leading bits: either is the larger
  c.mx = x.m;
  c.ex = x.e;
  c.my = y.m;
  c.ey = y.e;
  c.mhi = c.yhi ? y.m : x.m;
  c.ehi = c.yhi ? y.e : x.e;
  c.fhi = c.yhi ? y.f : x.f;
  c.imhi = c.yhi ? y.im : x.im;
  c.mlo = c.yhi ? x.m : y.m;
  c.elo = c.yhi ? x.e : y.e;
  c.flo = c.yhi ? x.f : y.f;
  c.imlo = c.yhi ? x.im : y.im;
  fx_add_sq(x.q, x.qe, y.q, y.qe, c.p, c.pe);  // [2^60, 2^63)
  c.pf = x.f2 + y.f2;
  c.negx = x.neg;
  c.negy = y.neg;
  c.neghi = c.yhi ? y.neg : x.neg;
  c.neglo = c.yhi ? x.neg : y.neg;
  c.axial = c.mhi == 0;
  c.ifhi = c.axial ? 0.0f : fx_rcp(c.fhi);
  // zeros come as +0 (a difference of equal coordinates)
  c.bad = (x.bad | y.bad) != 0 || (c.axial && (x.neg | y.neg));
  c.logp = MASK & 16 ? fx_log(c.p, c.pe, T) : 0;
  return c;
}

// log(max(d + r, eps)) of one offset d = +-m 2^e where the other two are
// mb 2^eb and mc 2^ec.  A negative offset that takes off more than ten bits
// of r goes through d + r = (b^2 + c^2) / (r - d).
J3G_FX int64_t fx_log_sum(uint64_t m, int e, uint32_t neg, uint64_t mb, int eb, uint64_t mc,
                          int ec, const FxRadius &r, const FxTables &T) {
  const uint64_t a = fx_shr(m, r.e - e);
  const uint64_t u = neg ? r.R - a : r.R + a;
  // (signed: u may come out a few units below zero)
  if ((int32_t)fx_hi(u) >= (int32_t)(fx_hi(r.R) >> 10)) return fx_log(u, r.e, T);
  uint64_t s;
  int es;
  fx_add_sq(fx_mul64(mb, mb), 2 * eb + 64, fx_mul64(mc, mc), 2 * ec + 64, s, es);
  const int64_t l = fx_log(s, es, T) - fx_log(r.R + a, r.e, T);
  return l < kFxLogEps ? kFxLogEps : l;
}

// v 2^-scale (v below 2^63, high word not zero) rounded to a double of sign neg.
J3G_FX double fx_to_double(uint64_t v, int scale, uint32_t neg) {
  const int n = fx_clz(fx_hi(v));
  const uint64_t b = ((v << (n - 1)) + 0x200u) >> 10;  // [2^52, 2^53]
  const uint32_t hi = fx_hi(b) + ((uint32_t)(1085 - scale - n) << 20);
  return fx_double(fx_pair(hi | neg << 31, fx_lo(b)));
}

// v 2^-scale as a double by the conversion instruction (one FP64 operation, a
// dozen integer ones less than fx_to_double; the kernels leave the FP64 pipe
// room for a few).  The last bit is set, so that v is not zero.
J3G_FX double fx_convert(int64_t v, int scale, uint32_t neg) {
  const uint64_t b = fx_bits((double)(v | 1));
  return fx_double(fx_pair((fx_hi(b) - ((uint32_t)scale << 20)) ^ neg << 31, fx_lo(b)));
}

// An angle: v 2^-scale, and the same at scale 2^61.
struct FxAngle {
  uint64_t v, v61;
  int scale;
};

// atan(N / D) <= pi/4 for N = n1 2^-s, s >= 0, n1 in [2^60, 2^64) or 0, D in
// [2^58, 2^61); t = N / D and idy = 2^88 / D as floats.
J3G_FX FxAngle fx_atan(uint64_t n1, int s, uint64_t D, float t, float idy, const FxTables &T) {
  // ratios below 2^-12 (j = 0) are scaled by 2^x into [2^-12, 2^-11), so that
  // small angles keep their leading bits
  const int x = fx_max(115 - (int)(fx_bits(t) >> 23), 0);
  s -= x;  // below 32
  // N with 32 bits below its unit: (nh:nl:nx), and 2^10 N modulo 2^64
  const uint32_t nh = fx_hi(n1) >> (s & 31), nl = fx_funnel(fx_lo(n1), fx_hi(n1), s);
  const uint32_t nx = fx_funnel(0, fx_lo(n1), s);
  const uint64_t n10 = fx_pair(fx_funnel(nl, nh, 22), fx_funnel(nx, nl, 22));
  const uint64_t n8 = fx_pair(nh >> 8, fx_funnel(nl, nh, 8));
  const float jf = fx_fmaf(t, 1024.0f, 8388608.0f);  // the nearest integer in its low bits
  uint32_t j = fx_bits(jf) - 0x4b000000u;
  j = j < 1024u ? j : 1024u;
  const int64_t num = (int64_t)(n10 - (uint64_t)j * D);            // |num| <= D / 2
  const uint64_t den = D + ((uint64_t)j * n8 >> 2);                // below 2^62
  const float ct = (jf - 8388608.0f) * (1.0f / 1024.0f);
  const int32_t y0 = (int32_t)fx_f2u(idy * fx_rcp(fx_fmaf(ct, t, 1.0f)));  // 2^88 / den
  const int64_t d = (int64_t)((1ull << 58) - (uint64_t)(uint32_t)(den >> 30) * (uint32_t)y0);
  const int32_t y = y0 + (int32_t)((int64_t)y0 * (int32_t)(d >> 10) >> 48);
  const int32_t q0 = fx_mulhi_s((int32_t)(num >> 30), y);  // 2^26 num / den
  const int64_t rem = (int64_t)(((uint64_t)num << 26) - (uint64_t)(int64_t)q0 * den);
  // 2^56 rem / den, then 2^61 num / den = 2^71 d (scaled by 2^x)
  const int64_t q1 =
      (int64_t)(int32_t)(rem >> 32) * y + fx_mulhi(fx_lo((uint64_t)rem), (uint32_t)y);
  const int64_t q = (int64_t)((uint64_t)(int64_t)q0 << 35) + (q1 >> 21);
  // d - d^3/3 + d^5/5 with d = 2^-10 dh 2^-31
  const int32_t dh = (int32_t)((q + (1 << 29)) >> 30);  // to nearest: its error counts thrice
  const uint32_t d2 = (uint32_t)((uint64_t)((int64_t)dh * dh) >> 29);  // 2^33 (2^10 d)^2
  const uint32_t c5 = fx_mulhi(d2, 858993459u) >> fx_min(20 + 2 * x, 31);
  const uint32_t c = fx_mulhi(d2, 2863311531u - c5);  // 2^54 d^2 (1/3 - d^2/5)
  const int64_t cube = (int64_t)dh * (int32_t)c;      // 2^95 (d^3/3 - d^5/5), 2^x thrice
  const int64_t small = q - (cube >> fx_min(24 + 2 * x, 63));  // scale 2^71 (2^x)
  FxAngle r;
  const uint64_t v63 =
      T.atan[j] + (uint64_t)(x ? (int64_t)fx_shr((uint64_t)small, 8 + x) : small >> 8);
  r.v61 = v63 >> 2;
  r.v = j ? v63 : (uint64_t)small;
  r.scale = j ? 63 : 71 + x;
  return r;
}

// atan2 from the angle of the magnitudes: `own` the sign of the abscissa's
// offset, neg the sign of the ordinate.  Zero angles come from zero offsets.
J3G_FX double fx_quadrant(uint64_t v, int scale, uint64_t v61, uint32_t own, uint32_t neg) {
  const uint64_t w = own ? nodetab::kPiS61 - v61 : v;
  const double d = fx_to_double(w, own ? 61 : scale, neg);
  return fx_hi(w) == 0 ? fx_double((uint64_t)neg << 63) : d;
}

// The node terms of MASK (component bits as node_terms) for the offsets of
// column c and z.  In place of the g_z term out[0] is its angle atan2(dz r, dx dy)
// (TIMES_DZ: times dz) and out[5], out[6] are ln(dy + r), ln(dx + r): g_z is
// dx out[5] + dy out[6] + dz out[0], which the kernels fold into their weights
// or sums.  False where the offsets are left to node_terms.
template <int MASK, bool TIMES_DZ = false>
J3G_FX bool fx_node(const FxColumn &c, const FxAxis &z, const FxTables &T, double *out) {
  constexpr bool need_gz = (MASK & 1) != 0;
  constexpr bool need_xx = (MASK & 2) != 0, need_yy = (MASK & 4) != 0, need_zz = (MASK & 8) != 0;
  constexpr bool need_xy = (MASK & 16) != 0, need_xz = (MASK & 32) != 0;
  constexpr bool need_yz = (MASK & 64) != 0;
  const bool bad = c.bad || z.bad != 0 || (c.mlo == 0 && z.m == 0);
  const FxRadius r = fx_radius(c.p, c.pe, c.pf, z);
  if constexpr (need_gz || need_yz)
    out[6] = fx_convert(fx_log_sum(c.mx, c.ex, c.negx, c.my, c.ey, z.m, z.e, r, T), 57, 0);
  if constexpr (need_gz || need_xz)
    out[5] = fx_convert(fx_log_sum(c.my, c.ey, c.negy, c.mx, c.ex, z.m, z.e, r, T), 57, 0);
  if constexpr (need_xy) {
    // log(dx^2 + dy^2) belongs to the column: below the station (dz < 0)
    // log(dz + r) is that less log(r - dz), above it log(r + dz)
    const int64_t t = fx_log(r.R + fx_shr(z.m, r.e - z.e), r.e, T);
    int64_t l = z.neg ? c.logp - t : t;
    l = l < kFxLogEps || (c.axial && z.neg) ? kFxLogEps : l;
    out[4] = fx_convert(l, 57, 0);
  }
  const uint64_t R4 = r.R << 2;
  uint64_t az = 0;  // the angle of z, scale 2^61
  if constexpr (need_xx || need_yy) {
    // hi, M = max(lo, |dz|) and m = min(lo, |dz|): the angles of hi and M are
    // the two smaller ones (where the leading bits are equal either may be M)
    const bool zbig = z.f >= c.flo;
    const uint64_t M = zbig ? z.m : c.mlo, m = zbig ? c.mlo : z.m;
    const int eM = zbig ? z.e : c.elo, em = zbig ? c.elo : z.e;
    const float fM = zbig ? z.f : c.flo, fm = zbig ? c.flo : z.f;
    const float imM = zbig ? z.im : c.imlo;
    const uint64_t D1 = fx_mul64(c.mhi, R4), D2 = fx_mul64(M, R4);
    const uint64_t n1 = fx_mul64(m, M), n2 = fx_mul64(c.mhi, m);
    const float fr = fm * r.inv;
    const int e0 = r.e - 2 - em;
    const FxAngle ah = fx_atan(n1, c.ehi - eM + e0, D1, fr * fM * c.ifhi, c.imhi * r.ys, T);
    const FxAngle aM = fx_atan(n2, eM - c.ehi + e0, D2, fr * c.fhi * fx_rcp(fM), imM * r.ys, T);
    const uint64_t am = c.axial ? 0 : nodetab::kPio2S61 - ah.v61 - aM.v61;  // the complement
    az = zbig ? aM.v61 : am;
    // every angle from its own bits: Uzz as a constant less Uxx and Uyy would save
    // a conversion, but keeps none of a small angle's leading bits (stations below
    // the mesh) and adds up two roundings elsewhere
    const uint32_t negM = zbig ? z.neg : c.neglo, negm = zbig ? c.neglo : z.neg;
    const double Fh = fx_quadrant(ah.v, ah.scale, ah.v61, c.neghi, c.neglo ^ z.neg);
    const double FM = fx_quadrant(aM.v, aM.scale, aM.v61, negM, c.neghi ^ negm);
    const double Fm =
        fx_convert((int64_t)(negm ? nodetab::kPiS61 - am : am), 61, c.neghi ^ negM);
    const double Fl = zbig ? Fm : FM;
    out[3] = zbig ? FM : Fm;
    out[1] = c.yhi ? Fl : Fh;
    out[2] = c.yhi ? Fh : Fl;
  } else if constexpr (need_zz || need_gz) {
    // the angle of z alone, from the smaller of the ratio and its inverse
    const uint64_t n = fx_mul64(c.mhi, c.mlo), d = fx_mul64(z.m, R4);
    const int en = c.ehi + c.elo, ed = z.e + r.e - 2;
    const float fn = c.fhi * c.flo, fd = z.f * r.f;
    const bool inv = fn > fd;
    const float t = (inv ? fd : fn) * fx_rcp(inv ? fn : fd);
    const float id = inv ? c.imhi * c.imlo * 536870912.0f : z.im * r.ys;  // 2^88 / D
    const FxAngle a = fx_atan(inv ? d << 3 : n, inv ? en + 4 - ed : ed - en, inv ? n >> 1 : d, t,
                              id, T);
    az = inv ? nodetab::kPio2S61 - a.v61 : a.v61;
    if constexpr (need_zz)
      out[3] = fx_quadrant(inv ? az : a.v, inv ? 61 : a.scale, az, z.neg, c.negx ^ c.negy);
  }
  if constexpr (need_gz) {
    const uint64_t w = c.negx ^ c.negy ? nodetab::kPio2S61 + az : nodetab::kPio2S61 - az;
    if constexpr (TIMES_DZ)
      out[0] = z.m == 0 ? 0.0 : fx_convert((int64_t)fx_mul64(w, z.m), -3 - z.e, 0);
    else
      out[0] = fx_convert((int64_t)w, 61, z.neg);
  }
  return !bad;
}

}  // namespace j3g
