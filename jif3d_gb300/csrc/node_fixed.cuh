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
//             atan(N/D) = atan(j/512) + atan(d), d = (N - jD/512) / (D + jN/512),
//             |d| <= 2^-10, by two digits of long division with a Newton
//             reciprocal, atan d = d - d^3/3 + d^5/5
//
// Offsets beyond 2^+-40, dz and another offset both exactly zero, and logarithms
// of an argument within 2^-25 of one are left to node_terms (fx_node returns
// false).
// The same code compiles for the host, where its accuracy is tested.
#pragma once
#include <cstdint>
#include <cstring>

#include "node_tables.h"

#ifdef __CUDACC__
#define J3G_FX __device__ __forceinline__
#else
#include <cmath>
#define J3G_FX static inline
#endif

namespace j3g {

#ifdef __CUDACC__
J3G_FX uint32_t fx_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
J3G_FX int32_t fx_mulhi_s(int32_t a, int32_t b) { return __mulhi(a, b); }
J3G_FX int fx_clz(uint32_t a) { return __clz((int)a); }
J3G_FX float fx_rsqrt(float a) { return rsqrtf(a); }
J3G_FX float fx_rcp(float a) { return __fdividef(1.0f, a); }
J3G_FX uint32_t fx_f2u(float a) { return __float2uint_rz(a); }
J3G_FX uint32_t fx_bits(float a) { return __float_as_uint(a); }
J3G_FX float fx_float(uint32_t a) { return __uint_as_float(a); }
J3G_FX uint64_t fx_bits(double a) { return (uint64_t)__double_as_longlong(a); }
J3G_FX double fx_double(uint64_t a) { return __longlong_as_double((long long)a); }
J3G_FX double fx_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
J3G_FX uint32_t fx_mulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
J3G_FX int32_t fx_mulhi_s(int32_t a, int32_t b) { return (int32_t)((int64_t)a * b >> 32); }
J3G_FX int fx_clz(uint32_t a) { return a ? __builtin_clz(a) : 32; }
J3G_FX float fx_rsqrt(float a) { return 1.0f / sqrtf(a); }
J3G_FX float fx_rcp(float a) { return 1.0f / a; }
J3G_FX uint32_t fx_f2u(float a) { return (uint32_t)a; }
J3G_FX uint32_t fx_bits(float a) { uint32_t u; memcpy(&u, &a, 4); return u; }
J3G_FX float fx_float(uint32_t a) { float f; memcpy(&f, &a, 4); return f; }
J3G_FX uint64_t fx_bits(double a) { uint64_t u; memcpy(&u, &a, 8); return u; }
J3G_FX double fx_double(uint64_t a) { double d; memcpy(&d, &a, 8); return d; }
J3G_FX double fx_fma(double a, double b, double c) { return std::fma(a, b, c); }
#endif

J3G_FX uint32_t fx_hi(uint64_t v) { return (uint32_t)(v >> 32); }
J3G_FX uint32_t fx_lo(uint64_t v) { return (uint32_t)v; }
J3G_FX int fx_min(int a, int b) { return a < b ? a : b; }
// floor(x y / 2^64) up to two units (the lo x lo product is left out)
J3G_FX uint64_t fx_mul64(uint64_t x, uint64_t y) {
  return (uint64_t)fx_hi(x) * fx_hi(y) + fx_mulhi(fx_hi(x), fx_lo(y)) +
         fx_mulhi(fx_lo(x), fx_hi(y));
}
// floor(x y / 2^32) for a 32-bit y, up to one unit (no overflow: x y < 2^96)
J3G_FX uint64_t fx_mul32(uint64_t x, uint32_t y) {
  return (uint64_t)fx_hi(x) * y + fx_mulhi(fx_lo(x), y);
}

// log(DBL_EPSILON) = -52 log 2, scale 2^57
constexpr int64_t kFxLogEpsS57 =
    -52 * (int64_t)nodetab::kLn2 - (int64_t)((52ull * nodetab::kLn2Low) >> 32);
constexpr int kFxZeroExp = -4096;  // exponent of a zero offset: shifted out of every sum

// One offset |d| = m 2^e (m = 0 or top bit set), d^2 = q 2^qe with q in
// [2^61, 2^63) and qe even, and FP32 values |d|, d^2 and 2^63 / m.
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
  a.m = zero ? 0 : ((b << 11) | 0x8000000000000000ull);
  a.e = zero ? kFxZeroExp : (int)eb - 1023 - 63;
  // the leading 24 bits as a float: 2^(eb - 1023) [1, 2)
  const uint32_t frac = fx_hi(a.m) >> 8 & 0x7fffffu;
  a.f = zero || a.bad ? 0.0f : fx_float((eb - 1023u + 127u) << 23 | frac);
  a.f2 = a.f * a.f;
  a.im = fx_rcp(fx_float(127u << 23 | frac));
  const uint64_t q = fx_mul64(a.m, a.m);  // [2^62, 2^64)
  const bool big = (q >> 63) != 0;
  a.q = big ? q >> 2 : q;
  a.qe = zero ? kFxZeroExp : 2 * a.e + 64 + (big ? 2 : 0);
  return a;
}

// q 2^qe of two sums of squares, aligned at the larger exponent.
J3G_FX void fx_add_sq(uint64_t qa, int ea, uint64_t qb, int eb, uint64_t &s, int &es) {
  const int d = ea - eb;
  const uint64_t big = d >= 0 ? qa : qb, small = d >= 0 ? qb : qa;
  es = d >= 0 ? ea : eb;
  s = big + (small >> fx_min(d >= 0 ? d : -d, 63));
}

// The offsets of one node column (fixed x and y, all z) from one station:
// the larger (hi) and the smaller (lo) of |dx| and |dy|, and dx^2 + dy^2.
struct FxColumn {
  uint64_t mx, my, mhi, mlo, p;
  int64_t logp;  // log(dx^2 + dy^2), scale 2^57 (where Uxy is wanted)
  int ex, ey, ehi, elo, pe;
  float fhi, flo, imhi, imlo, pf;
  uint32_t negx, negy;
  bool yhi;    // |dy| > |dx|
  bool axial;  // dx = dy = 0: the station is above or below the column
  bool bad;
};

J3G_FX FxColumn fx_column_base(const FxAxis &x, const FxAxis &y) {
  FxColumn c;
  c.yhi = y.e > x.e || (y.e == x.e && y.m > x.m);
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
  fx_add_sq(x.q, x.qe, y.q, y.qe, c.p, c.pe);  // below 2^64
  const bool big = (c.p >> 63) != 0;
  c.p = big ? c.p >> 2 : c.p;
  c.pe += big ? 2 : 0;
  c.pf = x.f2 + y.f2;
  c.negx = x.neg;
  c.negy = y.neg;
  c.axial = c.mhi == 0;
  // zeros come as +0 (a difference of equal coordinates)
  c.bad = (x.bad | y.bad) != 0 || (c.axial && (x.neg | y.neg));
  return c;
}

// r = R 2^e with R in [2^59.5, 2^61); 2^90 / R, r and 1/r as floats.
struct FxRadius {
  uint64_t R;
  int e;
  float ys, f, inv;
};

J3G_FX FxRadius fx_radius(const FxColumn &c, const FxAxis &z) {
  uint64_t s;
  int es;
  fx_add_sq(c.p, c.pe, z.q, z.qe, s, es);  // [2^61, 2^64), es even
  FxRadius r;
  const float sf = c.pf + z.f2;
  r.inv = fx_rsqrt(sf);
  r.f = sf * r.inv;
  // 2^61 / sqrt(s): r.inv times 2^(61 + es/2)
  r.ys = r.inv * fx_float((uint32_t)(127 + 61 + es / 2) << 23);
  const uint32_t y0 = fx_f2u(r.ys);  // (2^29, 2^30.5]
  const uint32_t yy = (uint32_t)((uint64_t)y0 * y0 >> 30);  // 2^92 / s
  const int64_t d = (int64_t)((1ull << 60) - (uint64_t)fx_hi(s) * yy);
  const uint32_t y = y0 + (uint32_t)((int64_t)(int32_t)y0 * (int32_t)(d >> 10) >> 51);
  const uint64_t p = fx_mul32(s, y);  // sqrt(s) 2^29
  const int32_t t = (int32_t)((1ull << 58) - fx_mul32(p, y));
  r.R = p + (uint64_t)((int64_t)(int32_t)fx_hi(p) * t >> 27);
  r.e = es / 2 - 29;
  return r;
}

// log(u 2^e) at scale 2^57 for u in [2^32, 2^63).
J3G_FX int64_t fx_log(uint64_t u, int e, const uint32_t *G, const uint64_t *L) {
  const int n = fx_clz(fx_hi(u));
  const uint64_t m = u << n;
  const uint32_t j = fx_hi(m) >> 22 & 511u;
  const int64_t z = (int64_t)(fx_mul32(m, G[j]) << 9);  // z 2^72 (the leading one shifts out)
  const int32_t zh = (int32_t)(z >> 32);                // z 2^40
  const int32_t zl = (int32_t)(fx_lo(z) >> 1);
  const int64_t zz = (int64_t)zh * zh + ((int64_t)zh * zl >> 30);  // z^2 2^80
  const int32_t zc = zh >> 8;                                      // z 2^32
  const int32_t c = 1431655765 - fx_mulhi_s(zc, 1073741824 - fx_mulhi_s(zc, 858993459));
  const int32_t z3 = (int32_t)((int64_t)(int32_t)(zz >> 32) * zh >> 27);  // z^3 2^61
  const uint32_t k = (uint32_t)(e + 63 - n + nodetab::kLogBias);
  const int64_t t = (z >> 15) - (zz >> 24) + (fx_mulhi_s(z3, c) >> 4);
  return (int64_t)(k * nodetab::kLn2 + fx_mulhi(k, nodetab::kLn2Low) + L[j]) + t;
}

// log(max(d + r, eps)) of one offset d = +-m 2^e (a = m aligned to r) where
// the other two are mb 2^eb and mc 2^ec.  A negative offset that takes off
// more than ten bits of r goes through d + r = (b^2 + c^2) / (r - d).
J3G_FX int64_t fx_log_sum(uint64_t m, int e, uint32_t neg, uint64_t mb, int eb, uint64_t mc,
                          int ec, const FxRadius &r, const uint32_t *G, const uint64_t *L) {
  const uint64_t a = m >> fx_min(r.e - e, 63);
  const uint64_t u = neg ? r.R - a : r.R + a;
  if (fx_hi(u) >= fx_hi(r.R) >> 10) return fx_log(u, r.e, G, L);
  const uint64_t qb = fx_mul64(mb, mb), qc = fx_mul64(mc, mc);
  uint64_t s;
  int es;
  fx_add_sq(qb >> 2, mb ? 2 * eb + 66 : kFxZeroExp, qc >> 2, mc ? 2 * ec + 66 : kFxZeroExp, s, es);
  const int64_t l = fx_log(s, es, G, L) - fx_log(r.R + a, r.e, G, L);
  return l < kFxLogEpsS57 ? kFxLogEpsS57 : l;
}

template <int MASK>
J3G_FX FxColumn fx_column(const FxAxis &x, const FxAxis &y, const uint32_t *G,
                          const uint64_t *L) {
  FxColumn c = fx_column_base(x, y);
  c.logp = MASK & 16 ? fx_log(c.p, c.pe, G, L) : 0;
  return c;
}

// v 2^-scale as a double (v unsigned below 2^63; hi word zero counts as zero).
J3G_FX double fx_to_double(uint64_t v, int scale, uint32_t neg) {
  const int n = fx_clz(fx_hi(v));
  const uint64_t m = v << n;
  const uint64_t b = (m >> 11) + (m >> 10 & 1);
  const uint32_t hi = fx_hi(b) + ((uint32_t)(1023 + 62 - scale - n) << 20);
  const uint64_t r = ((uint64_t)hi << 32) | fx_lo(b);
  return fx_double((n >= 32 ? 0 : r) | (uint64_t)neg << 63);
}

J3G_FX double fx_log_double(int64_t l, bool &bad) {
  const uint32_t neg = (uint32_t)((uint64_t)l >> 63);
  const uint64_t v = (uint64_t)(l ^ (l >> 63));
  bad |= fx_hi(v) == 0;
  return fx_to_double(v, 57, neg);
}

// An angle: v 2^-scale, and the same at scale 2^61.
struct FxAngle {
  uint64_t v, v61;
  int scale;
};

// atan(N / D) <= pi/4 for N = n1 2^-s (n1 in [2^62, 2^64) or 0), D in
// [2^58, 2^61), t = N / D and idy = 2^89 / D as floats.
J3G_FX FxAngle fx_atan(uint64_t n1, int s, uint64_t D, float t, float idy,
                       const uint64_t *A) {
  // ratios below 2^-11 (j = 0) are scaled by 2^x into [2^-11, 2^-10), so that
  // small angles keep their leading bits; N is then at 2^9 the scale of D
  int x = 116 - (int)(fx_bits(t) >> 23);
  x = x > 0 ? x : 0;
  s -= x;
  const bool wide = s < 9;
  const uint64_t nb = n1 >> fx_min(wide ? s : s - 9, 63);
  const uint64_t n9 = wide ? nb << 9 : nb;  // modulo 2^64, as the difference below
  uint32_t j = fx_f2u(t * 512.0f + 0.5f);
  j = j < 512u ? j : 512u;
  const int64_t num = (int64_t)(n9 - (uint64_t)j * D);                    // |num| <= D / 2
  const uint64_t den = D + ((uint64_t)j * (nb >> (wide ? 7 : 16)) >> 2);  // below 2^62
  const uint32_t y0 = fx_f2u(idy * fx_rcp(1.0f + (float)j * (1.0f / 512.0f) * t));  // 2^89 / den
  const int64_t d = (int64_t)((1ull << 59) - (uint64_t)(uint32_t)(den >> 30) * y0);
  const int32_t y = (int32_t)(y0 + (uint32_t)((int64_t)(int32_t)y0 * (int32_t)(d >> 10) >> 49));
  const int32_t q0 = (int32_t)((int64_t)(int32_t)(num >> 30) * y >> 33);  // 2^26 num / den
  const int64_t rem = (int64_t)(((uint64_t)num << 26) - (uint64_t)(int64_t)q0 * den);
  // 2^57 rem / den, then 2^61 num / den = 2^70 d (scaled by 2^x)
  const int64_t q1 = (int64_t)(int32_t)(rem >> 32) * y + fx_mulhi(fx_lo((uint64_t)rem), (uint32_t)y);
  const int64_t q = ((int64_t)q0 << 35) + (q1 >> 22);
  // d - d^3/3 + d^5/5 with d = 2^-9 dh 2^-31
  const int32_t dh = (int32_t)(q >> 30);
  const uint32_t d2 = (uint32_t)((uint64_t)((int64_t)dh * dh) >> 29);  // 2^33 (2^9 d)^2
  const uint32_t c = fx_mulhi(d2, 1431655765u - (fx_mulhi(d2, 858993459u) >> fx_min(19 + 2 * x, 31)));
  const int64_t cube = (int64_t)dh * (int32_t)c;  // 2^91 (d^3/3 - d^5/5)
  const int64_t small = q - (cube >> fx_min(21 + 2 * x, 63));  // scale 2^70 (2^x)
  FxAngle r;
  const uint64_t sum = A[j] + (uint64_t)(small >> 8);  // scale 2^62
  r.v = j ? sum : (uint64_t)small;
  r.scale = j ? 62 : 70 + x;
  r.v61 = j ? sum >> 1 : (uint64_t)small >> fx_min(9 + x, 63);
  return r;
}

// atan2 from the angle of the magnitudes: `own` the sign of the abscissa's
// offset, neg the sign of the ordinate.
J3G_FX double fx_quadrant(const FxAngle &a, uint32_t own, uint32_t neg) {
  const uint64_t v = own ? nodetab::kPiS61 - a.v61 : a.v;
  return fx_to_double(v, own ? 61 : a.scale, neg);
}

// The node terms of MASK (component bits as node_terms) for the offsets of
// column c and z; dx, dy, dz the same offsets as doubles.  False where the
// offsets are left to node_terms.
template <int MASK>
J3G_FX bool fx_node(const FxColumn &c, const FxAxis &z, double dx, double dy, double dz,
                    const uint32_t *G, const uint64_t *L, const uint64_t *A, double *out) {
  constexpr bool need_gz = (MASK & 1) != 0;
  constexpr bool need_xx = (MASK & 2) != 0, need_yy = (MASK & 4) != 0, need_zz = (MASK & 8) != 0;
  constexpr bool need_xy = (MASK & 16) != 0, need_xz = (MASK & 32) != 0;
  constexpr bool need_yz = (MASK & 64) != 0;
  bool bad = c.bad || z.bad != 0 || (c.mlo == 0 && z.m == 0);
  const FxRadius r = fx_radius(c, z);
  double lx = 0.0, ly = 0.0;
  if constexpr (need_gz || need_yz) {
    lx = fx_log_double(fx_log_sum(c.mx, c.ex, c.negx, c.my, c.ey, z.m, z.e, r, G, L), bad);
    if constexpr (need_yz) out[6] = lx;
  }
  if constexpr (need_gz || need_xz) {
    ly = fx_log_double(fx_log_sum(c.my, c.ey, c.negy, c.mx, c.ex, z.m, z.e, r, G, L), bad);
    if constexpr (need_xz) out[5] = ly;
  }
  if constexpr (need_xy) {
    // log(dx^2 + dy^2) belongs to the column: below the station (dz < 0)
    // log(dz + r) is that less log(r - dz), above it log(r + dz)
    const int64_t t = fx_log(r.R + (z.m >> fx_min(r.e - z.e, 63)), r.e, G, L);
    int64_t l = z.neg ? c.logp - t : t;
    l = l < kFxLogEpsS57 ? kFxLogEpsS57 : l;
    out[4] = fx_log_double(c.axial && z.neg ? kFxLogEpsS57 : l, bad);
  }
  FxAngle az;
  if constexpr (need_xx || need_yy) {
    // hi, M = max(lo, |dz|) and m = min(lo, |dz|): the angles of hi and M are
    // the two smaller ones
    const bool zbig = z.e > c.elo || (z.e == c.elo && z.m >= c.mlo);
    const uint64_t M = zbig ? z.m : c.mlo, m = zbig ? c.mlo : z.m;
    const int eM = zbig ? z.e : c.elo, em = zbig ? c.elo : z.e;
    const float fM = zbig ? z.f : c.flo, fm = zbig ? c.flo : z.f;
    const float imM = zbig ? z.im : c.imlo;
    const float ihi = c.imhi * r.ys, iM = imM * r.ys;  // 2^89 / D of both
    const uint64_t D1 = fx_mul64(c.mhi, r.R), D2 = fx_mul64(M, r.R);
    const uint64_t n1 = fx_mul64(m, M), n2 = fx_mul64(c.mhi, m);
    const float fr = fm * r.inv;
    const FxAngle ah = fx_atan(n1, fx_min(c.ehi + r.e - em - eM, 4000), D1,
                               fr * fM * fx_rcp(c.fhi), ihi, A);
    const FxAngle aM = fx_atan(n2, fx_min(eM + r.e - em - c.ehi, 4000), D2,
                               fr * c.fhi * fx_rcp(fM), iM, A);
    FxAngle am;  // the complement
    am.v61 = c.axial ? 0 : nodetab::kPio2S61 - ah.v61 - aM.v61;
    am.v = am.v61;
    am.scale = 61;
    az = zbig ? aM : am;
    const FxAngle al = zbig ? am : aM;
    const FxAngle ax = c.yhi ? al : ah, ay = c.yhi ? ah : al;
    out[1] = fx_quadrant(ax, c.negx, c.negy ^ z.neg);
    out[2] = fx_quadrant(ay, c.negy, c.negx ^ z.neg);
  } else if constexpr (need_zz || need_gz) {
    // the angle of z alone, from the smaller of the ratio and its inverse;
    // with t the smaller ratio and F the common scale of its terms
    const uint64_t n = fx_mul64(c.mhi, c.mlo), d = fx_mul64(z.m, r.R << 2);
    const int en = c.ehi + c.elo, ed = z.e + r.e - 2;
    const float fn = c.fhi * c.flo, fd = z.f * r.f;
    const bool inv = fn > fd;
    const float t = (inv ? fd : fn) * fx_rcp(inv ? fn : fd);
    const float id = inv ? c.imhi * c.imlo * 1073741824.0f : z.im * r.ys;  // 2^89 / D
    az = fx_atan(inv ? d : n, fx_min(inv ? en + 3 - ed : ed + 2 - en, 4000),
                 inv ? n >> 3 : d >> 2, t, id, A);
    az.v61 = inv ? nodetab::kPio2S61 - az.v61 : az.v61;
    az.v = inv ? az.v61 : az.v;
    az.scale = inv ? 61 : az.scale;
  }
  if constexpr (need_zz) out[3] = fx_quadrant(az, z.neg, c.negx ^ c.negy);
  if constexpr (need_gz) {
    const uint64_t h = nodetab::kPio2S61;
    const double a = fx_to_double(c.negx ^ c.negy ? h + az.v61 : h - az.v61, 61, z.neg);
    out[0] = fx_fma(dx, ly, fx_fma(dy, lx, dz * a));
  }
  return !bad;
}

}  // namespace j3g
