// f64_node.cuh -- the pointwise terms and the 2-D neighbour sum of the complex128 paths with few
// FP64 instructions (sm_103a).
//
// What bounds the complex128 kernels is the FP64 pipe: on GB300 one FP64 instruction of a warp
// occupies its sub-partition for 64 cycles (76 with all four sub-partitions busy; measured with
// chains of DFMA, DADD and DMUL: 1.68 lane operations per cycle and SM), a conversion between
// double and float about 100, while FP32 and integer instructions issue every cycle.  So whatever
// keeps its accuracy in other arithmetic leaves the FP64 pipe:
//   * the reservoir and the coefficients a and b of the right-hand side (nls/nls.f90:570-650) are
//     evaluated in pairs of floats, 2^-45 of their terms at most.  About 150 FP32 and integer
//     instructions in place of 9 FP64 ones and two conversions;
//   * doubles are split into such pairs and put together again by integer operations;
//   * the neighbour part of the 2-D cross stencil (whose weights are whole numbers in units of
//     1/h^2 or 1/(12 h^2)) is one 64-bit fixed-point sum aligned to the largest neighbour, times
//     the unit, rounded once from 3-8 bits below a double's last place, so it is closer to the
//     exact value than the FP64 chain it replaces (8 FP64 instructions a node at order 3, 16 at
//     order 5).
// Values the float pairs cannot hold (non-finite, huge, or a denominator outside 2^+-60) and steps
// so long that the pairs' error would reach the state's last place (dt/2 times c3 r, c4, c5 |u|^2 or
// c6 r above 2^-8: the terms, since the error is a part of them, also where a or b vanishes because they
// cancel) take the plain FP64 expressions instead, decided per node.
//
// Where the pairs are coarser than FP64 with a one-Newton-step quotient, which they replaced (rms errors,
// measured on the GPU over the benchmark's coefficients, |u| <= 1): a is off by 2.8e-15 of its terms against
// 1.8e-15 with pumps up to 8, b by 3.2e-15 against 2.0e-15; without a pump, where FP64 has no quotient to
// form, a by 5.8e-16 against 0 and b by 2.3e-15 against 5e-17.  A slope also has the stencil in it, whose
// fixed-point sum is closer than the FP64 chain it replaced, so the whole slope is off by 0.69 to 0.97
// times as much at grid steps of 0.04 and with pumps up to 0.1 at 0.1 and 0.16, by 1.0 to 1.4 times at 0.1 and
// 0.16 with pumps up to 8, and by 1.5 to 8 times at a grid step of 1, where the stencil is small: there the
// limit above keeps it below the state's last place.  Final states against long double, geometric means of
// the error over that of the FP64 form: with a pump 0.67 (radial, 300 to 2501 nodes) and 0.76 (square, 40 to
// 100 a side) over 56 runs of 400 to 1000 steps at grid steps of 0.04 to 0.16; without one 0.91 to 1.05 by
// order and grid step, 0.04 to 1, over 96 runs.
// FP64 for everything but the quotient kept the coefficients at the former error and took 1.37 times
// as long at 900^2 order 3 (107.8 against 78.7 us a step), 1.25 times on radial grids.
//
// The pair operations are the published ones: f2_sum is Knuth's two-sum, f2_quick Dekker's fast
// two-sum, the products Dekker's with a fused multiply-add for the error.
#pragma once

#include <stdint.h>

#include <cstring>

#include "nls_types.h"

namespace nlsg {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float fbits(uint32_t v) { return __uint_as_float(v); }
__device__ __forceinline__ uint32_t bitsf(float v) { return __float_as_uint(v); }
__device__ __forceinline__ double dbits(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
__device__ __forceinline__ uint32_t dhi(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint32_t dlo(double v) { return (uint32_t)__double2loint(v); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float frcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float i2f(int x) { return __int2float_rn(x); }
__device__ __forceinline__ float fmax_abs(float a, float b) { return fmaxf(fabsf(a), fabsf(b)); }
__device__ __forceinline__ int f2i(float x) { return __float2int_rn(x); }
__device__ __forceinline__ uint32_t shf_l(uint32_t lo, uint32_t hi, int s) { return __funnelshift_l(lo, hi, s); }
// hi:lo >> s, zero from 64 on
__device__ __forceinline__ uint64_t shr64(uint32_t hi, uint32_t lo, uint32_t s) {
  uint64_t r;
  asm("{ .reg .b64 t; mov.b64 t, {%1, %2}; shr.u64 %0, t, %3; }" : "=l"(r) : "r"(lo), "r"(hi), "r"(s));
  return r;
}
__device__ __forceinline__ int clz64(uint64_t v) { return __clzll((long long)v); }
__device__ __forceinline__ uint32_t umulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ double dfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
#else
// Host forms, so that the arithmetic can be checked on the CPU.
static inline float fbits(uint32_t v) { float f; std::memcpy(&f, &v, 4); return f; }
static inline uint32_t bitsf(float v) { uint32_t u; std::memcpy(&u, &v, 4); return u; }
static inline double dbits(uint32_t hi, uint32_t lo) {
  const uint64_t u = ((uint64_t)hi << 32) | lo;
  double d;
  std::memcpy(&d, &u, 8);
  return d;
}
static inline uint32_t dhi(double v) { uint64_t u; std::memcpy(&u, &v, 8); return (uint32_t)(u >> 32); }
static inline uint32_t dlo(double v) { uint64_t u; std::memcpy(&u, &v, 8); return (uint32_t)u; }
static inline float ffma(float a, float b, float c) { return __builtin_fmaf(a, b, c); }
static inline float fadd(float a, float b) { return a + b; }
static inline float fmul(float a, float b) { return a * b; }
static inline float frcp(float x) { return 1.0f / x; }
static inline float i2f(int x) { return (float)x; }
static inline float fmax_abs(float a, float b) {
  a = a < 0.f ? -a : a;
  b = b < 0.f ? -b : b;
  return a > b ? a : b;
}
static inline int f2i(float x) { return (int)lrintf(x); }
static inline uint32_t shf_l(uint32_t lo, uint32_t hi, int s) { return (hi << s) | (lo >> (32 - s)); }
static inline uint64_t shr64(uint32_t hi, uint32_t lo, uint32_t s) {
  return s > 63 ? 0u : (((uint64_t)hi << 32) | lo) >> s;
}
static inline int clz64(uint64_t v) { return v ? __builtin_clzll(v) : 64; }
static inline uint32_t umulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline double dfma(double a, double b, double c) { return __builtin_fma(a, b, c); }
static inline double dadd(double a, double b) { return a + b; }
static inline double dmul(double a, double b) { return a * b; }
#endif

// Quotient of the plain expressions: a * (1/b), the reciprocal by two Newton steps from an FP32
// seed (good to a double's last place; one step leaves 2^-42); denominators outside the FP32 normal
// range take the IEEE division.
NLSG_HD inline double f64_div(double a, double b) {
  const float bf = (float)b;
  const float m = bf < 0.f ? -bf : bf;
  if (!(m >= 1e-30f && m <= 1e30f)) return a / b;
  double y = (double)frcp(bf);
  y = dfma(y, dfma(-b, y, 1.0), y);
  y = dfma(y, dfma(-b, y, 1.0), y);
  return a * y;
}

// A value held as hi + lo, |lo| at most about 2^-23 |hi|.
struct F2 {
  float h, l;
};

NLSG_HD inline F2 f2_quick(float a, float b) {  // a + b renormalised, |a| >= |b|
  F2 r;
  r.h = fadd(a, b);
  r.l = fadd(b, -fadd(r.h, -a));
  return r;
}

// A double as hi + lo, split by integer operations, hi the nearest float and lo its remainder to 24 bits,
// so to 2^-49 of it; values below 2^-96 become zero.  |v| must be below 2^60.
NLSG_HD inline F2 f2_split(double v) {
  const uint32_t hi = dhi(v), lo = dlo(v);
  const uint32_t mag = hi & 0x7fffffffu;
  const bool tiny = mag < ((1023u - 96u) << 20);
  const uint32_t t = mag - (896u << 20);
  const uint32_t f = shf_l(lo, t, 3) | (hi & 0x80000000u);  // sign, exponent - 896, 23 mantissa bits
  const uint32_t base = (f & 0xff800000u) - (23u << 23);    // the value of f's last place
  // the 29 bits below f's last place as a signed number: from half a place on, f is one place more
  const float rest = fmul(fmul(i2f((int)(lo << 3) >> 3), 0x1p-29f), fbits(base));
  return F2{tiny ? 0.f : fbits(f + ((lo >> 28) & 1u)), tiny ? 0.f : rest};
}

// hi + lo as a double, by integer operations.  |hi| in [2^-70, 2^60] keeps all of lo; smaller
// values keep hi alone (their lo is below 2^-93).
NLSG_HD inline double f2_join(F2 v) {
  // lo in units of a double's last place at hi's exponent (a whole number below 2^29), signed as it
  // changes hi's magnitude
  const uint32_t hb = bitsf(v.h), mag = hb & 0x7fffffffu;
  const uint32_t e = mag >> 23;
  const bool small = e < 57u;
  const float scale = fbits(((127u + 52u + 127u - (small ? 57u : e)) << 23) | (hb & 0x80000000u));
  int inc = small ? 0 : f2i(fmul(v.l, scale));
  // below a power of two the last place is half as large
  if ((mag & 0x7fffffu) == 0u && inc < 0) inc *= 2;
  const uint32_t dl = mag << 29;
  const uint32_t sl = dl + (uint32_t)inc;
  const uint32_t sh = (mag >> 3) + (896u << 20) + (uint32_t)(inc >> 31) + (sl < dl ? 1u : 0u);
  return mag == 0u ? 0.0 : dbits(sh | (hb & 0x80000000u), sl);
}

NLSG_HD inline F2 f2_sum(float a, float b) {    // a + b exactly
  F2 r;
  r.h = fadd(a, b);
  const float z = fadd(r.h, -a);
  r.l = fadd(fadd(a, -fadd(r.h, -z)), fadd(b, -z));
  return r;
}
NLSG_HD inline F2 f2_mul(F2 a, F2 b) {          // product, not renormalised
  F2 r;
  r.h = fmul(a.h, b.h);
  r.l = ffma(a.h, b.l, ffma(a.l, b.h, ffma(a.h, b.h, -r.h)));
  return r;
}
NLSG_HD inline F2 f2_add(F2 a, F2 b) {
  F2 s = f2_sum(a.h, b.h);
  s.l = fadd(s.l, fadd(a.l, b.l));
  return f2_quick(s.h, s.l);
}

// |v|^2 of one part as a pair, not renormalised: h exact with l.
NLSG_HD inline F2 f2_square(F2 x) {
  F2 r;
  r.h = fmul(x.h, x.h);
  r.l = ffma(x.l, x.l, ffma(fadd(x.h, x.h), x.l, ffma(x.h, x.h, -r.h)));
  return r;
}
// |u|^2 from the two squares.
NLSG_HD inline F2 f2_density(F2 x, F2 y) {
  const F2 s = f2_sum(x.h, y.h);
  return f2_quick(s.h, fadd(s.l, fadd(x.l, y.l)));
}
// p / d: a quotient whose remainder is exact in single precision, corrected twice; what is lost is below
// the last place of the low part.
NLSG_HD inline F2 f2_quotient(F2 p, F2 d) {
  const float yr = frcp(d.h);
  const float y0 = ffma(yr, ffma(-d.h, yr, 1.f), yr);
  const float q0 = fmul(p.h, y0);
  const float rem = ffma(-q0, d.h, p.h), low = ffma(-q0, d.l, p.l);
  const float q1 = fmul(rem, y0);
  return f2_quick(q0, ffma(fadd(ffma(-q1, d.h, rem), ffma(-q1, d.l, low)), y0, q1));
}
// p / (c13 + c14 s); ok: the denominator is in range.
NLSG_HD inline F2 f2_reservoir(F2 p, F2 s, const F64Consts& c, bool& ok) {
  const F2 d = f2_add(F2{c.h[0], c.l[0]}, f2_mul(F2{c.h[1], c.l[1]}, s));
  const float ad = d.h < 0.f ? -d.h : d.h;
  ok = ad > 0x1p-60f && ad < 0x1p60f;
  return f2_quotient(p, d);
}
// In range for the pairs: finite and below 2^40.
NLSG_HD inline bool f64_in_range(double v) { return (dhi(v) & 0x7fffffffu) < ((1023u + 40u) << 20); }

// A = c3 r - c4 and B = c5 |u|^2 + c6 r, r = c12 P / (c13 + c14 |u|^2) (a and b of nls_common.cuh),
// in pairs; false where they do not hold (the plain form then).  p: the pump split, p_ok: in range.
// The limit is on the terms (c4's is the host's part): A and B vanish where their terms cancel.
NLSG_HD inline bool f64_coeffs_pairs(double ux, double uy, F2 p, bool p_ok, const F64Consts& c, double& A, double& B) {
  const F2 s = f2_density(f2_square(f2_split(ux)), f2_square(f2_split(uy)));
  bool ok;
  const F2 r = f2_reservoir(p, s, c, ok);
  const F2 t3 = f2_mul(F2{c.h[2], c.l[2]}, r), t5 = f2_mul(F2{c.h[4], c.l[4]}, s), t6 = f2_mul(F2{c.h[5], c.l[5]}, r);
  A = f2_join(f2_add(F2{-c.h[3], -c.l[3]}, t3));
  B = f2_join(f2_add(t5, t6));
  return ok && c.fast != 0 && p_ok && f64_in_range(ux) && f64_in_range(uy) &&
         fmax_abs(fmax_abs(t5.h, t6.h), t3.h) < c.lim;
}
NLSG_HD inline void f64_coeffs_plain(double ux, double uy, double P, const F64Consts& c, double& A, double& B) {
  const double s = dfma(ux, ux, dmul(uy, uy));
  const double r = f64_div(P, dfma(c.d[1], s, c.d[0]));
  A = dfma(c.d[2], r, -c.d[3]);
  B = dfma(c.d[4], s, dmul(c.d[5], r));
}

// Neighbour part of the 2-D cross stencil: the unit times (v[0] + .. + v[3]) at K = 1, times
// (16 (v[0] + .. + v[3]) - (v[4] + .. + v[7])) at K = 2, v[0..3] at distance 1 and v[4..7] at distance 2.
// ok: false for neighbours all below 2^-900, near overflow, infinite or NaN (the plain form then).
template <int K>
NLSG_HD inline double cross_sum_fixed(const double (&v)[4 * K], const F64Consts& c, bool& ok) {
  constexpr int HEAD = K == 1 ? 3 : 8;   // bits above the largest neighbour's leading bit
  uint32_t h[4 * K], m = 0;
#pragma unroll
  for (int i = 0; i < 4 * K; ++i) {
    h[i] = dhi(v[i]) & 0x7fffffffu;
    m = h[i] > m ? h[i] : m;
  }
  const int emax = (int)(m >> 20), ebase = emax + c.unit_e - 1023;
  // (m in [123 << 20, 2030 << 20) and ebase in [80, 2030])
  ok = m - (123u << 20) < (1907u << 20) && (unsigned)(ebase - 80) <= 1950u && c.unit_e != 0;
  uint64_t sum = 0;
#pragma unroll
  for (int i = 0; i < 4 * K; ++i) {
    const uint32_t hi = dhi(v[i]), lo = dlo(v[i]);
    const uint32_t sh = (uint32_t)(emax + ((K == 2 && i < 4) ? HEAD - 4 : HEAD)) - (h[i] >> 20);
    // leading bit at bit 63, then shifted to the common scale (what falls off is below the last
    // place of the largest one by HEAD's complement to 11 bits; zeros shift out)
    const uint64_t x = shr64(shf_l(lo, (hi & 0xfffffu) | 0x100000u, 11), lo << 11, sh);
    const uint64_t neg = (uint64_t)((int64_t)(int32_t)(i < 4 ? hi : ~hi) >> 31);
    sum += (x ^ neg) - neg;
  }
  const uint64_t sgn = (uint64_t)((int64_t)sum >> 63);
  const uint64_t mag = (sum ^ sgn) - sgn;
  // times the unit's mantissa, both with bit 63 set: the product's bit 127 or 126 leads (its lowest
  // partial product and the carries out of the middle ones are below 2^-62)
  const int lz = clz64(mag);
  const uint64_t a = mag << (lz & 63);
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(c.unit_m >> 32), bl = (uint32_t)c.unit_m;
  uint64_t prod = (uint64_t)ah * bh + umulhi32(ah, bl) + umulhi32(al, bh);
  const int one = (int)(prod >> 63);
  prod <<= 1 - one;
  const uint64_t bits = ((uint64_t)(ebase + HEAD - 1 - lz + one) << 52) + (prod >> 11) + ((prod >> 10) & 1u);
  return mag == 0 ? 0.0 : dbits((uint32_t)(bits >> 32) | ((uint32_t)sgn & 0x80000000u), (uint32_t)bits);
}
template <int K>
NLSG_HD inline double cross_sum_plain(const double (&v)[4 * K], const F64Consts& c) {
  double s = dadd(dadd(v[0], v[1]), dadd(v[2], v[3]));
  if (K == 2) s = dfma(16.0, s, -dadd(dadd(v[4 * K - 4], v[4 * K - 3]), dadd(v[4 * K - 2], v[4 * K - 1])));
  return dmul(c.unit, s);
}

// A pump as a pair for the 2-D kernels; out of range: NaN, recognised by f2_pump_ok.
NLSG_HD inline F2 f2_pump(double P) {
  F2 p = f2_split(P);
  if (!f64_in_range(P)) p.l = fbits(0x7fc00000u);
  return p;
}
NLSG_HD inline bool f2_pump_ok(F2 p) { return p.l == p.l; }

// Slope of the 2-D model at a node u with the stencil's centre weight folded into B:
//   k_re = A u_re + (B - centre) u_im - S_im,   k_im = A u_im - (B - centre) u_re + S_re
// where S is the neighbour part.  Every complex128 2-D kernel uses these functions, so their results
// agree bit for bit.  The pairs and the fixed-point sums are evaluated without a branch between them
// (a warp alone on its sub-partition is bound by the latency of that arithmetic, which overlaps
// only within one block of code), the plain forms only where one of them does not hold.  *P is the
// pump that p was split from.
// In two parts: f64_coeffs_2d needs the node alone and gives A and B - centre, f64_slope_2d the rest.
NLSG_HD inline void f64_coeffs_2d(double ux, double uy, F2 p, bool p_ok, const double* P, const F64Consts& c, double& A,
                                  double& bw) {
  double B;
  if (!f64_coeffs_pairs(ux, uy, p, p_ok, c, A, B)) f64_coeffs_plain(ux, uy, *P, c, A, B);
  bw = dadd(B, -c.centre);
}
template <int K>
NLSG_HD inline void f64_slope_2d(double ux, double uy, const double (&vx)[4 * K], const double (&vy)[4 * K], double A,
                                 double bw, const F64Consts& c, double& kx, double& ky) {
  bool okx, oky;
  double sx = cross_sum_fixed<K>(vx, c, okx), sy = cross_sum_fixed<K>(vy, c, oky);
  if (!(okx && oky)) {
    if (!okx) sx = cross_sum_plain<K>(vx, c);
    if (!oky) sy = cross_sum_plain<K>(vy, c);
  }
  kx = dfma(A, ux, dfma(bw, uy, -sy));
  ky = dfma(A, uy, dfma(-bw, ux, sx));
}
template <int K>
NLSG_HD inline void f64_slope_2d(double ux, double uy, const double (&vx)[4 * K], const double (&vy)[4 * K],
                                 F2 p, bool p_ok, const double* P, const F64Consts& c, double& kx, double& ky) {
  double A, B;
  bool okx, oky;
  const bool ok = f64_coeffs_pairs(ux, uy, p, p_ok, c, A, B);
  double sx = cross_sum_fixed<K>(vx, c, okx), sy = cross_sum_fixed<K>(vy, c, oky);
  if (!(ok && okx && oky)) {
    if (!ok) f64_coeffs_plain(ux, uy, *P, c, A, B);
    if (!okx) sx = cross_sum_plain<K>(vx, c);
    if (!oky) sy = cross_sum_plain<K>(vy, c);
  }
  const double bw = dadd(B, -c.centre);
  kx = dfma(A, ux, dfma(bw, uy, -sy));
  ky = dfma(A, uy, dfma(-bw, ux, sx));
}

// Stage s of an RK4 step from its slope k: accumulates into acc and returns the next stage's input
// (s < 4) or the new state (s = 4).
template <typename C>
NLSG_HD inline C f64_stage(int s, const C& u, C& acc, const C& k, const F64Consts& c) {
  C t;
  if (s == 4) {
    t.x = dfma(c.dt6, dadd(acc.x, k.x), u.x);
    t.y = dfma(c.dt6, dadd(acc.y, k.y), u.y);
    return t;
  }
  if (s == 1) {
    acc = k;
  } else {
    acc.x = dfma(2.0, k.x, acc.x);
    acc.y = dfma(2.0, k.y, acc.y);
  }
  const double w = s == 3 ? c.dt : c.half_dt;
  t.x = dfma(w, k.x, u.x);
  t.y = dfma(w, k.y, u.y);
  return t;
}

// Slope of the 1-D model: row holds the operator's weights of u_{p-K} .. u_{p+K}.
template <int K>
NLSG_HD inline void f64_slope_1d(const double (&vx)[2 * K + 1], const double (&vy)[2 * K + 1],
                                 const double (&row)[2 * K + 1], F2 p, double P, bool p_ok, const F64Consts& c,
                                 double& kx, double& ky) {
  double A, B;
  if (!f64_coeffs_pairs(vx[K], vy[K], p, p_ok, c, A, B)) f64_coeffs_plain(vx[K], vy[K], P, c, A, B);
  double lx = dmul(row[0], vx[0]), ly = dmul(row[0], vy[0]);
#pragma unroll
  for (int d = 1; d <= 2 * K; ++d)
    if (d != K) {
      lx = dfma(row[d], vx[d], lx);
      ly = dfma(row[d], vy[d], ly);
    }
  const double bw = dadd(B, -row[K]);
  kx = dfma(A, vx[K], dfma(bw, vy[K], -ly));
  ky = dfma(A, vy[K], dfma(-bw, vx[K], lx));
}

#ifdef __CUDACC__
// The same with two adjacent lanes a node, part 0 its real and part 1 its imaginary part: each lane
// splits and squares its own part, the lanes exchange the squares, lane 0 forms A and lane 1 B.
struct F64Lane {
  F2 alpha, beta;   // lane 0: -c4 and c3 c12, lane 1: c5 and c6 c12
  int part;
};
__device__ __forceinline__ F64Lane f64_lane(int part, const F64Consts& c) {
  F64Lane l;
  l.part = part;
  l.alpha = part ? F2{c.h[4], c.l[4]} : F2{-c.h[3], -c.l[3]};
  l.beta = part ? F2{c.h[5], c.l[5]} : F2{c.h[2], c.l[2]};
  return l;
}
__device__ __forceinline__ float f64_other(float v) { return __shfl_xor_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double f64_other(double v) { return __shfl_xor_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ bool f64_coeffs_lanes(double mine, F2 p, bool p_ok, const F64Lane& l, const F64Consts& c,
                                                 double& A, double& B) {
  const F2 x = f2_square(f2_split(mine));
  const F2 o = F2{f64_other(x.h), f64_other(x.l)};
  const F2 s = l.part ? f2_density(o, x) : f2_density(x, o);
  bool ok;
  const F2 r = f2_reservoir(p, s, c, ok);
  const F2 ts = f2_mul(l.alpha, l.part ? s : F2{1.f, 0.f}), tr = f2_mul(l.beta, r);
  ok = ok && c.fast != 0 && p_ok && f64_in_range(mine) && fmax_abs(ts.h, tr.h) < c.lim;
  const double val = f2_join(f2_add(ts, tr)), his = f64_other(val);
  A = l.part ? his : val;
  B = l.part ? val : his;
  // every lane takes part in the exchange, whatever its own answer
  const int other_ok = __shfl_xor_sync(0xffffffffu, (int)ok, 1);
  return ok && other_ok != 0;
}
// The two parts of the slope for a lane of a pair: v the node, other the other part's neighbours.
__device__ __forceinline__ void f64_coeffs_2d_lanes(double2 v, F2 p, bool p_ok, const double* P, const F64Lane& l,
                                                    const F64Consts& c, double& A, double& bw) {
  double B;
  if (!f64_coeffs_lanes(l.part ? v.y : v.x, p, p_ok, l, c, A, B)) f64_coeffs_plain(v.x, v.y, *P, c, A, B);
  bw = dadd(B, -c.centre);
}
template <int K>
__device__ __forceinline__ double f64_slope_2d_lanes(double2 v, const double (&other)[4 * K], double A, double bw,
                                                     const F64Lane& l, const F64Consts& c) {
  bool oks;
  double s = cross_sum_fixed<K>(other, c, oks);
  if (!oks) s = cross_sum_plain<K>(other, c);
  // k_re = A u_re + m, k_im = A u_im - m with m = (B - centre) times the other part minus S
  const double m = dfma(bw, l.part ? v.x : v.y, -s);
  return dfma(A, l.part ? v.y : v.x, l.part ? -m : m);
}
// between(): FP64 work of the caller that does not depend on this slope, placed like the products.
template <int K, typename F>
__device__ __forceinline__ double f64_slope_1d_lanes(double2 v, const double (&other)[2 * K + 1],
                                                     const double (&row)[2 * K + 1], F2 p, double P, bool p_ok,
                                                     const F64Lane& l, const F64Consts& c, F&& between) {
  const double mine = l.part ? v.y : v.x, his = l.part ? v.x : v.y;
  // f64_coeffs_lanes with the operator's products placed where it waits (for the exchange of the
  // squares, the reciprocal, the exchange of the results): a warp alone on its sub-partition has
  // nothing else to issue there
  double s;
  auto tap = [&](int d) {
    if (d == 0) asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(s) : "d"(row[0]), "d"(other[0]));
    else asm volatile("fma.rn.f64 %0, %1, %2, %0;" : "+d"(s) : "d"(row[d]), "d"(other[d]));
  };
  const F2 x = f2_square(f2_split(mine));
  const F2 o = F2{f64_other(x.h), f64_other(x.l)};
  tap(0);
  if (K > 1) tap(1);
  const F2 q = l.part ? f2_density(o, x) : f2_density(x, o);
  bool ok;
  const F2 r = f2_reservoir(p, q, c, ok);
  if (K > 2) tap(2);
  tap(K + 1);
  const F2 t = f2_mul(l.alpha, l.part ? q : F2{1.f, 0.f}), tr = f2_mul(l.beta, r);
  ok = ok && c.fast != 0 && p_ok && f64_in_range(mine) && fmax_abs(t.h, tr.h) < c.lim;
  const double val = f2_join(f2_add(t, tr)), hval = f64_other(val);
  const int other_ok = __shfl_xor_sync(0xffffffffu, (int)ok, 1);
#pragma unroll
  for (int d = K + 2; d <= 2 * K; ++d) tap(d);
  between();
  double A = l.part ? hval : val, B = l.part ? val : hval;
  if (!(ok && other_ok != 0)) f64_coeffs_plain(v.x, v.y, P, c, A, B);
  const double m = dfma(dadd(B, -row[K]), his, -s);
  return dfma(A, mine, l.part ? -m : m);
}
// This lane's part of f64_stage.
__device__ __forceinline__ double f64_stage_lane(int s, double u, double& acc, double k, const F64Consts& c) {
  if (s == 4) return dfma(c.dt6, dadd(acc, k), u);
  acc = s == 1 ? k : dfma(2.0, k, acc);
  return dfma(s == 3 ? c.dt : c.half_dt, k, u);
}
#endif

}  // namespace nlsg
