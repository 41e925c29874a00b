// FP64 arithmetic of one exposure sample of the transit and eclipse models,
// written for a chip whose FP64 pipe is 1/64 of its FP32 pipe.
//
// What bounds the FP64 kernels is the number of FP64 instructions: a warp's
// FP64 instruction holds its quarter of the SM for ~75 cycles (1.70 lanes per
// clock and SM, measured), as long as 75 FP32 instructions.  So every FP64
// step here is there because FP64 accuracy needs it, and seeds, indices,
// conversions and corrections far below the last place are FP32 or integer:
//   z = sqrt(x^2 + y^2): the polynomial of r^2 in t (8 FP64 instructions
//     instead of 10 for x, y and the sum), then one third-order step from the
//     FP32 reciprocal root (4, against 7-8 for sqrt);
//   the LD-mean lerp with reciprocals (3, against ~25 with two divisions);
//   the limb's overlap area with two table-based angles (21, against ~90 for
//     two atan2, a square root and a sorted product).
// Each operation is written with its rounding (__fma_rn, __dmul_rn,
// __dadd_rn), so a sample has the same bits in every kernel that calls it.
//
// Error: each FP64 result is within an ulp or two of its exact value, as the
// reference's operations are; over 8192 x 19,700 points the flux differs from
// the reference's operations by at most 1.1e-16 (4.4e-16 with 10 samples).
#pragma once
#include "rr_device.cuh"

namespace rr {

// ---------------------------------------------------------------------------
// sin and cos of i/512, i/512 in [0, pi]: made at compile time in
// double-double arithmetic (Dekker's error-free sum and product) by rotating
// (1, 0) through 1/512, whose sine and cosine come from their Taylor series,
// so that every entry is the rounded exact value.
// ---------------------------------------------------------------------------
constexpr int ANG_PER_RAD = 512;
constexpr int ANG_N = 1610;   // up to 1609/512 > pi

struct DD {
  double h, l;
};
constexpr DD dd_norm(double a, double b) {
  const double s = a + b;
  const double bb = s - a;
  return DD{s, (a - (s - bb)) + (b - bb)};
}
constexpr DD dd_prod(double a, double b) {
  const double p = a * b;
  const double ca = 134217729.0 * a, cb = 134217729.0 * b;   // 2^27 + 1 (Dekker's split)
  const double ah = ca - (ca - a), al = a - ah, bh = cb - (cb - b), bl = b - bh;
  return DD{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr DD dd_mul(DD a, DD b) {
  const DD p = dd_prod(a.h, b.h);
  return dd_norm(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr DD dd_add(DD a, DD b) {
  const DD s = dd_norm(a.h, b.h);
  return dd_norm(s.h, s.l + (a.l + b.l));
}
constexpr DD dd_neg(DD a) { return DD{-a.h, -a.l}; }
constexpr DD dd_div_int(DD a, double n) {
  const double q = a.h / n;
  const DD r = dd_prod(q, n);
  return dd_norm(q, (((a.h - r.h) - r.l) + a.l) / n);
}

struct alignas(16) AngleTable {
  double sc[ANG_N][2];   // sin, cos
};

constexpr AngleTable make_angle_table() {
  const DD h{1.0 / ANG_PER_RAD, 0.0}, h2 = dd_mul(h, h);
  DD s1{0, 0}, c1{0, 0}, term{1.0, 0.0};
  for (int n = 0; n < 12; n += 2) {   // the term h^n / n! with its sign
    c1 = dd_add(c1, term);
    s1 = dd_add(s1, dd_div_int(dd_mul(term, h), n + 1.0));
    term = dd_neg(dd_div_int(dd_div_int(dd_mul(term, h2), n + 1.0), n + 2.0));
  }
  AngleTable t{};
  DD s{0, 0}, c{1.0, 0.0};
  for (int i = 0; i < ANG_N; ++i) {
    t.sc[i][0] = s.h;
    t.sc[i][1] = c.h;
    const DD sn = dd_add(dd_mul(s, c1), dd_mul(c, s1));
    c = dd_add(dd_mul(c, c1), dd_neg(dd_mul(s, s1)));
    s = sn;
  }
  return t;
}

__device__ constexpr AngleTable ANGLES = make_angle_table();

// ---------------------------------------------------------------------------
// Conversions on the integer pipe (a conversion between FP32 and FP64 costs as
// much as an FP64 operation).
// ---------------------------------------------------------------------------
constexpr int F64_BIAS = (1023 - 127) << 20;

// FP32 (truncated) of a positive double in FP32's normal range.
__device__ __forceinline__ float f32_of_pos(double d) {
  return __uint_as_float(__funnelshift_l(__double2loint(d), __double2hiint(d) - F64_BIAS, 3));
}
// FP32 (truncated) of any double: 0 below FP32's normal range, 2^127 or more
// (never NaN) above it and for NaN.
__device__ __forceinline__ float f32_of(double d) {
  const unsigned hi = __double2hiint(d);
  const unsigned m = min(max((int)(hi & 0x7fffffffu), F64_BIAS), F64_BIAS + (254 << 20)) - F64_BIAS;
  return __uint_as_float(__funnelshift_l(__double2loint(d), m, 3) | (hi & 0x80000000u));
}
// Neither infinite nor NaN.
__device__ __forceinline__ bool f64_finite(double d) { return (__double2hiint(d) & 0x7ff00000) != 0x7ff00000; }
// FP32 of a double, its magnitude rounded up by an ulp; NaN and infinity stay.
__device__ __forceinline__ float f32_up(double d) {
  return f64_finite(d) ? __uint_as_float(__float_as_uint(f32_of(d)) + 1u) : (float)d;
}
// FP64 of a non-negative FP32 value (0 becomes 2^-127).
__device__ __forceinline__ double f64_of_pos(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)(b >> 3) + F64_BIAS, (int)(b << 29));
}
// FP64 of an FP32 value of either sign (0 becomes +-2^-127).
__device__ __forceinline__ double f64_of(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + F64_BIAS)), (int)(b << 29));
}
// Magnitude between 2^-100 and 2^100 and a positive sign (excludes NaN).
__device__ __forceinline__ bool f64_moderate(double d) {
  return (unsigned)__double2hiint(d) - ((1023u - 100u) << 20) < (200u << 20);
}

// FP32 of any double, rounded to nearest even as the conversion does.
__device__ __forceinline__ float f32_near(double d) {
  if (!f64_moderate(fabs(d))) return (float)d;
  const unsigned long long u = __double_as_longlong(d);
  const unsigned long long b = u + 0x0fffffffull + ((u >> 29) & 1u);   // a carry goes into the exponent
  const unsigned hi = (unsigned)(b >> 32);
  return __uint_as_float(__funnelshift_l((unsigned)b, (hi & 0x7fffffffu) - F64_BIAS, 3) | (hi & 0x80000000u));
}

// FP32 pair (48 bits) of a double: its upper 24 bits and the rest.  Below 2^-70, where
// FP32 does not hold the rest, the rounded value alone; so too above 2^100 and for NaN.
__device__ __forceinline__ float2 f32_pair(double d) {
  const int e = (__double2hiint(d) >> 20) & 0x7ff;
  if (e < 1023 - 70 || e > 1023 + 100) return make_float2((float)d, 0.0f);
  const float h = f32_of(d), rest = (float)(__double2loint(d) & 0x1fffffff) * __int_as_float((e - 1023 - 52 + 127) << 23);
  return make_float2(h, copysignf(rest, h));
}

// Square root of a moderate x and its reciprocal, from the FP32 reciprocal
// root g: with e = 1 - x g^2 (|e| < 4e-7), 1/sqrt(x) = g (1 + e/2 + 3 e^2/8 +
// O(e^3)), the quadratic term (below 1e-13) in FP32.
struct F64Root {
  double s0, g, w;   // sqrt = s0 + s0 w, 1/sqrt = g + g w
};
__device__ __forceinline__ F64Root f64_root(double x) {
  F64Root r;
  r.g = f64_of_pos(rsqrtf(f32_of_pos(x)));
  r.s0 = __dmul_rn(x, r.g);
  const double e = __fma_rn(-r.s0, r.g, 1.0);
  const float ef = f32_of(e);
  r.w = __fma_rn(e, 0.5, f64_of_pos(0.375f * ef * ef));
  return r;
}
__device__ __forceinline__ double f64_sqrt(const F64Root& r) { return __fma_rn(r.s0, r.w, r.s0); }
__device__ __forceinline__ double f64_rsqrt(const F64Root& r) { return __fma_rn(r.g, r.w, r.g); }

// 1 / x: a third-order step from the FP32 reciprocal for a moderate x (3 FP64
// instructions, against 7-8 for the division).
__device__ __forceinline__ double f64_recip(double x) {
  if (!f64_moderate(x)) return __ddiv_rn(1.0, x);
  const double y = f64_of_pos(1.0f / f32_of_pos(x));
  const double e = __fma_rn(-x, y, 1.0);
  return __fma_rn(y, __fma_rn(e, e, e), y);
}

// floor of a quotient from its FP32 value q, where q's error (tol) leaves no
// doubt about it.
__device__ __forceinline__ bool f64_floor_sure(float q, float& n) {
  n = floorf(q);
  const float tol = fmaf(fabsf(q), 2e-6f, 1e-30f);
  return fabsf(q) < 4e5f && q - n > tol && q - n < 1.0f - tol;
}
__device__ __forceinline__ double f64_int(float n) { return n == 0.0f ? 0.0 : f64_of(n); }

// floor(a / b): the FP32 quotient decides unless it comes within its own
// error of an integer.
__device__ __forceinline__ double f64_floor_div(double a, double b, float inv_b) {
  float n;
  if (f64_floor_sure(f32_of(a) * inv_b, n)) return f64_int(n);
  return floor(__ddiv_rn(a, b));
}

// FP64 of any FP32 value, on the integer pipe where it is a normal one.
__device__ __forceinline__ double f64_of_f32(float f) {
  const unsigned e = (__float_as_uint(f) >> 23) & 0xffu;
  return e - 1u < 254u ? f64_of(f) : (double)f;
}

// FP32 of the FP64 quotient a / b (rounded to FP64, then to FP32), from the product
// with inv_b = 1 / b, whose error is below two units in the last place: the
// division itself only where the product comes within 8 of the middle of two FP32
// values.
__device__ __forceinline__ float f32_quotient(double a, double b, double inv_b) {
  const double q = __dmul_rn(a, inv_b);
  const unsigned tail = (unsigned)__double2loint(q) & 0x1fffffffu;
  if (f64_moderate(fabs(q)) && tail - (0x10000000u - 8u) > 16u) return f32_near(q);
  return (float)__ddiv_rn(a, b);
}

// A radius ratio's place in the weight table: rows ik and ik + 1, the second's
// share ak (ik = -1: past the table's end).
__device__ __forceinline__ void table_place(double k, double kmin, double dk, double, int nk, int& ik, double& ak) {
  ik = (int)floor((k - kmin) / dk);
  ak = (k - kmin - ik * dk) / dk;
  if (ik + 1 >= nk || ik < 0) ik = -1;
}
__device__ __forceinline__ void table_place(double k, double kmin, double dk, double inv_dk, int nk, int& ik, float& ak) {
  const double x = __dsub_rn(k, kmin);
  float n;
  double nd;
  if (f64_floor_sure(f32_of(x) * f32_of(inv_dk), n)) {
    nd = f64_int(n);
  } else {
    nd = floor(__ddiv_rn(x, dk));
    n = (float)nd;
  }
  ik = (int)n;
  ak = f32_quotient(__fma_rn(-nd, dk, x), dk, inv_dk);
  if (ik + 1 >= nk || ik < 0) ik = -1;
}

// ---------------------------------------------------------------------------
// r^2(t) = x(t)^2 + y(t)^2 of a Taylor orbit c[0..9], degree 8.
// ---------------------------------------------------------------------------
constexpr int R2_N = 9;
__device__ inline void r2_poly(const double* c, double* d) {
#pragma unroll
  for (int m = 0; m < R2_N; ++m) {
    double s = 0.0;   // twice the products c_j c_{m-j}, j < m - j, then the square
#pragma unroll
    for (int j = 0; 2 * j < m; ++j) {
      if (m - j > 4) continue;
      s = __fma_rn(c[j], c[m - j], s);
      s = __fma_rn(c[5 + j], c[5 + m - j], s);
    }
    s = __dadd_rn(s, s);
    if (m % 2 == 0) {
      s = __fma_rn(c[m / 2], c[m / 2], s);
      s = __fma_rn(c[5 + m / 2], c[5 + m / 2], s);
    }
    d[m] = s;
  }
}
// `even`: the odd coefficients are zero (a circular orbit, whose r^2 is a
// polynomial of t^2: 5 FP64 instructions instead of 8).
__device__ __forceinline__ double r2_at(const double* d, bool even, double t) {
  double r = d[R2_N - 1];
  if (even) {
    const double t2 = __dmul_rn(t, t);
#pragma unroll
    for (int m = R2_N - 3; m >= 0; m -= 2) r = __fma_rn(r, t2, d[m]);
  } else {
#pragma unroll
    for (int m = R2_N - 2; m >= 0; --m) r = __fma_rn(r, t, d[m]);
  }
  return r;
}
__device__ __forceinline__ bool r2_is_even(const double* d) {
  int any = 0;
#pragma unroll
  for (int m = 1; m < R2_N; m += 2) any |= (__double2hiint(d[m]) << 1) | __double2loint(d[m]);
  return any == 0;
}

// ---------------------------------------------------------------------------
// Outer contact times for the bounding box: contact_point's bisection (bracket [0,
// +-2/vx], 1e-6 d), whose end is a fixed fraction of the bracket that the signs of z -
// (1 + k) at the midpoints choose.  The box belongs to the vector's first radius
// ratio (and a grazing or close orbit may have no contact in the bracket), so its edge
// can cut through a transit and has to be that fraction exactly.  But a sign does not
// need FP64: most are sure in FP32 within its error bound, and the others, next to
// the contact, from r^2's value in FP64 at one point and its derivatives in FP32.
// (FP64 throughout: ~1350 dependent FP64 instructions, 40 us; a sign in FP64 or in
// FP32 pairs wherever FP32 leaves a doubt: 7 or 5 us more than FP32 alone.)
// ---------------------------------------------------------------------------
static __device__ __noinline__ void contact_times_general(double k, const double* c, double& t1, double& t4) {
  t1 = contact_point(k, 1, c);
  t4 = contact_point(k, 4, c);
}

// Sign of r^2 - zt2 at t; 0 for neither, as NaN.
static __device__ __noinline__ int r2_sign(const double* d, double zt2, double t) {
  const double D = __dadd_rn(r2_at(d, false, t), -zt2);
  return D < 0.0 ? -1 : (D > 0.0 ? 1 : 0);
}

// One contact (dir -1 or 1): FP32 bisection of [0, dir T].
struct ContactBisection {
  int a, sign0;        // bracket [a, a + 1] / 2^n of T; sign at its lower end
  int n_u, a_u, s_u;   // level and state at the first sign in doubt, n_u < 0: none
};

__device__ __forceinline__ void contact_step(const float* cf, float zt2, float T, float dir, int n, ContactBisection& B) {
  const float t = dir * T * ((float)(2 * B.a + 1) * __int_as_float((126 - n) << 23)), ta = fabsf(t);
  float x = cf[4], y = cf[9], xa = fabsf(cf[4]), ya = fabsf(cf[9]);
#pragma unroll
  for (int j = 3; j >= 0; --j) {
    x = fmaf(x, t, cf[j]);
    y = fmaf(y, t, cf[5 + j]);
    xa = fmaf(xa, ta, fabsf(cf[j]));
    ya = fmaf(ya, ta, fabsf(cf[5 + j]));
  }
  // 56 roundings of the partial sums' magnitudes: coefficients (1), time (4 in t, up to
  // the fourth power), Horner (9), each twice in the squares
  const float diff = fmaf(x, x, fmaf(y, y, -zt2)), tol = 3.5e-6f * fmaf(xa, xa, fmaf(ya, ya, zt2));
  const int s = diff < 0.0f ? -1 : 1;
  if (!(fabsf(diff) > tol) && B.n_u < 0) {
    B.n_u = n;
    B.a_u = B.a;
    B.s_u = B.sign0;
  }
  const bool lower = B.sign0 * s < 0;
  B.a = 2 * B.a + (lower ? 0 : 1);
  if (!lower) B.sign0 = s;
}

// The bisection again from its first sign in doubt, with r^2 - zt2 about its end tc:
// f0 in FP64, and in x = t / tc - 1 its first two derivatives g1, g2 in FP32 and a bound of
// the rest.
__device__ __forceinline__ int contact_refine(const double* d, const float* df, double zt2, double T, float dir,
                                              int halvings, const ContactBisection& B) {
  const int mc = 2 * B.a + 1;   // tc in units of T / 2^(halvings + 1)
  const double unit = __dmul_rn(dir < 0.0f ? -T : T, __hiloint2double((1022 - halvings) << 20, 0));
  const double tc = __dmul_rn(unit, (double)mc);
  const float f0 = (float)__dadd_rn(r2_at(d, false, tc), -zt2), t = f32_of(tc), ta = fabsf(t);
  float g1 = 8.0f * df[8], g2 = 28.0f * df[8], mag = fabsf(df[8]);
#pragma unroll
  for (int m = 7; m >= 0; --m) {
    g1 = fmaf(g1, t, (float)m * df[m]);
    g2 = fmaf(g2, t, (float)(m * (m - 1) / 2) * df[m]);
    mag = fmaf(mag, ta, fabsf(df[m]));
  }
  int a = B.a_u, s0 = B.s_u;
  const float ic = 1.0f / (float)mc;
  for (int n = B.n_u; n < halvings; ++n) {
    const int g = (2 * a + 1) << (halvings - n);
    const float x = (float)(g - mc) * ic, xa = fabsf(x);
    const float L = fmaf(x, fmaf(x, g2, g1), f0);
    // g1 and g2 within 2e-5 and 6e-5, the third derivative's share within 60 of the magnitude
    const float tol = fmaf(2e-7f, fabsf(f0) + fabsf(x * g1), mag * fmaf(xa, fmaf(xa, fmaf(xa, 60.0f, 6e-5f), 2e-5f), 1e-13f));
    int s = L < 0.0f ? -1 : 1;
    if (!(fabsf(L) > tol && xa < 0.01f)) s = r2_sign(d, zt2, __dmul_rn(unit, (double)g));
    const bool lower = s0 * s < 0;
    a = 2 * a + (lower ? 0 : 1);
    if (!lower) s0 = s;
  }
  return a;
}

// c: the orbit, d: its r^2.
__device__ __forceinline__ void contact_times(double k, const double* c, const double* d, double& t1, double& t4) {
  const double zt = __dadd_rn(1.0, k), vx = fabs(c[1]);
  // brackets of at most 512 d, so that a midpoint's number is an int; k > -1
  if (!f64_moderate(vx) || vx < 1.0 / 256 || __double2hiint(zt) <= 0) {
    contact_times_general(k, c, t1, t4);
    return;
  }
  double T = f64_recip(vx);
  T = __dadd_rn(T, T);
  const double zt2 = __dmul_rn(zt, zt);
  float cf[10];
#pragma unroll
  for (int i = 0; i < 10; ++i) cf[i] = f32_near(c[i]);
  const float Tf = f32_of(T), zt2f = f32_near(zt2);
  // halvings until the bracket is no longer than 1e-6 d: at most 29
  const long long bt = __double_as_longlong(T), b6 = __double_as_longlong(1e-6), frac = (1ll << 52) - 1;
  const int halvings = max((int)((bt >> 52) - (b6 >> 52)) + ((bt & frac) > (b6 & frac) ? 1 : 0), 0);
  const double D0 = __dadd_rn(d[0], -zt2);
  const int s0 = D0 < 0.0 ? -1 : (D0 > 0.0 ? 1 : 0);
  ContactBisection A{0, s0, -1, 0, 0}, B = A;
  const bool even = r2_is_even(d);   // a circular orbit: the two are mirror images, in every rounding
  if (even) {
#pragma unroll 1
    for (int n = 0; n < halvings; ++n) contact_step(cf, zt2f, Tf, -1.0f, n, A);
  } else {
#pragma unroll 1
    for (int n = 0; n < halvings; ++n) {
      contact_step(cf, zt2f, Tf, -1.0f, n, A);
      contact_step(cf, zt2f, Tf, 1.0f, n, B);
    }
  }
  if (A.n_u >= 0 || B.n_u >= 0) {
    float df[R2_N];
#pragma unroll
    for (int m = 0; m < R2_N; ++m) df[m] = f32_near(d[m]);
    if (A.n_u >= 0) A.a = contact_refine(d, df, zt2, T, -1.0f, halvings, A);
    if (B.n_u >= 0) B.a = contact_refine(d, df, zt2, T, 1.0f, halvings, B);
  }
  if (even) B.a = A.a;
  const double unit = __dmul_rn(T, __hiloint2double((1022 - halvings) << 20, 0));
  t1 = -__dmul_rn(unit, (double)(2 * A.a + 1));
  t4 = __dmul_rn(unit, (double)(2 * B.a + 1));
}

// ---------------------------------------------------------------------------
// Constants of one radius ratio k (and of the LD table's step dg).
// ---------------------------------------------------------------------------
struct F64Disk {
  double k, k2;
  double s1;        // (1 + k)^2
  double s2q;       // (1 - k)^2 / 4
  double c1h;       // (1 - k^2) / 2
  double km;        // k^2 - 1
  double area_in;   // pi k^2
  double cg;        // 1 / ((1 + k) dg)
  double ik;        // 1 / k, for kappa0 alone (f64_disk's IK)
  float inv_k, cgf, k2f;
  float r2in, r2out;   // FP32 r^2 surely inside / outside the star
  int fast;            // 0 < k < 1: the kite form below
};

// marg: a bound of the FP32 r^2's error.
template <bool IK = false>
__device__ __forceinline__ void f64_disk(double k, double dg, float marg, F64Disk& D) {
  const double opk = __dadd_rn(1.0, k), omk = __dadd_rn(1.0, -k);
  D.k = k;
  D.k2 = __dmul_rn(k, k);
  D.s1 = __dmul_rn(opk, opk);
  D.s2q = __dmul_rn(__dmul_rn(omk, 0.25), omk);
  D.c1h = __fma_rn(__dmul_rn(k, -0.5), k, 0.5);
  D.km = __fma_rn(k, k, -1.0);
  D.area_in = __dmul_rn(PI, D.k2);
  D.cg = f64_recip(__dmul_rn(opk, dg));
  if (IK) D.ik = f64_recip(k);
  const float kf = f32_of(k);
  D.inv_k = 1.0f / kf;
  D.cgf = f32_of(D.cg);
  D.k2f = kf * kf;
  D.fast = k > 1e-6 && k < 1.0;
  D.r2in = D.fast ? (1.0f - kf) * (1.0f - kf) - marg : -INFINITY;
  D.r2out = (1.0f + kf) * (1.0f + kf) + marg;
  if (isnan(k) || !(D.r2out == D.r2out)) D.r2out = INFINITY;   // no sample is surely outside
}

// arcsin(x) - x for |x| < 2^-9.
__device__ __forceinline__ float asin_tail(float x) {
  const float x2 = x * x;
  return x * x2 * fmaf(x2, 0.075f, 1.0f / 6.0f);
}

// The limb: 1 - k < z < 1 + k, 0 < k < 1, from r2 = z^2 and iz = 1 / z.  With
// u = (1 + k)^2 - z^2 and v = (z^2 - (1 - k)^2) / 4 the kite's area is
// a = sqrt(u v), and the half-angles kappa1 (star) and kappa0 (planet) are the
// polar angles of (x1, a) and (x0, a), x1 = (1 - k^2 + z^2) / 2, x0 =
// (z^2 + k^2 - 1) / 2, whose lengths are z and k z (the circle-circle
// intersection of common.py:53-73 with its two arctangents).  An angle is the
// table's nearest angle plus the arcsine of the small rest (the sine of a
// difference), whose cubic term is FP32; the FP32 arctangent only picks the
// entry.  Returns the area A = kappa1 + k^2 kappa0 - a; kappa0 and a as asked.
struct F64Limb {
  double area, kite, kappa0;
};
template <bool KAPPA>
__device__ __forceinline__ F64Limb f64_limb(const F64Disk& D, double r2, double iz) {
  F64Limb L;
  const double u = __dadd_rn(D.s1, -r2), v = __fma_rn(0.25, r2, -D.s2q);
  const double P = __dmul_rn(u, v);
  if (__double2hiint(u) <= 0 || __double2hiint(v) <= 0 || !f64_moderate(P)) {
    // at a contact to the last place: no overlap, or the whole planet
    const bool out = __double2hiint(u) <= 0 || (__double2hiint(v) > 0 && u < v);
    L.area = out ? 0.0 : D.area_in;
    L.kite = 0.0;
    L.kappa0 = out ? 0.0 : PI;
    return L;
  }
  const double a = f64_sqrt(f64_root(P));
  const double x1 = __fma_rn(0.5, r2, D.c1h), x0 = __dadd_rn(x1, D.km);
  const float af = f32_of_pos(a);
  const float q1 = rintf(atan2f(af, f32_of_pos(x1)) * (float)ANG_PER_RAD);
  const float q0 = rintf(atan2f(af, f32_of(x0)) * (float)ANG_PER_RAD);
  const double2 t1 = __ldg(reinterpret_cast<const double2*>(ANGLES.sc[min(max((int)q1, 0), ANG_N - 1)]));
  const double2 t0 = __ldg(reinterpret_cast<const double2*>(ANGLES.sc[min(max((int)q0, 0), ANG_N - 1)]));
  const double n1 = __dmul_rn(__fma_rn(a, t1.y, -__dmul_rn(x1, t1.x)), iz);   // sin(kappa1 - th1)
  const double n0 = __dmul_rn(__fma_rn(a, t0.y, -__dmul_rn(x0, t0.x)), iz);   // k sin(kappa0 - th0)
  const double th1 = f64_of_pos(q1 * (1.0f / ANG_PER_RAD)), th0 = f64_of_pos(q0 * (1.0f / ANG_PER_RAD));
  const float e1 = asin_tail(f32_of(n1)), e0 = asin_tail(f32_of(n0) * D.inv_k);
  double A = __dadd_rn(__fma_rn(D.k2, th0, th1), -a);
  A = __dadd_rn(A, __fma_rn(D.k, n0, n1));
  L.area = __dadd_rn(A, f64_of(fmaf(D.k2f, e0, e1)));
  L.kite = a;
  if constexpr (KAPPA) L.kappa0 = __dadd_rn(__fma_rn(n0, D.ik, th0), f64_of(e0));
  else L.kappa0 = 0.0;
  return L;
}

// The LD means' lerp at separation z (common.py:225-233 with the two
// divisions folded into D.cg): the cell from the FP32 position, moved by one
// where its FP64 fraction falls outside [0, 1).
__device__ __forceinline__ void f64_ld_pos(const F64Disk& D, double z, int ng, int& i, double& fr) {
  float fi = fminf(truncf(f32_of_pos(z) * D.cgf), (float)(ng - 2));
  fr = __fma_rn(z, D.cg, -f64_of_pos(fi));
  const float ff = f32_of(fr);
  if ((ff < 0.0f && fi > 0.0f) || (ff >= 1.0f && fi < (float)(ng - 2))) {
    fi += ff < 0.0f ? -1.0f : 1.0f;
    fr = __fma_rn(z, D.cg, -f64_of_pos(fi));
  }
  i = (int)fi;
}
__device__ __forceinline__ void f64_ld_cell(const F64Disk& D, double z, const double* __restrict__ lda, int ng, int& i,
                                            double& fr, double& l0, double& dl) {
  f64_ld_pos(D, z, ng, i, fr);
  l0 = __ldg(lda + i);
  dl = __dadd_rn(__ldg(lda + i + 1), -l0);
}
__device__ __forceinline__ double f64_ld_mean(const F64Disk& D, double z, const double* __restrict__ lda, int ng) {
  int i;
  double fr, l0, dl;
  f64_ld_cell(D, z, lda, ng, i, fr, l0, dl);
  return __fma_rn(fr, dl, l0);
}

}  // namespace rr
