// Forward-mode dual numbers with one derivative direction, for the derivatives
// of the orbit's Taylor coefficients with respect to (p, a, i, e, w) in the
// adjoint prologue, a thread per direction.
#pragma once
#include <cuda_runtime.h>

namespace rr {

struct Dual {
  double v, d;
};

__device__ inline Dual dconst(double v) { return {v, 0.0}; }
__device__ inline Dual dvar(double v, bool on) { return {v, on ? 1.0 : 0.0}; }
__device__ inline Dual operator+(const Dual& a, const Dual& b) {
  Dual r; r.v = a.v + b.v;
  r.d = a.d + b.d;
  return r;
}
__device__ inline Dual operator-(const Dual& a, const Dual& b) {
  Dual r; r.v = a.v - b.v;
  r.d = a.d - b.d;
  return r;
}
__device__ inline Dual operator-(const Dual& a) {
  Dual r; r.v = -a.v;
  r.d = -a.d;
  return r;
}
__device__ inline Dual operator*(const Dual& a, const Dual& b) {
  Dual r; r.v = a.v * b.v;
  r.d = a.d * b.v + a.v * b.d;
  return r;
}
__device__ inline Dual operator*(double s, const Dual& a) {
  Dual r; r.v = s * a.v;
  r.d = s * a.d;
  return r;
}
__device__ inline Dual operator/(const Dual& a, const Dual& b) {
  Dual r; r.v = a.v / b.v;
  const double ib = 1.0 / b.v;
  r.d = (a.d - r.v * b.d) * ib;
  return r;
}
__device__ inline Dual operator/(const Dual& a, double s) {
  Dual r; r.v = a.v / s;
  r.d = a.d / s;
  return r;
}
__device__ inline Dual dsqrt(const Dual& a) {
  Dual r; r.v = sqrt(a.v);
  const double h = 0.5 / r.v;
  r.d = a.d * h;
  return r;
}
__device__ inline void dsincos(const Dual& a, Dual& s, Dual& c) {
  sincos(a.v, &s.v, &c.v);
  s.d = a.d * c.v;
  c.d = a.d * -s.v;
}

// solve2d_conj (rr_device.cuh) on dual numbers: c[0..9] with their
// derivatives with respect to the j-th of (p, a, i, e, w).
__device__ inline void solve2d_conj_dual(double p_, double a_, double inc_, double e_, double w_, int j, Dual* c) {
  const Dual p = dvar(p_, j == 0), a = dvar(a_, j == 1), inc = dvar(inc_, j == 2), e = dvar(e_, j == 3),
             w = dvar(w_, j == 4);
  const Dual one = dconst(1.0);
  const Dual n = dconst(2.0 * 3.141592653589793238462643383279502884) / p;
  const Dual se = dsqrt(one - e * e);
  Dual sf, cf, si, ci;
  dsincos(w, cf, sf);
  dsincos(inc, si, ci);
  const Dual r = a * (one - e * e) / (one + e * cf);
  const Dual vr = n * a * e * sf / se;
  const Dual vt = n * a * (one + e * cf) / se;
  const Dual P0x = dconst(0.0), P0y = r;
  const Dual P1x = -vt, P1y = vr;
  const Dual mu = n * n * a * a * a;
  const double alpha = -1.5;
  const Dual q0 = P0x * P0x + P0y * P0y;
  const Dual q1 = 2.0 * (P0x * P1x + P0y * P1y);
  const Dual s0 = one / (q0 * dsqrt(q0));
  const Dual P2x = -(mu * s0 * P0x) / 2.0, P2y = -(mu * s0 * P0y) / 2.0;
  const Dual s1 = alpha * (q1 * s0 / q0);
  const Dual P3x = -(mu * (s0 * P1x + s1 * P0x)) / 6.0;
  const Dual P3y = -(mu * (s0 * P1y + s1 * P0y)) / 6.0;
  const Dual q2 = 2.0 * (P0x * P2x + P0y * P2y) + (P1x * P1x + P1y * P1y);
  const Dual s2 = ((alpha - 1.0) * (q1 * s1) + (2.0 * alpha) * (q2 * s0)) / (2.0 * q0);
  const Dual P4x = -(mu * (s0 * P2x + s1 * P1x + s2 * P0x)) / 12.0;
  const Dual P4y = -(mu * (s0 * P2y + s1 * P1y + s2 * P0y)) / 12.0;
  c[0] = -P0x; c[1] = -P1x; c[2] = -P2x; c[3] = -P3x; c[4] = -P4x;
  c[5] = -(ci * P0y); c[6] = -(ci * P1y); c[7] = -(ci * P2y); c[8] = -(ci * P3y); c[9] = -(ci * P4y);
}

}  // namespace rr
