// The points of the plain FP64 RoadRunner path (model_full.py:75-99): fold,
// box, samples, and the walk of a warp over its tiles that the flux and the
// log-likelihood kernels share.
#pragma once
#include "rr_f64.cuh"
#include "rr_internal.h"

namespace rr {

// Data, parameters and prologue tables of one call.
struct F64Args {
  const double* times;
  const double *k, *t0, *p, *exptimes, *istar, *ldm, *orb64;
  const int32_t *lcids, *pbids, *epids, *nsamples;
  int npt, npv, nkc, ldt0, npb, nlc, ng;
  double dg;
  bool nan_istar;      // a non-finite disk integral makes in-box points NaN
  // the eclipse models: no LD tables (istar, pbids null, npb = nkc = 1); the
  // eclipse's shift and light travel time at shift[pv * ORB64]
  const double* shift;
  double pad0 = 0.003; // box padding beyond the contacts and the exposure
  float pad0f = 0.00300001f;
  int ns0;             // for null nsamples / exptimes
  double ex0;
};

// Zero epoch of a light curve: t0, or ((t0 + shift) + light travel time).
__device__ __forceinline__ double f64_t0(const F64Args& A, int pv, int lc) {
  const double t0 = A.t0[(size_t)pv * A.ldt0 + (A.epids ? A.epids[lc] : 0)];
  if (!A.shift) return t0;
  const double* s = A.shift + (size_t)pv * ORB64;
  return __dadd_rn(__dadd_rn(t0, s[0]), s[1]);
}

// Phase fold of the reference (model_full.py:84-86) with its rounding: the
// epoch's conjunction t0 + epoch p, epoch = floor(((t - t0) + p/2) / p).
__device__ __forceinline__ double f64_epoch(double t, double t0, double p, float inv_p) {
  return f64_floor_div(__dadd_rn(__dsub_rn(t, t0), __dmul_rn(0.5, p)), p, inv_p);
}
__device__ __forceinline__ double f64_conjunction(double t, double t0, double p, float inv_p) {
  return __dadd_rn(t0, __dmul_rn(f64_epoch(t, t0, p, inv_p), p));
}

// Constants of one parameter vector: r^2(t) in FP64 and FP32.
struct F64Orbit {
  double d[R2_N];
  float df[R2_N];
  double t1, t4;       // contacts
  float t1f, t4f;      // rounded outwards
  int even;
  int finite;          // every coefficient is
};

__device__ __forceinline__ void f64_orbit(const double* o, F64Orbit& P) {
  bool fin = true;
#pragma unroll
  for (int m = 0; m < R2_N; ++m) {
    P.d[m] = o[ORB64_R2 + m];
    P.df[m] = f32_of(P.d[m]);
    fin = fin && f64_finite(P.d[m]);
  }
  P.finite = fin;
  P.t1 = o[10];
  P.t4 = o[11];
  P.t1f = f32_up(P.t1);
  P.t4f = f32_up(P.t4);
  P.even = r2_is_even(P.d);
}

// Constants of one light curve of one pv.
struct F64Lc {
  F64Disk disk;
  double w;            // 1 / (istar nsamples); NaN for a non-finite istar (A.nan_istar)
  double ex, step;     // exposure time and its share of one sample
  float lo, hi;        // box, its edges rounded outwards
  int hlo, hhi;        // upper words of FP64 magnitudes surely inside them
  int ns, pb;
};

// Box: the contact times padded by 0.003 d + exposure (model_full.py:87-89), the
// edges rounded outwards to FP32 (by less than 5e-7 of its width).
__device__ __forceinline__ void f64_box_edges(const F64Args& A, const F64Orbit& P, double ex, float& lo, float& hi) {
  const float pad = __fadd_ru(A.pad0f, f32_up(ex));
  lo = __fsub_rd(P.t1f, pad);
  hi = __fadd_ru(P.t4f, pad);
}

// Is a point that the FP32 edges put in the box there by the FP64 ones?  They decide
// close to an edge: the flux need not be 1 on its inside (several radius ratios with
// the first one's box, contacts that are not in the bisection's bracket).  A walk
// queues points by the FP32 edges and its flush asks this of each.
static __device__ __noinline__ bool f64_in_box_exact(const F64Args& A, const F64Orbit& P, double ex, double tc) {
  const double pad = __dadd_rn(A.pad0, ex);
  return __dsub_rn(P.t1, pad) <= tc && tc <= __dadd_rn(P.t4, pad);
}
__device__ __forceinline__ bool f64_in_box(const F64Args& A, const F64Orbit& P, const F64Lc& R, double tc) {
  const int h = __double2hiint(tc);
  return (h & 0x7fffffff) < (h < 0 ? R.hlo : R.hhi) || f64_in_box_exact(A, P, R.ex, tc);
}

template <bool IK = false>
__device__ __forceinline__ void f64_lc(const F64Args& A, int pv, int lc, const F64Orbit& P, F64Lc& R) {
  R.pb = A.pbids ? A.pbids[lc] : 0;
  R.ns = max(A.nsamples ? A.nsamples[lc] : A.ns0, 0);
  R.ex = A.exptimes ? A.exptimes[lc] : A.ex0;
  R.step = R.ns > 1 ? __ddiv_rn(R.ex, (double)R.ns) : R.ex;
  const float ex = f32_up(R.ex);
  f64_box_edges(A, P, R.ex, R.lo, R.hi);
  // an upper word's last place is 5e-7 to 1e-6 of the value, the edges' rounding 5e-7
  R.hlo = (int)((__float_as_uint(R.lo) & 0x7fffffffu) >> 3) + F64_BIAS - 2;
  R.hhi = (int)((__float_as_uint(R.hi) & 0x7fffffffu) >> 3) + F64_BIAS - 2;
  // bound of the FP32 r^2's error at any sample: 16 roundings of the largest partial sums
  const float tb = fmaxf(fabsf(R.lo), fabsf(R.hi)) + ex;
  float sum = fabsf(P.df[R2_N - 1]);
#pragma unroll
  for (int m = R2_N - 2; m >= 0; --m) sum = fmaf(sum, tb, fabsf(P.df[m]));
  f64_disk<IK>(A.k[(size_t)pv * A.nkc + (A.nkc == A.npb ? R.pb : 0)], A.dg, fmaf(4e-6f, sum, 2e-6f), R.disk);
  // f32_of knows no NaN: with a coefficient that is not finite (a NaN inclination,
  // say) no sample is sure, and general() gives the reference's NaN
  if (!P.finite) {
    R.disk.r2out = INFINITY;
    R.disk.r2in = -INFINITY;
  }
  const double is = A.istar ? A.istar[(size_t)pv * A.npb + R.pb] : 1.0;
  R.w = isfinite(is) || !A.nan_istar ? f64_recip(R.ns == 1 ? is : __dmul_rn(is, (double)R.ns)) : CUDART_NAN;
}

// Time of sample s (0 based) from conjunction: tc + ex ((s + 1/2) / ns - 1/2).
__device__ __forceinline__ double f64_sample_time(const F64Lc& R, double tc, int s) {
  if (R.ns == 1) return tc;
  return __fma_rn(f64_of_pos((float)s + 0.5f), R.step, __fma_rn(-0.5, R.ex, tc));
}

// Class of the sample at t from the FP32 r^2: 0 surely outside the star, 1
// surely inside (the planet's whole disk), 2 the limb or unsure.
__device__ __forceinline__ int f64_class(const F64Lc& R, const F64Orbit& P, double t) {
  const float tf = f32_of(t);
  float r = P.df[R2_N - 1];
#pragma unroll
  for (int m = R2_N - 2; m >= 0; --m) r = fmaf(r, tf, P.df[m]);
  return r > R.disk.r2out ? 0 : (r < R.disk.r2in ? 1 : 2);
}

// The terms that a point sums over its samples, and its value from the sum:
// the flux 1 - sum_s I A / (ns istar) (F64Transit) and the visible planet area
// sum_s (pi k^2 - A) / ns (F64Eclipse).  general(): a sample by the reference's
// own expressions, for the separations and radius ratios that the kernels'
// forms leave out: z = 0, k <= 0, k >= 1, NaN.
struct F64Transit {
  const double *o, *lda;
  int ng;
  double dg;

  __device__ __forceinline__ double none(const F64Lc&) const { return 0.0; }
  __device__ __forceinline__ double inner(const F64Lc& R, const F64Orbit& P, double t) const {
    const double r2 = r2_at(P.d, P.even, t);
    if (!f64_moderate(r2)) return general(*this, R.disk.k, t);
    return __dmul_rn(f64_ld_mean(R.disk, f64_sqrt(f64_root(r2)), lda, ng), R.disk.area_in);
  }
  __device__ __forceinline__ double limb(const F64Lc& R, const F64Orbit& P, double t) const {
    const double r2 = r2_at(P.d, P.even, t);
    if (!R.disk.fast || !f64_moderate(r2)) return general(*this, R.disk.k, t);
    const F64Root q = f64_root(r2);
    const double ip = f64_ld_mean(R.disk, f64_sqrt(q), lda, ng);
    return __dmul_rn(ip, f64_limb<false>(R.disk, r2, f64_rsqrt(q)).area);
  }
  __device__ __forceinline__ double value(const F64Lc& R, double D) const { return __fma_rn(-D, R.w, 1.0); }

  static __device__ __noinline__ double general(const F64Transit& T, double k, double t) {
    double c[10];
    for (int i = 0; i < 10; ++i) c[i] = T.o[i];
    const double z = sep_c_f64(t, c);
    double kap;   // model_full.py:93-98
    return interp_ldm_f64(z / (1.0 + k), T.dg, T.lda, T.ng) * ccia_star<double>(k, z, kap);
  }
};

struct F64Eclipse {
  const double* o;

  __device__ __forceinline__ double none(const F64Lc& R) const { return R.disk.area_in; }
  __device__ __forceinline__ double inner(const F64Lc&, const F64Orbit&, double) const { return 0.0; }
  __device__ __forceinline__ double limb(const F64Lc& R, const F64Orbit& P, double t) const {
    const double r2 = r2_at(P.d, P.even, t);
    if (!R.disk.fast || !f64_moderate(r2)) return __dadd_rn(R.disk.area_in, -general(o, R.disk.k, t));
    return __dadd_rn(R.disk.area_in, -f64_limb<false>(R.disk, r2, f64_rsqrt(f64_root(r2))).area);
  }
  __device__ __forceinline__ double value(const F64Lc& R, double D) const { return R.ns == 1 ? D : __dmul_rn(D, R.w); }

  static __device__ __noinline__ double general(const double* o, double k, double t) {
    double c[10];
    for (int i = 0; i < 10; ++i) c[i] = o[i];
    double kap;
    return ccia_star<double>(k, sep_c_f64(t, c), kap);
  }
};

// The value of one in-box point at tc from conjunction by one thread: the same
// operations in the same order as f64_sums'.
template <class Terms>
__device__ __forceinline__ double f64_point_value(const F64Lc& R, const F64Orbit& P, const Terms& T, double tc) {
  double D = 0.0;
  for (int s = 0; s < R.ns; ++s) {
    const double t = f64_sample_time(R, tc, s);
    const int cls = f64_class(R, P, t);
    const double term = cls == 0 ? T.none(R) : (cls == 1 ? T.inner(R, P, t) : T.limb(R, P, t));
    D = s == 0 ? term : __dadd_rn(D, term);
  }
  return T.value(R, D);
}

constexpr int F64_Q = 256;        // points and (point, sample) pairs a warp holds
constexpr int F64_LC_SMEM = 32;   // light-curve constants staged per block
struct F64Queue {
  double tc[F64_Q];
  double term[F64_Q];
  int pt[F64_Q];
  unsigned short list[F64_Q];
};

__device__ __forceinline__ void f64_box(const F64Args& A, const F64Orbit& P, int lc, const F64Lc* recs, float& lo,
                                        float& hi) {
  if (lc < F64_LC_SMEM) {
    lo = recs[lc].lo;
    hi = recs[lc].hi;
  } else {
    f64_box_edges(A, P, A.exptimes[lc], lo, hi);
  }
}

// The terms of the samples [s0, s0 + ns) of the ni items from i0 on: each pair
// (item, sample) classified in FP32, then the inner and the limb pairs as full
// warps.  inner(f, it, s) and limb(f, it, s) do one pair (f = it ns + s - s0, at
// most F64_Q pairs), none(f) a pair outside the star.
template <class Inner, class Limb, class None>
__device__ __forceinline__ void f64_pairs(const F64Lc& R, const F64Orbit& P, F64Queue& Q, int i0, int ni, int s0,
                                          int ns, Inner inner, Limb limb, None none) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int np = ni * ns;
  const float ins = 1.0f / (float)ns;
  int nin = 0, nlimb = 0;   // pairs on the inner list (from the front) and the limb list (from the back)
  for (int f0 = 0; f0 < np; f0 += 32) {
    const int f = f0 + lane;
    int cls = 0;
    if (f < np) {
      const int it = (ns == 1) ? f : (int)(((float)f + 0.5f) * ins);
      cls = f64_class(R, P, f64_sample_time(R, Q.tc[i0 + it], s0 + f - it * ns));
      if (cls == 0) none(f);
    }
    const unsigned m1 = __ballot_sync(FULL, cls == 1), m2 = __ballot_sync(FULL, cls == 2);
    if (cls == 1) Q.list[nin + __popc(m1 & below)] = (unsigned short)f;
    if (cls == 2) Q.list[F64_Q - 1 - nlimb - __popc(m2 & below)] = (unsigned short)f;
    nin += __popc(m1);
    nlimb += __popc(m2);
  }
  __syncwarp();
  for (int j = lane; j < nin; j += 32) {
    const int f = Q.list[j], it = (ns == 1) ? f : (int)(((float)f + 0.5f) * ins);
    inner(f, it, s0 + f - it * ns);
  }
  for (int j = lane; j < nlimb; j += 32) {
    const int f = Q.list[F64_Q - 1 - j], it = (ns == 1) ? f : (int)(((float)f + 0.5f) * ins);
    limb(f, it, s0 + f - it * ns);
  }
  __syncwarp();
}

// The sums D of the n queued points' terms, all of the light curve R:
// point(i, D) is called once per point by one lane, chunk(i0, ni) by the warp
// after the points [i0, i0 + ni).
template <class Terms, class Point, class Chunk>
__device__ __forceinline__ void f64_sums(const F64Lc& R, const F64Orbit& P, const Terms& T, F64Queue& Q, int n,
                                         Point point, Chunk chunk) {
  const int lane = threadIdx.x & 31;
  // R, P and Q arrive as generic pointers (the callers are not inlined)
  __builtin_assume(__isShared(&R));
  __builtin_assume(__isShared(&P));
  __builtin_assume(__isShared(&Q));
  __syncwarp();
  const int sc = min(max(R.ns, 1), F64_Q);   // samples and points of a chunk of pairs
  const int ic = F64_Q / sc;
  for (int i0 = 0; i0 < n; i0 += ic) {
    const int ni = min(ic, n - i0);
    double D = 0.0;
    for (int s0 = 0; s0 < max(R.ns, 1); s0 += sc) {
      const int ns = min(sc, R.ns - s0);
      f64_pairs(R, P, Q, i0, ni, s0, ns,
                [&](int f, int it, int s) { Q.term[f] = T.inner(R, P, f64_sample_time(R, Q.tc[i0 + it], s)); },
                [&](int f, int it, int s) { Q.term[f] = T.limb(R, P, f64_sample_time(R, Q.tc[i0 + it], s)); },
                [&](int f) { Q.term[f] = T.none(R); });
      if (s0 + ns == R.ns) {
        for (int i = lane; i < ni; i += 32) {
          if (s0 == 0) D = ns > 0 ? Q.term[i * ns] : 0.0;
          for (int s = s0 == 0 ? 1 : 0; s < ns; ++s) D = __dadd_rn(D, Q.term[i * ns + s]);
          point(i0 + i, D);
        }
      } else if (lane == 0) {
        // more samples than a chunk holds: one point at a time, its sum carried by lane 0
        for (int s = 0; s < ns; ++s) D = s0 + s == 0 ? Q.term[0] : __dadd_rn(D, Q.term[s]);
      }
      __syncwarp();
    }
    chunk(i0, ni);
  }
}

// The slots q0 to q1 of a tile of several light curves: the in-box points of one light
// curve after another to the queue, so that its flushes take what the whole tile has
// of a light curve.  The adjoint's way, whose flushes and reductions are dear: points of
// four light curves interleaved (256 x 19,700) 1500 us slot by slot, 590 so.  The other
// kernels gain there too (flux of 512 490 -> 316 us), but the code costs them 7 %
// everywhere else (flux of 8192 x 19,700 517 -> 555 us).
template <class Sink>
__device__ __forceinline__ void f64_mixed_tile(const F64Args& A, int pv, const F64Orbit& P, const F64Lc* recs,
                                               F64Queue& Q, const Sink& sink, double p, float inv_p, int p0, int q0,
                                               int q1, int& n, int& qlc) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int lc[4];
  double tc[4];
  unsigned pend = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int pt = p0 + 32 * q + lane;
    lc[q] = -1;
    tc[q] = 0.0;
    if (q < q0 || q >= q1 || pt >= A.npt) continue;
    lc[q] = A.lcids[pt];
    float lo, hi;
    f64_box(A, P, lc[q], recs, lo, hi);
    const double t = __ldg(A.times + pt);
    tc[q] = __dsub_rn(t, f64_conjunction(t, f64_t0(A, pv, lc[q]), p, inv_p));
    const float tf = f32_of(tc[q]);
    if (lo <= tf && tf <= hi) pend |= 1u << q;
    else sink.outside(pt);
  }
  for (unsigned lanes; (lanes = __ballot_sync(FULL, pend != 0));) {
    int first = lc[3];
#pragma unroll
    for (int q = 2; q >= 0; --q) first = pend >> q & 1u ? lc[q] : first;
    const int kl = __shfl_sync(FULL, first, __ffs(lanes) - 1);
    if (n > 0 && (kl != qlc || n > F64_Q - TIME_TILE)) {
      sink.flush(qlc, n);
      n = 0;
    }
    qlc = kl;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool in = (pend >> q & 1u) && lc[q] == kl;
      const unsigned mem = __ballot_sync(FULL, in);
      if (in) {
        const int at = n + __popc(mem & ((1u << lane) - 1u));
        Q.tc[at] = tc[q];
        Q.pt[at] = p0 + 32 * q + lane;
        pend &= ~(1u << q);
      }
      n += __popc(mem);
    }
  }
}

// A warp's walk over its share of one pv's row: slots / 4 tiles from the
// block's first, or, in launches too small to fill the GPU, `slots` < 4 of one
// tile's four 32-point slots.  sink.tile(p0, q0, q1) gets a tile (slots q0 to
// q1) without in-box points, sink.outside(pt) a point out of the box,
// sink.flush(lc, n) the queued points.  Sink::BY_LIGHT_CURVE: f64_mixed_tile for tiles of
// several light curves.
template <class Sink>
__device__ __forceinline__ void f64_walk(const F64Args& A, int pv, const double* __restrict__ tiles64, int slots,
                                         bool valid, const F64Orbit& P, const F64Lc* recs, F64Queue& Q, const Sink& sink) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int ntiles = (A.npt + TIME_TILE - 1) / TIME_TILE;
  const int slot0 = blockIdx.x * slots;
  const int tb0 = slot0 >> 2, tb1 = min(ntiles, tb0 + max(slots >> 2, 1));
  const int q0 = slot0 & 3, q1 = slots < 4 ? q0 + slots : 4;
  const double p = A.p[pv], hp = __dmul_rn(0.5, p);
  const float inv_p = 1.0f / f32_of(p);
  int n = 0, qlc = -1;   // queued points and their light curve
  unsigned long long mixed = 0;   // tiles of several light curves, from tb0 on: at most F64_TILES
  for (int tbase = tb0; tbase < tb1; tbase += 32) {
    const int jn = min(32, tb1 - tbase);
    bool cull = !valid, tileone = false;   // tileone: one light curve and one epoch
    double conj = 0.0;
    int tlc = -1;
    float blo = 0.0f, bhi = 0.0f;
    if (valid && lane < jn) {
      const double2 tm = __ldg(reinterpret_cast<const double2*>(tiles64 + 4 * (size_t)(tbase + lane)));
      tlc = (int)f32_of(__ldg(tiles64 + 4 * (size_t)(tbase + lane) + 2));
      if (tlc >= 0) {
        const double t0 = f64_t0(A, pv, tlc);
        f64_box(A, P, tlc, recs, blo, bhi);
        // the epoch of both ends: in FP32 where that leaves no doubt
        const double h0 = __dadd_rn(__dsub_rn(tm.x, t0), hp);
        const float span = f32_of(__dsub_rn(tm.y, tm.x)) * 1.000001f;
        const float qe = f32_of(h0) * inv_p;
        float n0, n1;
        const bool sure0 = f64_floor_sure(qe, n0), sure1 = f64_floor_sure(fmaf(span, inv_p, qe), n1);
        const double e0 = sure0 ? f64_int(n0) : floor(__ddiv_rn(h0, p));
        conj = __dadd_rn(t0, __dmul_rn(e0, p));
        const float tc0 = f32_of(__dsub_rn(tm.x, conj));
        if (sure0 && sure1 && n0 == n1) {
          tileone = true;
          cull = tc0 > bhi || tc0 + span + 1e-6f * (fabsf(tc0) + span) < blo;
        } else {
          // an epoch or more begins inside the tile: its first points end at
          // +p/2, its last ones start at -p/2
          const double e1 = sure1 ? f64_int(n1) : floor(__ddiv_rn(__dadd_rn(__dsub_rn(tm.y, t0), hp), p));
          const float tc1 = f32_of(__dsub_rn(tm.y, __dadd_rn(t0, __dmul_rn(e1, p))));
          tileone = e0 == e1;
          cull = tileone ? (tc0 > bhi || tc1 < blo) : (e1 == e0 + 1.0 && tc0 > bhi && tc1 < blo);
        }
      }
    }
    const unsigned jmask = jn == 32 ? FULL : (1u << jn) - 1u;
    const unsigned cmask = __ballot_sync(FULL, cull) & jmask;
    unsigned mmask = 0;
    if constexpr (Sink::BY_LIGHT_CURVE) {   // after the others
      mmask = __ballot_sync(FULL, valid && tlc < 0) & jmask;
      mixed |= (unsigned long long)mmask << (tbase - tb0);
    }
    for (unsigned m = cmask; m; m &= m - 1u) sink.tile((tbase + __ffs(m) - 1) * TIME_TILE, q0, q1);
    for (unsigned m = ~(cmask | mmask) & jmask; m; m &= m - 1u) {
      const int j = __ffs(m) - 1;
      const int p0 = (tbase + j) * TIME_TILE;
      const int lc = __shfl_sync(FULL, tlc, j);
      const double cj = __shfl_sync(FULL, conj, j);
      const float lo = __shfl_sync(FULL, blo, j), hi = __shfl_sync(FULL, bhi, j);
      const bool one = __shfl_sync(FULL, (int)tileone, j) != 0;
      for (int q = q0; q < q1; ++q) {
        const int pt = p0 + 32 * q + lane;
        bool in = false;
        double tc = 0.0;
        int l = lc;
        if (pt < A.npt) {
          const double t = __ldg(A.times + pt);
          float plo = lo, phi = hi;
          if (one) {
            tc = __dsub_rn(t, cj);
          } else {
            if (lc < 0) {
              l = A.lcids[pt];
              f64_box(A, P, l, recs, plo, phi);
            }
            tc = __dsub_rn(t, f64_conjunction(t, f64_t0(A, pv, l), p, inv_p));
          }
          const float tf = f32_of(tc);
          in = plo <= tf && tf <= phi;
          if (!in) sink.outside(pt);
        }
        // the in-box points to the queue, one light curve at a time
        for (unsigned pend = __ballot_sync(FULL, in); pend;) {
          const int kl = __shfl_sync(FULL, l, __ffs(pend) - 1);
          const unsigned mem = __ballot_sync(FULL, l == kl) & pend;
          if (n > 0 && (kl != qlc || n > F64_Q - 32)) {
            sink.flush(qlc, n);
            n = 0;
          }
          qlc = kl;
          if (mem >> lane & 1u) {
            const int at = n + __popc(mem & ((1u << lane) - 1u));
            Q.tc[at] = tc;
            Q.pt[at] = pt;
          }
          n += __popc(mem);
          pend &= ~mem;
        }
      }
    }
  }
  if constexpr (Sink::BY_LIGHT_CURVE)
    for (; mixed; mixed &= mixed - 1ull)
      f64_mixed_tile(A, pv, P, recs, Q, sink, p, inv_p, (tb0 + __ffsll(mixed) - 1) * TIME_TILE, q0, q1, n, qlc);
  if (n > 0) sink.flush(qlc, n);
}

// The value v at slots q0 to q1 of the tile at p0 (vec: 16-byte aligned rows).
__device__ __forceinline__ void f64_fill_tile(double* row, int npt, int p0, int q0, int q1, double v, bool vec) {
  const int lane = threadIdx.x & 31;
  if (vec && q1 - q0 == 4 && p0 + TIME_TILE <= npt) {
    double2* q = reinterpret_cast<double2*>(row + p0) + 2 * lane;
    __stcs(q, make_double2(v, v));
    __stcs(q + 1, make_double2(v, v));
  } else {
    for (int q = q0; q < q1; ++q)
      if (p0 + 32 * q + lane < npt) row[p0 + 32 * q + lane] = v;
  }
}

// Launch shape of a walk: slots of 32 points per warp.  Below two rounds of 16
// warps per SM single slots or pairs, so that a small call's chain of FP64
// operations is as short as it can be (77 x 1501: 329 us with 32 tiles a warp,
// 14 us).  Above, whole tiles, evenly over the row's warps: up to 64 while that
// leaves four rounds (flux of 8192 x 19,700: 515 us with at most 32 tiles a
// warp, 491 with 64, 493 with 96), and down to 8 while that leaves one, since a
// warp's own cost (constants, cull test, partly filled last lists) is that of
// about two tiles (log-likelihood of 1500 x 2999: 156 us with 3, 142 with 8).
constexpr int F64_TILES = 64;
inline int f64_slots(int npt, int npv, int sms) {
  const int ntiles = (npt + TIME_TILE - 1) / TIME_TILE;
  const long long tiles = (long long)ntiles * npv, round = 16LL * sms;
  if (tiles < round) return 4 * tiles <= round ? 1 : (4 * tiles <= 2 * round ? 2 : 4);
  long long want = tiles / (4 * round);
  const long long least = tiles / round < 8 ? tiles / round : 8;
  want = want < least ? least : (want > F64_TILES ? F64_TILES : want);
  const int nblk = (int)((ntiles + want - 1) / want);
  return 4 * ((ntiles + nblk - 1) / nblk);
}
inline int f64_warps(int npt, int slots) {
  return (4 * ((npt + TIME_TILE - 1) / TIME_TILE) + slots - 1) / slots;
}

}  // namespace rr
