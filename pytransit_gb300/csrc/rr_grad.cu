// Gaussian log-likelihood of the RoadRunner model and its adjoint:
//   lnL[pv] = sum_i -log(sigma_i) - log(2 pi)/2 - ((o_i - m_i(theta_pv)) / sigma_i)^2 / 2
// (pytransit/lpf/loglikelihood/wnloglikelihood.py:23-35; lpf.py:51-66), fused
// with the model so the flux is never stored, and d lnL / d theta for
// theta = (k, t0, p, a, i, e, w, ldc), recomputing z, the table interpolation
// and the area per sample in the backward pass.
//
// The derivative is that of the discretised model: the k-interpolation of the
// weight table, the g-interpolation of the LD means, the kite area, the
// coefficient dependence of the LD profile and of its disk integral, and the
// orbit's Taylor coefficients (forward-mode duals through the jet solve).  The
// bounding box and the epoch count are piecewise constant and contribute no
// derivative.  Out-of-box points (F = 1 exactly) only enter through the
// pv-independent constant sum_i -log sigma_i - log(2 pi)/2 - (o_i - 1)^2/(2 sigma_i^2).
#include <algorithm>
#include <cmath>

#include "rr_device.cuh"
#include "rr_dual.cuh"
#include "rr_f64_points.cuh"
#include "rr_internal.h"

namespace rr {

constexpr int MAX_GRAD_PAR = 4;    // LD coefficients per passband in the adjoint
constexpr int MAX_NGRAD = 64;      // nkc + nep + 5 + npb * npar
constexpr size_t GLD_SMEM = 64 * 1024;   // weight slabs staged by the LD-table derivatives
constexpr int GLC_SMEM = 64;       // light-curve records staged in shared memory (split)

// Slots of one point's gradient contribution: destinations vary per point.
enum GSlot { GS_LNL = 0, GS_KK, GS_KW, GS_T0, GS_P, GS_A, GS_I, GS_E, GS_W, GS_C0, GS_NSLOT = GS_C0 + MAX_GRAD_PAR };

// ---------------------------------------------------------------------------
// Prologue 1: derivatives of the orbit's Taylor coefficients, one thread per
// (pv, j): dc[pv][j][m] = d c_m / d theta_j, theta = (p, a, i, e, w).  Bound by
// the thread's chain of FP64 instructions: with the five directions in one
// thread 37 us for 4096 pv, 24.8 us so.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void grad_orbit_kernel(const double* __restrict__ p, const double* __restrict__ a,
                                  const double* __restrict__ inc, const double* __restrict__ e,
                                  const double* __restrict__ w, int npv, R* __restrict__ dc) {
  overlap_next();
  const int i = blockIdx.x * blockDim.x + threadIdx.x, pv = i / 5;
  if (pv >= npv) return;
  Dual c[10];
  solve2d_conj_dual(p[pv], a[pv], inc[pv], e[pv], w[pv], i % 5, c);
  R* o = dc + (size_t)i * 10;
  for (int m = 0; m < 10; ++m) o[m] = (R)c[m].d;
}

// Row g of the derivatives from the 2D table at k (and at k +- h for the k
// derivative), FP64 rows; dl: [npar][64].  Not inlined: the rows of the 3D table,
// the common case, keep their registers.
template <typename R>
static __device__ __noinline__ void grad_ld_row_2d(double k, int g, int ng, int nz, int npar,
                                                   const double* __restrict__ ze, const R* l, const R* dl, R* out) {
  const double gstep = (1.0 - 1e-7) / (double)(ng - 1);
  double gg = (g == ng - 1) ? (1.0 - 1e-7) : (double)g * gstep;
  const double h = 1e-6 * fmax(k, 1e-3);
  double res[3][1 + MAX_GRAD_PAR];
  for (int v = 0; v < 3; ++v) {
    const double kv = k + (v - 1) * h;
    const double bb = gg * (1.0 + kv);
    double a0 = cci_acos(ze[0], kv, bb), s = a0;
    double acc[1 + MAX_GRAD_PAR];
    acc[0] = a0 * (double)l[0];
    for (int j = 0; j < npar; ++j) acc[1 + j] = a0 * (double)dl[j * 64];
    for (int z = 1; z < nz; ++z) {
      const double a1 = cci_acos(ze[z], kv, bb), wz = a1 - a0;
      a0 = a1;
      s += wz;
      acc[0] += wz * (double)l[z];
      for (int j = 0; j < npar; ++j) acc[1 + j] += wz * (double)dl[j * 64 + z];
    }
    for (int j = 0; j <= npar; ++j) res[v][j] = acc[j] / s;
  }
  out[g] = (R)((res[2][0] - res[0][0]) / (2.0 * h));
  for (int j = 0; j < npar; ++j) out[(size_t)(1 + j) * ng + g] = (R)res[1][1 + j];
}

// ---------------------------------------------------------------------------
// Prologue 2: LD-table derivatives, one block per (pv, pb):
//   dL/dk[g]   = (W[ik+1] @ ldp - W[ik] @ ldp)[g] / dk   (3D table), or a
//                central difference of the 2D table at k +- h;
//   dL/dc_j[g] = Wk @ (d ldp / d c_j), Wk the table the forward pass uses;
//   d istar / d c_j analytic, or the 200-point trapezoid of z dI/dc_j.
// FP32 is bound by the reads of W: a thread's rows element by element from global
// memory (95.5 us for 4096 pv, ng = 100, nz = 40), or, where rows are whole 16-byte
// words and the two slabs fit (STAGE), staged by words in shared memory (65.3 us;
// 51.2 with the FP64 divisions that place k in the table done by one warp; 41.2
// without divisions and with the 2D table's rows, which took registers and local
// memory, in a function of their own).
// tab layout per (pv, pb): [dL/dk (ng)][dL/dc_0 (ng)]...[dL/dc_{npar-1} (ng)],
// dis layout: [d istar/dc_j] (npar).
// ---------------------------------------------------------------------------
template <typename R, bool STAGE>
__global__ void __launch_bounds__(128)
grad_ld_kernel(int law, const double* __restrict__ ldc, int npb, int npar, const double* __restrict__ mu,
               int nz, const R* __restrict__ ldp, const double* __restrict__ kw, int kw_stride,
               const R* __restrict__ W, int nk, int ng, double dk, double inv_dk, double kmin, double kmax,
               const double* __restrict__ ze, R* __restrict__ tab, R* __restrict__ dis) {
  extern __shared__ __align__(16) unsigned char gld_smem[];   // STAGE: the slabs of W at ik and ik + 1
  __shared__ __align__(16) R l[64];
  __shared__ __align__(16) R dl[MAX_GRAD_PAR][64];
  __shared__ R pvs[16];
  const int pv = blockIdx.x, pb = blockIdx.y;
  const size_t ppb = (size_t)pv * npb + pb;
  overlap_next();
  // the block's place in the table, by one warp: FP64 work
  __shared__ int s_ik;
  __shared__ R s_ak;
  const double k = kw[(size_t)pv * kw_stride];
  const bool has_z = threadIdx.x < nz;
  const R lz0 = has_z ? ldp[ppb * nz + threadIdx.x] : R(0);   // nz <= 64 threads: loads with k's
  const double mu0 = has_z ? mu[threadIdx.x] : 0.0;
  if (threadIdx.x < 32) {
    int ik = -1;
    R ak = R(0);
    if (kmin <= k && k <= kmax) table_place(k, kmin, dk, inv_dk, nk, ik, ak);
    if (threadIdx.x == 0) { s_ik = ik; s_ak = ak; }
  }
  if (threadIdx.x < npar) pvs[threadIdx.x] = (R)ldc[ppb * npar + threadIdx.x];
  __syncthreads();
  const int ik = s_ik;
  const R ak = s_ak;
  using W16 = typename Word16<R>::T;
  constexpr int PER = 16 / sizeof(R);
  const R* slab = nullptr;
  if constexpr (STAGE) {
    // the two slabs are consecutive: one stretch of 2 ng nz elements
    W16* S = reinterpret_cast<W16*>(gld_smem);
    slab = reinterpret_cast<const R*>(gld_smem);
    if (ik >= 0) {
      const W16* V = reinterpret_cast<const W16*>(W + (size_t)ik * ng * nz);
      const int n = 2 * ng * nz / PER;
      for (int i0 = threadIdx.x; i0 < n; i0 += 8 * 128) {
        W16 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = __ldg(V + min(i0 + q * 128, n - 1));
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (i0 + q * 128 < n) S[i0 + q * 128] = v[q];
      }
    }
  }
  if (has_z) {
    l[threadIdx.x] = lz0;
    for (int j = 0; j < npar; ++j) dl[j][threadIdx.x] = ld_dvalue<R>(law, (R)mu0, pvs, npar, j);
  }
  if (threadIdx.x < npar) {
    const int j = threadIdx.x;
    R d;
    if (!ld_dintegral<R>(law, pvs, j, d)) {
      const int NT = 200;
      R s = R(0), z0 = R(0), y0 = R(0);
      for (int i = 0; i < NT; ++i) {
        R m = R(NT - 1 - i) / R(NT - 1);
        R z = sqrt(R(1) - m * m);
        R y = z * ld_dvalue<R>(law, m, pvs, npar, j);
        if (i > 0) s += (z - z0) * (y + y0) / R(2);
        z0 = z;
        y0 = y;
      }
      d = R(2.0 * PI) * s;
    }
    dis[ppb * npar + j] = d;
  }
  __syncthreads();
  R* out = tab + ppb * (size_t)(1 + npar) * ng;
  for (int g = threadIdx.x; g < ng; g += blockDim.x) {
    if (ik >= 0) {
      R d0 = R(0), d1 = R(0);
      R c0[MAX_GRAD_PAR] = {}, c1[MAX_GRAD_PAR] = {};
      if constexpr (STAGE) {
        const W16 *w0 = reinterpret_cast<const W16*>(slab + (size_t)g * nz);
        const W16 *w1 = reinterpret_cast<const W16*>(slab + (size_t)(ng + g) * nz);
#pragma unroll 2
        for (int z = 0; z < nz / PER; ++z) {
          const W16 a0 = w0[z], a1 = w1[z], lz = reinterpret_cast<const W16*>(l)[z];
          Word16<R>::dot(d0, a0, lz);
          Word16<R>::dot(d1, a1, lz);
#pragma unroll
          for (int j = 0; j < MAX_GRAD_PAR; ++j)
            if (j < npar) {
              const W16 dz = reinterpret_cast<const W16*>(dl[j])[z];
              Word16<R>::dot(c0[j], a0, dz);
              Word16<R>::dot(c1[j], a1, dz);
            }
        }
      } else {
        const R* w0 = W + ((size_t)ik * ng + g) * nz;
        const R* w1 = w0 + (size_t)ng * nz;
        for (int z = 0; z < nz; ++z) {
          const R a0 = __ldg(w0 + z), a1 = __ldg(w1 + z);
          d0 += a0 * l[z];
          d1 += a1 * l[z];
#pragma unroll
          for (int j = 0; j < MAX_GRAD_PAR; ++j)
            if (j < npar) {
              c0[j] += a0 * dl[j][z];
              c1[j] += a1 * dl[j][z];
            }
        }
      }
      if constexpr (sizeof(R) == 4)
        out[g] = f32_quotient(f64_of_f32(d1) - f64_of_f32(d0), dk, inv_dk);
      else
        out[g] = (d1 - d0) / dk;
#pragma unroll
      for (int j = 0; j < MAX_GRAD_PAR; ++j)
        if (j < npar) out[(size_t)(1 + j) * ng + g] = (R(1) - ak) * c0[j] + ak * c1[j];
    } else {
      grad_ld_row_2d<R>(k, g, ng, nz, npar, ze, l, &dl[0][0], out);
    }
  }
  overlap_end();
}

// ---------------------------------------------------------------------------
// Observations: dobs[i] = o_i - 1 and isig2[i] = 1/sigma_lc^2 in R, and the
// pv-independent constant of lnL in per-block parts (FP64, fixed order), one
// block per OBS_CHUNK points.  With tiles64 also the FP64 summaries of the
// chunk's 128-point tiles (rr_time_tiles_f64), a warp per tile.
// ---------------------------------------------------------------------------
constexpr int OBS_THREADS = 128;
constexpr int OBS_CHUNK = OBS_THREADS * 4;
constexpr int OBS_LC = 128;   // light curves whose constants a block stages

template <typename R>
__global__ void __launch_bounds__(OBS_THREADS) obs_kernel(const double* __restrict__ obs,
                                                          const double* __restrict__ sigma,
                                                          const int32_t* __restrict__ lcids, int npt, int nlc,
                                                          R* __restrict__ dobs, R* __restrict__ isig2,
                                                          double* __restrict__ cpart,
                                                          const double* __restrict__ times,
                                                          double* __restrict__ tiles64) {
  __shared__ double red[OBS_THREADS / 32];
  static_assert(OBS_CHUNK == (OBS_THREADS / 32) * TIME_TILE, "a warp summarises one tile of the block's chunk");
  if (tiles64) {
    const int tile = blockIdx.x * (OBS_CHUNK / TIME_TILE) + (threadIdx.x >> 5);
    if (tile * TIME_TILE < npt) {   // warp-uniform
      const int lane = threadIdx.x & 31;
      const int lc0 = lcids[tile * TIME_TILE];
      double tmin = INFINITY, tmax = -INFINITY;
      bool same = true;
      for (int q = 0; q < TIME_TILE / 32; ++q) {
        const int i = tile * TIME_TILE + 32 * q + lane;
        if (i >= npt) break;
        tmin = fmin(tmin, times[i]);
        tmax = fmax(tmax, times[i]);
        same = same && lcids[i] == lc0;
      }
      for (int o = 16; o > 0; o >>= 1) {
        tmin = fmin(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
        tmax = fmax(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
      }
      same = __all_sync(0xffffffffu, same);
      if (lane == 0) {
        double* t = tiles64 + 4 * (size_t)tile;
        t[0] = tmin;
        t[1] = tmax;
        t[2] = same ? (double)lc0 : -1.0;
        t[3] = 0.0;
      }
    }
  }
  // A light curve's constants once per block (a logarithm and two divisions
  // per point made this kernel 13.5 us for 3000 points; now 8)
  __shared__ double s_c[OBS_LC][3];   // -log(sigma) - log(2 pi) / 2, 1 / sigma, 1 / sigma^2
  const double hl2pi = 0.5 * log(2.0 * PI);
  auto constants = [&](int lc, double* c) {
    const double sg = sigma[lc];
    c[0] = -log(sg) - hl2pi;
    c[1] = 1.0 / sg;
    c[2] = 1.0 / (sg * sg);
  };
  const bool staged = nlc <= OBS_LC;
  if (staged)
    for (int lc = threadIdx.x; lc < nlc; lc += blockDim.x) constants(lc, s_c[lc]);
  __syncthreads();
  double acc = 0.0;
  const int i0 = blockIdx.x * OBS_CHUNK, i1 = min(npt, i0 + OBS_CHUNK);
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    double c[3];
    if (staged) {
      for (int j = 0; j < 3; ++j) c[j] = s_c[lcids[i]][j];
    } else {
      constants(lcids[i], c);
    }
    const double d = obs[i] - 1.0;
    dobs[i] = (R)d;
    isig2[i] = (R)c[2];
    acc += c[0] - 0.5 * (d * c[1]) * (d * c[1]);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sm = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) sm += red[i];
    cpart[blockIdx.x] = sm;
  }
  overlap_end();
}

// ---------------------------------------------------------------------------
// Main kernel: blocks over (chunk of points, pv), each thread a few points.
// For in-box points: per sample the sky position and its derivatives (Horner
// on c and on dc), z, the area and its partials, the interpolated mean
// intensity and its partials; per point D = sum_s I A / (ns istar); lnL gets
// -(do + D/2) D / sigma^2, the gradient -(r / sigma^2) dD/dtheta with
// r = do + D.  Block sums go to partials[pv][block][1 + ngrad] (FP64), summed
// per pv in block order by lnlike_reduce_kernel: no step depends on timing.
// ---------------------------------------------------------------------------
struct GradArgs {
  // data
  const float2* times_ff;
  const int32_t *lcids, *pbids, *epids;
  const float *dobs, *isig2;
  int nkc, nep;
  // prologue tables
  const float *orb32, *lc32, *ldm, *dc, *tab, *dis;
  int npt, npv, npb, nlc, ng, npar, ngrad;
  double dg;
  double* partials;
};

__device__ __forceinline__ int grad_col(int slot, int nkc, int nep, int npar, int pb, int ep, int j) {
  switch (slot) {
    case GS_KK: return (nkc == 1) ? 0 : pb;
    case GS_KW: return 0;
    case GS_T0: return nkc + ep;
    case GS_P: case GS_A: case GS_I: case GS_E: case GS_W: return nkc + nep + (slot - GS_P);
    default: return nkc + nep + 5 + pb * npar + j;
  }
}

// Launch shape of the likelihood kernel: blocks of LNL_THREADS threads over
// LNL_CHUNK consecutive points of one pv, LNL_PPT points per thread.
constexpr int LNL_THREADS = 128;
constexpr int LNL_PPT = 8;
constexpr int LNL_CHUNK = LNL_THREADS * LNL_PPT;
constexpr int LNL_NW = LNL_THREADS / 32;
constexpr int DC_ROW = 12;   // a row of dc in shared memory: ten coefficients, 16-byte aligned

// a b + c d with one rounding fewer, in FP32: the first product is exact.
// The likelihood's arithmetic is written out in fused operations, so that its
// bits do not depend on how the compiler contracts and schedules it.
__device__ __forceinline__ float fma2(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }

// The kite of ccia_star (|1 - k| < z < 1 + k): its area and the half-angles
// of planet and star.
__device__ __forceinline__ float kite_area(float k, float z) {
  const float a = fmaxf(1.0f, k), b = fminf(1.0f, k);
  const float x = fmaxf(a, z), t = fminf(a, z);
  const float y = fmaxf(b, t), w = fminf(b, t);
  return 0.5f * sqrtf((x + (y + w)) * (w - (x - y)) * (w + (x - y)) * (x + (y - w)));
}
constexpr int LNL_STASH = 8;   // samples per point kept in shared memory for the second pass

// Adds one point's terms to the slot accumulators acc (the lnL term and, with
// GRAD, the gradient terms of GS_KK ... GS_C0 + npar - 1); false for a point
// out of the box, which adds nothing.  Two passes over the samples: the first
// gives the point's deficit D and with it the residual weight
// -(r / sigma^2) / (ns istar); the second adds each sample's derivative terms,
// already scaled by that weight, straight into acc (no per-point sums are
// kept).  The first LNL_STASH samples' separations and areas are kept in
// shared memory between the passes.
template <bool GRAD>
__device__ __forceinline__ bool lnlike_point(const GradArgs& A, int pv, int pt, int lc, const float* lcs, bool lc_smem,
                                             const float* orbc, const float* dcs, float4* stash, float* acc) {
  const float* LCR = lc_smem ? lcs + lc * LC32 : A.lc32 + ((size_t)pv * A.nlc + lc) * LC32;
  const float* o = A.orb32 + (size_t)pv * ORB32;
  const float p_hi = o[10], p_lo = o[11], inv_p = o[12];
  const float2 tt = A.times_ff[pt];
  const float d0h = LCR[LC_D0H], d0l = LCR[LC_D0L];
  float n = floorf(fmaf(tt.x - d0h, inv_p, 0.5f));
  float s1, e1, q1, e2, s2, e3;
  two_sum(tt.x, -d0h, s1, e1);
  two_prod(n, p_hi, q1, e2);
  two_sum(s1, -q1, s2, e3);
  float tc = s2 + (((e1 + e3) - e2) + (tt.y - d0l) - n * p_lo);
  if (tc >= 0.5f * p_hi || tc < -0.5f * p_hi) {
    n += (tc >= 0.5f * p_hi) ? 1.0f : -1.0f;
    two_prod(n, p_hi, q1, e2);
    two_sum(s1, -q1, s2, e3);
    tc = s2 + (((e1 + e3) - e2) + (tt.y - d0l) - n * p_lo);
  }
  if (!(LCR[LC_LO] <= tc && tc <= LCR[LC_HI])) return false;
  const float kk = LCR[LC_K], inv_is = LCR[LC_INVIS], ex = LCR[LC_EXPT], inv_ns = LCR[LC_INVNS];
  const int ns = __float_as_int(LCR[LC_NS]);
  const float inv1pk = 1.0f / (1.0f + kk);
  const float inv_dg = 1.0f / (float)A.dg;
  const size_t ppb = (size_t)pv * A.npb + A.pbids[lc];
  const float* L = A.ldm + ppb * A.ng;
  const float lim = 1.0f + kk, lim_in = fabsf(1.0f - kk), area_in = kk < 1.0f ? float(PI) * kk * kk : float(PI);
  // pass 1: the deficit D = sum_s I A / (ns istar)
  float SQ = 0.0f;
  for (int s = 0; s < ns; ++s) {
    const float t = fmaf(ex, fmaf((float)s + 0.5f, inv_ns, -0.5f), tc);
    float x = orbc[4], y = orbc[9];
#pragma unroll
    for (int m = 3; m >= 0; --m) {
      x = fmaf(x, t, orbc[m]);
      y = fmaf(y, t, orbc[5 + m]);
    }
    const float z = sqrtf(fma2(x, x, y, y));
    float a_kite = 0.0f;
    if (z < lim) {   // A = 0 and I A = 0 beyond first contact
      const float gg = z * inv1pk * inv_dg;
      const int i = min(max((int)gg, 0), A.ng - 2);
      const float fr = __fsub_rn(gg, (float)i);
      const float l0 = L[i], l1 = L[i + 1];
      float area = area_in;
      if (lim_in < z) {
        a_kite = kite_area(kk, z);
        const float k0 = atan2f(2.0f * a_kite, fma2(z, z, kk - 1.0f, kk + 1.0f));
        const float k1 = atan2f(2.0f * a_kite, fma2(z, z, 1.0f - kk, 1.0f + kk));
        area = __fsub_rn(fmaf(kk * kk, k0, k1), a_kite);
      }
      SQ = fmaf(fmaf(fr, l1 - l0, l0), area, SQ);
    }
    if (GRAD && s < LNL_STASH) stash[s * LNL_THREADS] = make_float4(x, y, z, a_kite);
  }
  const float sc = inv_is * inv_ns;
  const float D = __fmul_rn(SQ, sc);
  const float do_ = A.dobs[pt], w = A.isig2[pt];
  acc[GS_LNL] = fmaf(__fmul_rn(-fmaf(0.5f, D, do_), D), w, acc[GS_LNL]);
  if constexpr (GRAD) {
    const float r = __fadd_rn(do_, D);
    const float gsc = -r * w * sc;    // -(r / sigma^2) / (ns istar)
    const float* T = A.tab + ppb * (size_t)(1 + A.npar) * A.ng;
    // pass 2: the derivative terms of every sample, times gsc
    for (int s = 0; s < ns; ++s) {
      asm volatile("" ::: "memory");   // keeps the 50 derivative coefficients out of registers: see below
      const float t = fmaf(ex, fmaf((float)s + 0.5f, inv_ns, -0.5f), tc);
      float x, y, z, a_kite = 0.0f;
      if (s < LNL_STASH) {
        const float4 st = stash[s * LNL_THREADS];
        x = st.x; y = st.y; z = st.z; a_kite = st.w;
        if (!(z < lim)) continue;
      } else {
        x = orbc[4]; y = orbc[9];
#pragma unroll
        for (int m = 3; m >= 0; --m) {
          x = fmaf(x, t, orbc[m]);
          y = fmaf(y, t, orbc[5 + m]);
        }
        z = sqrtf(fma2(x, x, y, y));
        if (!(z < lim)) continue;
        if (lim_in < z) a_kite = kite_area(kk, z);
      }
      // d(x, y)/dt from m c_m
      float xd = orbc[10 + 3], yd = orbc[14 + 3];
#pragma unroll
      for (int m = 2; m >= 0; --m) {
        xd = fmaf(xd, t, orbc[10 + m]);
        yd = fmaf(yd, t, orbc[14 + m]);
      }
      // the area with its partial derivatives dA/dk = 2 k kappa0 and
      // dA/dz = -2 A_kite / z (ccia_star_grad)
      float ar = area_in, dadk = kk < 1.0f ? 2.0f * float(PI) * kk : 0.0f, dadz = 0.0f;
      if (lim_in < z) {
        const float k0 = atan2f(2.0f * a_kite, fma2(kk - 1.0f, kk + 1.0f, z, z));
        const float k1 = atan2f(2.0f * a_kite, fma2(1.0f - kk, 1.0f + kk, z, z));
        dadk = 2.0f * kk * k0;
        dadz = -2.0f * a_kite / z;
        ar = __fsub_rn(fmaf(kk * kk, k0, k1), a_kite);
      }
      const float g = z * inv1pk;
      const float gg = g * inv_dg;
      const int i = min(max((int)gg, 0), A.ng - 2);
      const float fr = __fsub_rn(gg, (float)i);
      const float l0 = L[i], l1 = L[i + 1];
      const float ip = fmaf(fr, l1 - l0, l0);
      const float gar = gsc * ar;
      const float iz = 1.0f / z;
      const float dzdt = fma2(x, xd, y, yd) * iz;
      const float dIdg = (l1 - l0) * inv_dg;
      const float gdz = gsc * fma2(ip, dadz, dIdg * inv1pk, ar);   // gsc dQ/dz
      acc[GS_KK] = fmaf(gsc, fma2(ip, dadk, -dIdg * g * inv1pk, ar), acc[GS_KK]);
      acc[GS_KW] = fmaf(fmaf(fr, T[i + 1] - T[i], T[i]), gar, acc[GS_KW]);
#pragma unroll
      for (int j = 0; j < MAX_GRAD_PAR; ++j) {
        if (j < A.npar) {
          const float* Tj = T + (size_t)(1 + j) * A.ng;
          acc[GS_C0 + j] = fmaf(fmaf(fr, Tj[i + 1] - Tj[i], Tj[i]), gar, acc[GS_C0 + j]);
        }
      }
      // dz/dtheta: orbit coefficients (p, a, i, e, w) and the time shift of t0, p
      acc[GS_T0] = fmaf(gdz, -dzdt, acc[GS_T0]);
#pragma unroll
      for (int jj = 0; jj < 5; ++jj) {
        const float4 da = *reinterpret_cast<const float4*>(dcs + jj * DC_ROW);
        const float4 db = *reinterpret_cast<const float4*>(dcs + jj * DC_ROW + 4);
        const float2 de = *reinterpret_cast<const float2*>(dcs + jj * DC_ROW + 8);
        const float d[10] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w, de.x, de.y};
        float dx = d[4], dy = d[9];
#pragma unroll
        for (int m = 3; m >= 0; --m) {
          dx = fmaf(dx, t, d[m]);
          dy = fmaf(dy, t, d[5 + m]);
        }
        const float q = fma2(x, dx, y, dy);
        const float dz = jj == 0 ? fma2(q, iz, dzdt, -n) : __fmul_rn(q, iz);
        acc[GS_P + jj] = fmaf(gdz, dz, acc[GS_P + jj]);
      }
    }
    // the disk integral's dependence on the LD coefficients
    const float* dI = A.dis + ppb * A.npar;
#pragma unroll
    for (int j = 0; j < MAX_GRAD_PAR; ++j)
      if (j < A.npar) acc[GS_C0 + j] = fmaf(r * w * D * inv_is, dI[j], acc[GS_C0 + j]);
  }
  return true;
}

// Adds the accumulators of the lanes in `pending` to the warp's row of
// shared FP64 sums, one group of lanes sharing a light curve at a time
// (lowest lane first), each slot by the same shuffle tree; then clears them.
// Groups without a point in the box add nothing.  The tree sums FP32 (hi, lo)
// pairs with error-free two-sums, as accurate as an FP64 tree; lane s keeps
// slot s's pair, so that one FP64 addition serves all slots (one per slot, on
// the pipe of 1/64 rate, held that pipe for a quarter of the adjoint's time).  Every step is
// in a fixed order, so the sums are reproducible bit for bit.
template <int NS>
__device__ __forceinline__ void lnlike_flush(const GradArgs& A, float* acc, int key, bool pending, bool& dirty,
                                             double* row) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nsl = NS > 1 ? GS_C0 + A.npar : 1;
  unsigned pend = __ballot_sync(FULL, pending);
  const unsigned live = __ballot_sync(FULL, dirty);
  while (pend) {
    const int leader = __ffs(pend) - 1;
    const int kl = __shfl_sync(FULL, key, leader);
    const unsigned mem = __ballot_sync(FULL, pending && key == kl) & pend;
    pend &= ~mem;
    if (!(mem & live)) continue;
    const bool in = (mem >> lane) & 1u;
    float my_hi = 0.0f, my_lo = 0.0f;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      if (s >= nsl) break;
      float hi = in ? acc[s] : 0.0f, lo = 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float h2 = __shfl_down_sync(FULL, hi, o), l2 = __shfl_down_sync(FULL, lo, o);
        float sh, se;
        two_sum(hi, h2, sh, se);
        lo = lo + l2 + se;
        hi = sh;
      }
      if (NS > 1) {
        hi = __shfl_sync(FULL, hi, 0);
        lo = __shfl_sync(FULL, lo, 0);
      }
      if (lane == s) { my_hi = hi; my_lo = lo; }
    }
    if (lane < nsl) {
      const int pb = A.pbids[kl], ep = A.epids[kl];
      const int col = lane == GS_LNL ? -1 : grad_col(lane, A.nkc, A.nep, A.npar, pb, ep, lane - GS_C0);
      const double tot = (double)my_hi + (double)my_lo;
      if (lane != GS_KK && lane != GS_KW) row[col + 1] += tot;
      // both slots of the radius ratio can share a column
      __syncwarp((1u << nsl) - 1u);
      if (lane == GS_KK) row[col + 1] += tot;
      __syncwarp((1u << nsl) - 1u);
      if (lane == GS_KW) row[col + 1] += tot;
    }
    __syncwarp();
    if (in) {
#pragma unroll
      for (int s = 0; s < NS; ++s) acc[s] = 0.0f;
      dirty = false;
    }
  }
}

// One block: LNL_CHUNK consecutive points of pv.  Each thread sums its points'
// terms in registers while they share a light curve (the gradient columns
// depend on its passband and epoch), flushing to its warp's row of shared
// sums when the light curve changes and at the end; the block writes the sum
// of the warps' rows, in warp order, to its slot of partials.
//
// Bound by instruction issue and, at few warps, by its latency.  With the orbit
// coefficients' derivatives read from shared memory as 16-byte words for each
// sample instead of held in 50 registers, 20 warps fit on an SM instead of 16.
// Adjoint of 4096 pv x 5000 times x 5 samples: 887 us before, 890 with the FP64
// additions and the second pass's separations alone taken out (registers
// spilled), 819 with the coefficients out of the registers, 743 at 20 warps
// (739 at 24, which spills and costs the likelihood alone 2 %: 242 us, not 238).
template <bool GRAD>
__global__ void __launch_bounds__(LNL_THREADS, 5) lnlike_kernel(const __grid_constant__ GradArgs A) {
  constexpr int NS = GRAD ? GS_NSLOT : 1;
  __shared__ double wred[LNL_NW][1 + MAX_NGRAD];
  __shared__ __align__(16) float lcs[GLC_SMEM * LC32];
  __shared__ __align__(16) float orbc[18];   // c_m of x and y; m c_m (m = 1..4) of x and y
  __shared__ __align__(16) float dcs[5 * DC_ROW];
  __shared__ float4 stash[GRAD ? LNL_STASH * LNL_THREADS : 1];
  const int pv = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int i = tid; i < LNL_NW * (1 + MAX_NGRAD); i += blockDim.x) (&wred[0][0])[i] = 0.0;
  if (tid < 10) {
    const float c = A.orb32[(size_t)pv * ORB32 + tid];
    const int m = tid % 5;
    orbc[tid] = c;
    if (m > 0) orbc[10 + tid / 5 * 4 + m - 1] = __fmul_rn((float)m, c);
  }
  if (GRAD && tid < 50) dcs[tid / 10 * DC_ROW + tid % 10] = A.dc[(size_t)pv * 50 + tid];
  const bool lc_smem = A.nlc <= GLC_SMEM;
  if (lc_smem)
    for (int i = tid; i < A.nlc * LC32; i += blockDim.x) lcs[i] = A.lc32[(size_t)pv * A.nlc * LC32 + i];
  __syncthreads();
  const bool valid = __float_as_int(A.orb32[(size_t)pv * ORB32 + 14]) & FLAG_VALID;
  float acc[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) acc[s] = 0.0f;
  int key = -1;
  bool dirty = false;   // acc holds a point's terms
  for (int j = 0; j < LNL_PPT; ++j) {
    const int pt = blockIdx.x * LNL_CHUNK + j * LNL_THREADS + tid;
    const int lc = (valid && pt < A.npt) ? A.lcids[pt] : -1;
    const bool flush = key >= 0 && lc >= 0 && lc != key;
    if (__any_sync(0xffffffffu, flush)) {
      lnlike_flush<NS>(A, acc, key, flush, dirty, wred[warp]);
      if (flush) key = -1;
    }
    if (lc < 0) continue;
    dirty |= lnlike_point<GRAD>(A, pv, pt, lc, lcs, lc_smem, orbc, dcs, stash + (GRAD ? tid : 0), acc);
    key = lc;
  }
  lnlike_flush<NS>(A, acc, key, key >= 0, dirty, wred[warp]);
  __syncthreads();
  double* out = A.partials + ((size_t)pv * gridDim.x + blockIdx.x) * (1 + A.ngrad);
  for (int i = tid; i <= A.ngrad; i += blockDim.x) {
    double sm = 0.0;
#pragma unroll
    for (int w = 0; w < LNL_NW; ++w) sm += wred[w][i];
    out[i] = sm;
  }
}

// ---------------------------------------------------------------------------
// The FP64 likelihood and its adjoint, one warp per share of a pv's row, on the
// walk, queue and sample arithmetic of the FP64 flux (rr_f64_points.cuh): the
// FP64 pipe bounds both, so the in-box points are collected and their inner
// and limb samples run as full warps.
//
// The adjoint's sums are taken in the form that needs the fewest FP64
// instructions per sample:
//   * orbit coefficients: z depends on theta through x(t) and y(t), polynomials
//     whose coefficients' derivatives dc belong to the pv, so the samples only
//     accumulate the moments sum (x / z) t^m dL/dz and sum (y / z) t^m dL/dz
//     (18 instructions a sample, against 55 for five derivative polynomials);
//     the five columns follow from the ten moments once per share;
//   * disk integral: one sum of r D / sigma^2 per light curve.
// Sums are per lane in a fixed order, over lanes in lane order and over shares
// in order: reproducible bit for bit.
// ---------------------------------------------------------------------------
enum FSlot { FS_LNL = 0, FS_KK, FS_KW, FS_IS, FS_T, FS_P, FS_C0, FS_M0 = FS_C0 + MAX_GRAD_PAR, FS_NSLOT = FS_M0 + 10 };

struct LnlF64Args : F64Args {
  const double *dobs, *isig2, *dc, *tab, *dis;
  int npar, nep, ngrad;
  double* partials;
};

template <bool GRAD>
struct LnlF64Smem {
  static constexpr int NS = GRAD ? FS_NSLOT : 1;
  double acc[NS][33];                      // per-lane sums of the current light curve
  double tot[NS];
  double row[GRAD ? 1 + MAX_NGRAD : 1];    // the share's columns
  double g[GRAD ? F64_Q : 1];              // per point of a chunk: -(r / sigma^2) w
  double ep[GRAD ? F64_Q : 1];             // per point of a chunk: epoch
  int lc;                                  // a light curve of acc's passband and epoch, or -1
};

// I(z) A(z)'s value and partial derivatives at one sample.
struct F64Partials {
  double x, y, iz, ip, slope, ar, dadk, dadz, z, fr;   // slope = dI/dz
  int i;
  bool none;
};

static __device__ __noinline__ void f64_partials_general(const F64Disk& K, const F64Transit& T, double r2, F64Partials& S) {
  const double z = sqrt(r2);
  S.z = z;
  S.none = z >= 1.0 + K.k;   // NaN has partial derivatives: NaN
  S.iz = 1.0 / z;
  const double gg = z / (1.0 + K.k) / T.dg;
  S.i = min(max((int)gg, 0), T.ng - 2);
  S.fr = gg - (double)S.i;
  const double l0 = T.lda[S.i], l1 = T.lda[S.i + 1];
  S.ip = l0 + S.fr * (l1 - l0);
  S.slope = (l1 - l0) / ((1.0 + K.k) * T.dg);
  S.ar = ccia_star_grad<double>(K.k, z, S.dadk, S.dadz);
}

__device__ __forceinline__ void f64_partials(const F64Lc& R, const F64Transit& T, double t, bool limb, F64Partials& S) {
  const F64Disk& K = R.disk;
  const double* c = T.o;
  double x = c[4], y = c[9];
#pragma unroll
  for (int m = 3; m >= 0; --m) {
    x = __fma_rn(x, t, c[m]);
    y = __fma_rn(y, t, c[5 + m]);
  }
  S.x = x;
  S.y = y;
  S.none = false;
  const double r2 = __fma_rn(x, x, __dmul_rn(y, y));
  if (!f64_moderate(r2) || (limb && !K.fast)) {
    f64_partials_general(K, T, r2, S);
    return;
  }
  const F64Root q = f64_root(r2);
  S.z = f64_sqrt(q);
  S.iz = f64_rsqrt(q);
  double l0, dl;
  f64_ld_cell(K, S.z, T.lda, T.ng, S.i, S.fr, l0, dl);
  S.ip = __fma_rn(S.fr, dl, l0);
  S.slope = __dmul_rn(dl, K.cg);
  if (limb) {
    const F64Limb L = f64_limb<true>(K, r2, S.iz);
    S.ar = L.area;
    S.dadk = __dmul_rn(__dadd_rn(K.k, K.k), L.kappa0);
    S.dadz = __dmul_rn(-2.0 * L.kite, S.iz);
  } else {
    S.ar = K.area_in;
    S.dadk = __dmul_rn(2.0 * PI, K.k);
    S.dadz = 0.0;
  }
}

// The lanes' sums into the share's columns of the passband and epoch of light curve S.lc.
template <bool GRAD>
__device__ __noinline__ void lnl_f64_reduce(const LnlF64Args& A, LnlF64Smem<GRAD>& S, int pv) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  // lnL in the same order with and without the gradient
  double l = S.acc[FS_LNL][lane];
  for (int d = 16; d > 0; d >>= 1) l = __dadd_rn(l, __shfl_down_sync(0xffffffffu, l, d));
  if (lane == 0) S.row[0] += l;
  if constexpr (GRAD) {
    // a lane per slot, over the lanes in order: 31 FP64 instructions for all slots
    if (lane > FS_LNL && lane < S.NS) {
      double v = S.acc[lane][0];
      for (int i = 1; i < 32; ++i) v = __dadd_rn(v, S.acc[lane][i]);
      S.tot[lane] = v;
    }
    __syncwarp();
    const int pb = A.pbids[S.lc], ep = A.epids[S.lc], nkc = A.nkc, nep = A.nep;
    double* col = S.row + 1;
    if (lane < 5) {
      const double* d = A.dc + (size_t)pv * 50 + lane * 10;
      double v = lane == 0 ? -S.tot[FS_P] : 0.0;
      for (int m = 0; m < 10; ++m) v += d[m] * S.tot[FS_M0 + m];
      col[nkc + nep + lane] += v;
    } else if (lane == 6) {
      col[nkc == 1 ? 0 : pb] += S.tot[FS_KK];
      col[0] += S.tot[FS_KW];
    } else if (lane == 7) {
      col[nkc + ep] -= S.tot[FS_T];
    } else if (lane >= 8 && lane < 8 + A.npar) {
      const int j = lane - 8;
      const size_t ppb = (size_t)pv * A.npb + pb;
      col[nkc + nep + 5 + pb * A.npar + j] +=
          S.tot[FS_C0 + j] + S.tot[FS_IS] * A.dis[ppb * A.npar + j] / A.istar[ppb];
    }
  }
  __syncwarp();
  for (int i = lane; i < S.NS * 33; i += 32) (&S.acc[0][0])[i] = 0.0;
  __syncwarp();
}

// The terms of the n queued points, all of light curve lc, into the lanes' sums.
template <bool GRAD>
__device__ __noinline__ void lnl_f64_flush(const LnlF64Args& A, const F64Orbit& P, F64Lc* recs, F64Queue& Q,
                                           const double* o, LnlF64Smem<GRAD>& S, int pv, int lc, int n) {
  const int lane = threadIdx.x & 31, nrec = min(A.nlc, F64_LC_SMEM);
  const int before = S.lc;
  __syncwarp();   // every lane has read it
  if (lc != before) {
    // the sums' columns are those of the passband and the epoch
    if (before >= 0 && (A.pbids[lc] != A.pbids[before] || A.epids[lc] != A.epids[before]))
      lnl_f64_reduce<GRAD>(A, S, pv);
    if (lane == 0) S.lc = lc;
    __syncwarp();
  }
  if (lc >= F64_LC_SMEM) {
    if (lane == 0) f64_lc<GRAD>(A, pv, lc, P, recs[nrec]);
    __syncwarp();
  }
  const F64Lc& R = recs[min(lc, nrec)];
  const size_t ppb = (size_t)pv * A.npb + R.pb;
  const F64Transit T{o, A.ldm + ppb * A.ng, A.ng, A.dg};
  double lnl = S.acc[FS_LNL][lane], is = GRAD ? S.acc[GRAD ? FS_IS : 0][lane] : 0.0;
  const double t0 = GRAD ? A.t0[(size_t)pv * A.ldt0 + A.epids[lc]] : 0.0, p = A.p[pv];
  const float inv_p = 1.0f / f32_of(p);
  f64_sums(
      R, P, T, Q, n,
      [&](int i, double SQ) {
        const int pt = Q.pt[i];
        const bool in = f64_in_box(A, P, R, Q.tc[i]);
        const double D = in ? __dmul_rn(SQ, R.w) : 0.0, d = A.dobs[pt], w = A.isig2[pt];
        lnl = __fma_rn(-__dmul_rn(__fma_rn(0.5, D, d), D), w, lnl);
        if constexpr (GRAD) {
          const int j = i % (F64_Q / min(max(R.ns, 1), F64_Q));   // the point's place in its chunk
          const double rw = __dmul_rn(__dadd_rn(d, D), w);
          S.g[j] = in ? __dmul_rn(-rw, R.w) : 0.0;
          is = __fma_rn(rw, D, is);
          S.ep[j] = f64_epoch(A.times[pt], t0, p, inv_p);   // the fold's
        }
      },
      [&](int i0, int ni) {
        if constexpr (GRAD) {
          double a[FS_NSLOT];
#pragma unroll
          for (int s = 0; s < FS_NSLOT; ++s) a[s] = S.acc[s][lane];
          const double* tab = A.tab + ppb * (size_t)(1 + A.npar) * A.ng;
          const double inv1pk = __dmul_rn(R.disk.cg, A.dg);
          const int sc = min(max(R.ns, 1), F64_Q);
          __syncwarp();
          auto sample = [&](int it, int smp, bool limb) {
            const double t = f64_sample_time(R, Q.tc[i0 + it], smp);
            F64Partials q;
            f64_partials(R, T, t, limb, q);
            if (q.none) return;
            const double g = S.g[it], ga = __dmul_rn(g, q.ar);
            const double gi = __dmul_rn(g, q.ip);
            a[FS_KK] = __fma_rn(gi, q.dadk, a[FS_KK]);
            a[FS_KK] = __fma_rn(-__dmul_rn(__dmul_rn(q.slope, q.z), inv1pk), ga, a[FS_KK]);
            const double* Tt = tab + q.i;
#pragma unroll
            for (int j = -1; j < MAX_GRAD_PAR; ++j) {
              if (j >= A.npar) break;
              const double* Tj = Tt + (size_t)(1 + j) * A.ng;
              const double v = __fma_rn(q.fr, __dadd_rn(__ldg(Tj + 1), -__ldg(Tj)), __ldg(Tj));
              double& s = a[j < 0 ? FS_KW : FS_C0 + j];
              s = __fma_rn(v, ga, s);
            }
            // dL/dz over z, then its moments
            const double gz = __dmul_rn(__fma_rn(q.slope, ga, __dmul_rn(gi, q.dadz)), q.iz);
            double u = __dmul_rn(gz, q.x), v = __dmul_rn(gz, q.y);
            double xd = __dmul_rn(4.0, o[4]), yd = __dmul_rn(4.0, o[9]);
#pragma unroll
            for (int m = 3; m >= 1; --m) {
              xd = __fma_rn(xd, t, (double)m * o[m]);
              yd = __fma_rn(yd, t, (double)m * o[5 + m]);
            }
            const double gt = __fma_rn(u, xd, __dmul_rn(v, yd));   // dL/dz dz/dt
            a[FS_T] = __dadd_rn(a[FS_T], gt);
            a[FS_P] = __fma_rn(gt, S.ep[it], a[FS_P]);
#pragma unroll
            for (int m = 0; m < 5; ++m) {
              a[FS_M0 + m] = __dadd_rn(a[FS_M0 + m], u);
              a[FS_M0 + 5 + m] = __dadd_rn(a[FS_M0 + 5 + m], v);
              if (m < 4) {
                u = __dmul_rn(u, t);
                v = __dmul_rn(v, t);
              }
            }
          };
          for (int s0 = 0; s0 < R.ns; s0 += sc)
            f64_pairs(
                R, P, Q, i0, ni, s0, min(sc, R.ns - s0),
                [&](int, int it, int smp) { sample(it, smp, false); },
                [&](int, int it, int smp) { sample(it, smp, true); }, [](int) {});
#pragma unroll
          for (int s = 0; s < FS_NSLOT; ++s)
            if (s != FS_LNL && s != FS_IS) S.acc[s][lane] = a[s];
          __syncwarp();
        }
      });
  S.acc[FS_LNL][lane] = lnl;
  if constexpr (GRAD) S.acc[FS_IS][lane] = is;
}

template <bool GRAD>
struct LnlF64Sink {
  static constexpr bool BY_LIGHT_CURVE = true;   // with and without the gradient: the same sums
  const LnlF64Args& A;
  const F64Orbit& P;
  F64Lc* recs;
  F64Queue& Q;
  const double* o;
  LnlF64Smem<GRAD>& S;
  int pv;

  __device__ __forceinline__ void tile(int, int, int) const {}
  __device__ __forceinline__ void outside(int) const {}
  __device__ __forceinline__ void flush(int lc, int n) const { lnl_f64_flush<GRAD>(A, P, recs, Q, o, S, pv, lc, n); }
};

template <bool GRAD>
__global__ void __launch_bounds__(32, GRAD ? 12 : 20) lnlike_f64_kernel(const __grid_constant__ LnlF64Args A, const double* tiles64,
                                                                         int slots) {
  __shared__ double o[ORB64];
  __shared__ F64Orbit P;
  __shared__ F64Queue Q;
  __shared__ LnlF64Smem<GRAD> S;
  extern __shared__ __align__(16) unsigned char lnl_smem[];
  F64Lc* recs = reinterpret_cast<F64Lc*>(lnl_smem);
  const int pv = blockIdx.y, lane = threadIdx.x;
  if (lane < ORB64) o[lane] = A.orb64[(size_t)pv * ORB64 + lane];
  const int ncol = GRAD ? 1 + A.ngrad : 1;
  for (int i = lane; i < ncol; i += 32) S.row[i] = 0.0;
  if (lane == 0) S.lc = -1;
  for (int i = lane; i < S.NS * 33; i += 32) (&S.acc[0][0])[i] = 0.0;
  __syncwarp();
  const bool valid = o[12] != 0.0;
  if (valid) {
    if (lane == 0) f64_orbit(o, P);
    __syncwarp();
    for (int lc = lane; lc < min(A.nlc, F64_LC_SMEM); lc += 32) f64_lc<GRAD>(A, pv, lc, P, recs[lc]);
    __syncwarp();
    f64_walk(A, pv, tiles64, slots, true, P, recs, Q, LnlF64Sink<GRAD>{A, P, recs, Q, o, S, pv});
    if (S.lc >= 0) lnl_f64_reduce<GRAD>(A, S, pv);
  }
  double* out = A.partials + ((size_t)pv * gridDim.x + blockIdx.x) * (1 + A.ngrad);
  for (int i = lane; i < ncol; i += 32) out[i] = S.row[i];
}

// Sum the block partials of each pv in a fixed order; invalid pv -> NaN.
__global__ void lnlike_reduce_kernel(const double* __restrict__ partials, int nblk, int ngrad, int npv,
                                     const double* __restrict__ cpart, int ncpart, const double* __restrict__ orb64,
                                     const float* __restrict__ orb32, double* __restrict__ lnl,
                                     double* __restrict__ grad) {
  const int pv = blockIdx.x;
  const bool valid = orb32 ? (__float_as_int(orb32[(size_t)pv * ORB32 + 14]) & FLAG_VALID)
                           : (orb64[(size_t)pv * ORB64 + 12] != 0.0);
  for (int i = threadIdx.x; i <= (grad ? ngrad : 0); i += blockDim.x) {
    double s = 0.0;
    for (int b = 0; b < nblk; ++b) s += partials[((size_t)pv * nblk + b) * (1 + ngrad) + i];
    if (!valid) s = CUDART_NAN;
    if (i == 0) {
      double c = 0.0;
      for (int b = 0; b < ncpart; ++b) c += cpart[b];
      lnl[pv] = s + c;
    }
    else if (grad) grad[(size_t)pv * ngrad + i - 1] = s;
  }
}

template <typename R>
struct GradWs {
  R *dc, *tab, *dis, *dobs, *isig2;
  double *partials, *cconst;   // cconst: the constant of lnL in per-block parts
  double* tiles64;             // FP64 path: tile summaries
};

template <typename R>
static GradWs<R> carve_grad(Carve& cv, int npv, int npb, int npar, int ng, int npt, size_t npart, int ngrad) {
  GradWs<R> g;
  g.dc = cv.take<R>((size_t)npv * 50);
  g.tab = cv.take<R>((size_t)npv * npb * (1 + npar) * ng);
  g.dis = cv.take<R>((size_t)npv * npb * (npar > 0 ? npar : 1));
  g.dobs = cv.take<R>((size_t)npt);
  g.isig2 = cv.take<R>((size_t)npt);
  g.partials = cv.take<double>(npart * (1 + ngrad));
  g.cconst = cv.take<double>((size_t)(npt + OBS_CHUNK - 1) / OBS_CHUNK);
  g.tiles64 = sizeof(R) == 8 ? cv.take<double>(4 * (((size_t)npt + TIME_TILE - 1) / TIME_TILE)) : nullptr;
  return g;
}

// Shares of a pv's row.  In FP64 they follow the launch's size, counted for the
// GB300's 152 SMs whatever device is current, so that a workspace holds for every
// device.  (A partial sum per 2, 4 or 8 tiles in every launch would make the last
// bits independent of the vectors beside one, and one vector's adjoint over 3000 x 5
// samples 311, 411 or 712 us instead of 116.)
constexpr int LNL64_SMS = 152;
static int lnlike_f64_slots(int npt, int npv) { return f64_slots(npt, npv, LNL64_SMS); }
static int lnlike_blocks(int split, int npt, int npv) {
  return split ? (npt + LNL_CHUNK - 1) / LNL_CHUNK : f64_warps(npt, lnlike_f64_slots(npt, npv));
}

// Partial sums that a workspace has room for: at least npv lnlike_blocks(...) of
// this and of every smaller call, so that one workspace for the largest population
// serves all.  In FP64, with R = 16 x 152 warps a round and T = npv ntiles, f64_slots
// gives a row at most four shares a tile, at most R shares in all below R tiles,
// less than 2 R below 9 R tiles, and above T / w rounded up per row with w = 8, or
// T / 4 R from 36 R on, or 64.
static size_t lnlike_partials(int split, int npt, int npv) {
  if (split) return (size_t)npv * lnlike_blocks(split, npt, npv);
  const size_t ntiles = ((size_t)npt + TIME_TILE - 1) / TIME_TILE, n = (size_t)npv;
  return std::min(4 * ntiles * n, 5 * 16 * (size_t)LNL64_SMS + n * (1 + ntiles / 64 + 1));
}

}  // namespace rr

using namespace rr;

extern "C" {

int rr_lnlike_ngrad(int nkc, int nep, int npb, int npar) { return nkc + nep + 5 + npb * npar; }

size_t rr_lnlike_workspace_bytes(int split, int npv, int npb, int nlc, int nep, int ng, int npar, int npt,
                                 int nkc) {
  const size_t npart = lnlike_partials(split, npt, npv);
  const int ngrad = rr_lnlike_ngrad(nkc, nep, npb, npar);
  size_t base = split ? rr_full_split_workspace_bytes(npv, npb, nlc, nep, ng) : rr_full_f64_workspace_bytes(npv, npb, ng);
  Carve c(nullptr);
  if (split) carve_grad<float>(c, npv, npb, npar, ng, npt, npart, ngrad);
  else carve_grad<double>(c, npv, npb, npar, ng, npt, npart, ngrad);
  return base + c.used + 512;
}

}  // extern "C"

template <typename R>
static int lnlike_impl(int split, int law, const double* ldc, int npar, const double* mu, const double* times,
                       const float* times_ff, double t_ref, double t_absmax, int npt, const double* k, int nkc,
                       const double* t0, int ldt0, int nep, const double* p, const double* a, const double* inc,
                       const double* e, const double* w, int npv, int nlc, int npb, const int32_t* lcids,
                       const int32_t* pbids, const int32_t* epids, const int32_t* nsamples,
                       const double* exptimes, const R* ldp, const R* istar, const R* weights, int nk, int ng,
                       int nz, double dk, double kmin, double kmax, double dg, const double* z_edges,
                       const double* obs, const double* sigma, void* workspace, size_t workspace_bytes,
                       double* lnl, double* grad, void* stream, const double* basis = nullptr, int nb = 0,
                       bool make_ld = false) {
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (law < 0 || law >= LD_NLAWS) return RR_ERR_LAW;
  if (npt < 1 || npv < 0 || nlc < 1 || npb < 1 || nk < 2 || ng < 2 || nz < 1 || nz > 64 || nkc < 1 || nep < 1 ||
      nep > ldt0 || npar < 0 || npar > MAX_GRAD_PAR)
    return RR_ERR_ARG;
  const int ngrad = rr_lnlike_ngrad(nkc, nep, npb, npar);
  if (ngrad > MAX_NGRAD) return RR_ERR_ARG;
  if (npv == 0) return RR_OK;
  if (npv > 65535) return RR_ERR_ARG;
  if (workspace_bytes < rr_lnlike_workspace_bytes(split, npv, npb, nlc, nep, ng, npar, npt, nkc))
    return RR_ERR_WORKSPACE;
  const int nblk = lnlike_blocks(split, npt, npv);
  const size_t npart = lnlike_partials(split, npt, npv);
  if ((size_t)npv * nblk > npart) return RR_ERR_WORKSPACE;   // never: see lnlike_partials
  cudaStream_t s = as_stream(stream);
  size_t base = split ? rr_full_split_workspace_bytes(npv, npb, nlc, nep, ng) : rr_full_f64_workspace_bytes(npv, npb, ng);
  int st;
  if (split)
    st = rr_prepare_split(t_ref, t_absmax, k, nkc, t0, ldt0, nep, p, a, inc, e, w, npv, nlc, npb, pbids, epids,
                          nsamples, exptimes, (const float*)ldp, (const float*)istar, (const float*)weights, nk, ng,
                          nz, dk, kmin, kmax, z_edges, workspace, base, stream, 0, nullptr, 0, nullptr, 0);
  else if (make_ld) {
    // the adjoint reads the whole profile, which the fused prologue leaves out
    double *ldp64 = (double*)const_cast<R*>(ldp), *istar64 = (double*)const_cast<R*>(istar);
    st = grad && prepare_f64_fused(law, npar, npb, ldc, mu, basis, nb)
             ? rr_ld_tables_f64(law, ldc, npv, npb, npar, mu, nz, ldp64, istar64, stream)
             : RR_OK;
    if (st == RR_OK)
      st = rr_prepare_f64_ld(k, nkc, p, a, inc, e, w, npv, npb, law, ldc, npar, mu, nz, basis, nb,
                             (const double*)weights, nk, ng, dk, kmin, kmax, z_edges, ldp64, istar64, workspace, base,
                             stream);
  } else
    st = rr_prepare_f64(k, nkc, p, a, inc, e, w, npv, npb, (const double*)ldp, (const double*)weights, nk, ng, nz,
                        dk, kmin, kmax, z_edges, workspace, base, stream, 0, nullptr, 0, nullptr, 0);
  if (st) return st;
  Carve cv(static_cast<char*>(workspace) + base);
  GradWs<R> g = carve_grad<R>(cv, npv, npb, npar, ng, npt, npart, ngrad);
  // prologue tables of the forward pass (inside the base workspace)
  Carve pcv(workspace);
  const double* orb64 = nullptr;
  const float *orb32 = nullptr, *lc32 = nullptr;
  const R* ldm;
  if (split) {
    orb32 = pcv.take<float>((size_t)npv * ORB32);
    lc32 = pcv.take<float>((size_t)npv * nlc * LC32);
    ldm = (const R*)pcv.take<float>((size_t)npv * npb * ng);
  } else {
    orb64 = pcv.take<double>((size_t)npv * ORB64);
    ldm = (const R*)pcv.take<double>((size_t)npv * npb * ng);
  }
  if (grad) {   // the derivative tables, read by the adjoint alone
    // an ordinary launch: beside the end of the LD means its blocks crowd the first
    // SMs with room, where they share a few FP64 pipes (77 us, against 25)
    grad_orbit_kernel<R><<<(5 * npv + 63) / 64, 64, 0, s>>>(p, a, inc, e, w, npv, g.dc);
    // rows of whole 16-byte words, two slabs within what four blocks of an SM can have
    const size_t slabs = 2 * sizeof(R) * (size_t)ng * nz;
    const bool stage = nz % (16 / sizeof(R)) == 0 && (reinterpret_cast<uintptr_t>(weights) & 15) == 0 && slabs <= GLD_SMEM;
    auto fn = stage ? grad_ld_kernel<R, true> : grad_ld_kernel<R, false>;
    if (stage && slabs > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)slabs);
    launch_overlap(fn, dim3(npv, npb), 128, stage ? slabs : 0, s, law, ldc, npb, npar, mu, nz, ldp, k, nkc, weights, nk,
                   ng, dk, 1.0 / dk, kmin, kmax, z_edges, g.tab, g.dis);
  }
  const int nobs = (npt + OBS_CHUNK - 1) / OBS_CHUNK;
  launch_overlap(obs_kernel<R>, nobs, OBS_THREADS, 0, s, obs, sigma, lcids, npt, nlc, g.dobs, g.isig2, g.cconst, times,
                 g.tiles64);
  if constexpr (sizeof(R) == 4) {
    GradArgs A{};
    A.times_ff = reinterpret_cast<const float2*>(times_ff);
    A.lcids = lcids; A.pbids = pbids; A.epids = epids;
    A.dobs = g.dobs; A.isig2 = g.isig2; A.nkc = nkc; A.nep = nep;
    A.orb32 = orb32; A.lc32 = lc32;
    A.ldm = ldm; A.dc = g.dc; A.tab = g.tab; A.dis = g.dis;
    A.npt = npt; A.npv = npv; A.npb = npb; A.nlc = nlc; A.ng = ng; A.npar = npar; A.ngrad = ngrad;
    A.dg = dg; A.partials = g.partials;
    const dim3 grid(nblk, npv);
    if (grad) lnlike_kernel<true><<<grid, LNL_THREADS, 0, s>>>(A);
    else lnlike_kernel<false><<<grid, LNL_THREADS, 0, s>>>(A);
  } else {
    LnlF64Args A{};
    A.times = times; A.k = k; A.t0 = t0; A.p = p; A.exptimes = exptimes; A.istar = (const double*)istar;
    A.ldm = (const double*)ldm; A.orb64 = orb64;
    A.lcids = lcids; A.pbids = pbids; A.epids = epids; A.nsamples = nsamples;
    A.npt = npt; A.npv = npv; A.nkc = nkc; A.ldt0 = ldt0; A.npb = npb; A.nlc = nlc; A.ng = ng; A.dg = dg;
    A.dobs = g.dobs; A.isig2 = g.isig2; A.dc = g.dc; A.tab = g.tab; A.dis = g.dis;
    A.npar = npar; A.nep = nep; A.ngrad = ngrad; A.partials = g.partials;
    const dim3 grid(nblk, npv);
    const int slots = lnlike_f64_slots(npt, npv);
    const size_t smem = sizeof(F64Lc) * (std::min(nlc, F64_LC_SMEM) + 1);
    if (grad) lnlike_f64_kernel<true><<<grid, 32, smem, s>>>(A, g.tiles64, slots);
    else lnlike_f64_kernel<false><<<grid, 32, smem, s>>>(A, g.tiles64, slots);
  }
  lnlike_reduce_kernel<<<npv, 64, 0, s>>>(g.partials, nblk, ngrad, npv, g.cconst, nobs, orb64, orb32, lnl, grad);
  return check_launch("rr_lnlike");
}

extern "C" {


int rr_lnlike_f64(int law, const double* ldc, int npar, const double* mu, const double* times, int npt,
                  const double* k, int nkc, const double* t0, int ldt0, int nep, const double* p, const double* a,
                  const double* inc, const double* e, const double* w, int npv, int nlc, int npb,
                  const int32_t* lcids, const int32_t* pbids, const int32_t* epids, const int32_t* nsamples,
                  const double* exptimes, const double* ldp, const double* istar, const double* weights, int nk,
                  int ng, int nz, double dk, double kmin, double kmax, double dg, const double* z_edges,
                  const double* obs, const double* sigma, void* workspace, size_t workspace_bytes, double* lnl,
                  double* grad, void* stream) {
  return lnlike_impl<double>(0, law, ldc, npar, mu, times, nullptr, 0.0, 0.0, npt, k, nkc, t0, ldt0, nep, p, a, inc,
                             e, w, npv, nlc, npb, lcids, pbids, epids, nsamples, exptimes, ldp, istar, weights, nk,
                             ng, nz, dk, kmin, kmax, dg, z_edges, obs, sigma, workspace, workspace_bytes, lnl, grad,
                             stream);
}

int rr_lnlike_f64_ld(int law, const double* ldc, int npar, const double* mu, const double* basis, int nb,
                     const double* times, int npt, const double* k, int nkc, const double* t0, int ldt0, int nep,
                     const double* p, const double* a, const double* inc, const double* e, const double* w, int npv,
                     int nlc, int npb, const int32_t* lcids, const int32_t* pbids, const int32_t* epids,
                     const int32_t* nsamples, const double* exptimes, double* ldp, double* istar,
                     const double* weights, int nk, int ng, int nz, double dk, double kmin, double kmax, double dg,
                     const double* z_edges, const double* obs, const double* sigma, void* workspace,
                     size_t workspace_bytes, double* lnl, double* grad, void* stream) {
  if (!mu || !ldp || !istar) return RR_ERR_ARG;
  return lnlike_impl<double>(0, law, ldc, npar, mu, times, nullptr, 0.0, 0.0, npt, k, nkc, t0, ldt0, nep, p, a, inc,
                             e, w, npv, nlc, npb, lcids, pbids, epids, nsamples, exptimes, ldp, istar, weights, nk,
                             ng, nz, dk, kmin, kmax, dg, z_edges, obs, sigma, workspace, workspace_bytes, lnl, grad,
                             stream, basis, nb, true);
}

int rr_lnlike_split(int law, const double* ldc, int npar, const double* mu, const float* times_ff, double t_ref,
                    double t_absmax, int npt, const double* k, int nkc, const double* t0, int ldt0, int nep,
                    const double* p, const double* a, const double* inc, const double* e, const double* w, int npv,
                    int nlc, int npb, const int32_t* lcids, const int32_t* pbids, const int32_t* epids,
                    const int32_t* nsamples, const double* exptimes, const float* ldp, const float* istar,
                    const float* weights, int nk, int ng, int nz, double dk, double kmin, double kmax, double dg,
                    const double* z_edges, const double* obs, const double* sigma, void* workspace,
                    size_t workspace_bytes, double* lnl, double* grad, void* stream) {
  return lnlike_impl<float>(1, law, ldc, npar, mu, nullptr, times_ff, t_ref, t_absmax, npt, k, nkc, t0, ldt0, nep, p,
                            a, inc, e, w, npv, nlc, npb, lcids, pbids, epids, nsamples, exptimes, ldp, istar, weights,
                            nk, ng, nz, dk, kmin, kmax, dg, z_edges, obs, sigma, workspace, workspace_bytes, lnl,
                            grad, stream);
}

}  // extern "C"
