// FP64 transmission spectroscopy for the affine limb-darkening laws.
//
// The FP64 pipe bounds this path (1.7 lanes per clock and SM, against 24
// million outputs of the 100 pv x 200 channels x 1203 times workload), so the
// sums are ordered to need the fewest FP64 instructions.  Every affine law's
// profile is I_b(mu) = sum_j u_bj phi_j(mu) with a few fixed functions phi_j, so
// its LD means are sum_j u_bj B_j[g] with B_j = W(kmean) phi_j per parameter
// vector, and a channel's flux at a point
//   F_b = 1 - (1 / (istar_b ns)) sum_s I_b(z_s) area_b(s)
// (model_trspec.py:74-93) separates into the point's sums
//   Sin_j = sum_inside B_j(z_s) A,  Sout_j = sum_limb B_j(z_s) A,
//   Sd_j  = sum_limb B_j(z_s) dA/dk
// and the channel's numbers:
//   F_b = 1 - sum_j (u_bj / (istar_b ns)) (afac_b Sin_j + Sout_j + dk_b Sd_j).
// The prologue reduces NB columns instead of npb, and an output takes NB
// multiply-adds inside the star and 2 NB on the limb (3 and 6 for quadratic
// limb darkening), against three products per touched table row.
#pragma once
#include "rr_f64.cuh"
#include "rr_ts.cuh"

namespace rr {

constexpr int TS64_MAXNB = 5;
constexpr int TS64_R2 = 16;     // record fields 16..24: r^2(t)
constexpr int TS64_NB = 25;     // record field: NB, or 0 for a full LD-mean table
constexpr int TS64_CH = 64;     // channels staged at a time
// The pv's block of the LD-mean workspace, npb * ng doubles: B[NB][ng], then
// the channels' coefficients u[npb][NB].
__host__ __device__ inline bool ts64_fits(int nb, int npb, int ng) {
  return nb > 0 && nb <= TS64_MAXNB && (long long)nb * (ng + npb) <= (long long)npb * ng;
}

struct Ts64Smem {
  double S[3 * TS64_MAXNB][TS_TILE];   // Sin_j, Sout_j, Sd_j per point
  double cin[TS64_CH][TS64_MAXNB], cout[TS64_CH][TS64_MAXNB], dk[TS64_CH];
  int act[TS_TILE];                    // points with an overlapped sample
  int flags[TS_TILE / 32];             // per 32-point slot: 1 inside sums, 2 limb sums
  F64Disk disk;                        // at kmean
  float df[R2_N];
  int even;
};

// Once per block and pv: the constants of the record o.
__device__ __forceinline__ void ts64_stage(const TsArgs<double>& A, const double* o, Ts64Smem& S) {
  if (threadIdx.x == 0) {
    const float tb = fmaxf(fabsf((float)o[10]), fabsf((float)o[11])) + f32_of(A.exptime0);
    float sum = 0.0f;
#pragma unroll
    for (int m = R2_N - 1; m >= 0; --m) {
      S.df[m] = f32_of(o[TS64_R2 + m]);
      sum = fmaf(sum, tb, fabsf(S.df[m]));
    }
    S.even = r2_is_even(o + TS64_R2);
    const float marg = fmaf(4e-6f, sum, 2e-6f);
    f64_disk<true>(o[12], A.dg, marg, S.disk);
    // surely inside every channel's planet: z <= 1 - max k
    const float lim = f32_of(o[14]);
    S.disk.r2in = S.disk.fast && lim > 0.0f ? lim * lim - marg : -INFINITY;
  }
}

// One sample by the reference's own expressions: kmean <= 0 or >= 1, z = 0, NaN.
static __device__ __noinline__ bool ts64_general(const double* o, double inv_dg, int ng, double t, double& a,
                                                 double& dadk, int& gi, double& fr, bool& inner) {
  double c[10];
  for (int i = 0; i < 10; ++i) c[i] = o[i];
  return ts_sample<double>(t, c, o[12], o[13], inv_dg, ng, o[14], a, dadk, gi, fr, inner);
}

// Phase 1: the sums of the tile's point threadIdx.x into S (all threads of the block's 128).
template <int NB>
__device__ __forceinline__ void ts64_point(const TsArgs<double>& A, int pv, int pt, const double* o, Ts64Smem& S) {
  const int tid = threadIdx.x;
  double s[3][NB];
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int j = 0; j < NB; ++j) s[x][j] = 0.0;
  bool act = false;
  int fl = 0;
  if (pt < A.npt) {
    const double tc = ts_fold<double, false>(pt, A.times, nullptr, A.t0[pv], A.p[pv], o);
    if (o[10] <= tc && tc <= o[11]) {
      const F64Disk& K = S.disk;
      const double* B = A.ldm + (size_t)pv * A.npb * A.ng;
      const int ns = A.nsamples0;
      const double step = ns > 1 ? A.exptime0 / ns : 0.0, tc0 = ns > 1 ? tc - 0.5 * A.exptime0 : tc;
      for (int smp = 0; smp < ns; ++smp) {
        const double t = ns > 1 ? __fma_rn(f64_of_pos((float)smp + 0.5f), step, tc0) : tc;
        const float tf = f32_of(t);
        float rf = S.df[R2_N - 1];
#pragma unroll
        for (int m = R2_N - 2; m >= 0; --m) rf = fmaf(rf, tf, S.df[m]);
        if (rf > K.r2out) continue;
        const double r2 = r2_at(o + TS64_R2, S.even, t);
        double a, dadk = 0.0, fr;
        int gi;
        bool in;
        if (!K.fast || !f64_moderate(r2)) {
          if (!ts64_general(o, 1.0 / A.dg, A.ng, t, a, dadk, gi, fr, in)) continue;
        } else {
          const F64Root q = f64_root(r2);
          const double z = f64_sqrt(q);
          in = rf < K.r2in || z <= o[14];
          if (in) {
            a = K.area_in;
          } else {
            const F64Limb L = f64_limb<true>(K, r2, f64_rsqrt(q));
            a = L.area;
            dadk = __dmul_rn(__dadd_rn(K.k, K.k), L.kappa0);
            if (a == 0.0) continue;
          }
          f64_ld_pos(K, z, A.ng, gi, fr);
        }
        act = true;
        fl |= in ? 1 : 2;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const double l0 = __ldg(B + j * A.ng + gi);
          const double v = __fma_rn(fr, __dadd_rn(__ldg(B + j * A.ng + gi + 1), -l0), l0);
          if (in) {
            s[0][j] = __fma_rn(v, a, s[0][j]);
          } else {
            s[1][j] = __fma_rn(v, a, s[1][j]);
            s[2][j] = __fma_rn(v, dadk, s[2][j]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int j = 0; j < NB; ++j) S.S[x * NB + j][tid] = s[x][j];
  S.act[tid] = act;
  const int any = __reduce_or_sync(0xffffffffu, fl);
  if ((tid & 31) == 0) S.flags[tid >> 5] = any;
}

// Phase 2: warps over channels, lanes over the 32 points of a slot.
template <int NB>
__device__ __forceinline__ void ts64_channels(const TsArgs<double>& A, int pv, int pt0, const double* o, Ts64Smem& S) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
  const double* u = A.ldm + (size_t)pv * A.npb * A.ng + NB * A.ng;
  const double* ch = A.ch + (size_t)pv * A.npb * TS_CH;
  double* fpv = A.flux + (size_t)pv * A.npb * A.ldflux;
  const double inv_ns = 1.0 / (double)A.nsamples0;
  for (int b0 = 0; b0 < A.npb; b0 += TS64_CH) {
    const int nb = min(TS64_CH, A.npb - b0);
    if (b0 > 0) __syncthreads();   // the previous channels are consumed
    for (int i = tid; i < nb; i += blockDim.x) {
      const double* c = ch + (size_t)(b0 + i) * TS_CH;
      const double scale = -c[2] * inv_ns;
      S.dk[i] = c[1];
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double v = u[(size_t)(b0 + i) * NB + j] * scale;
        S.cout[i][j] = v;
        S.cin[i][j] = v * c[0];
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int q = 0; q < TS_TILE / 32; ++q) {
      const int pt = pt0 + 32 * q + lane, fl = S.flags[q];
      const bool act = S.act[32 * q + lane], st = pt < A.npt;
      double* dst = fpv + (size_t)(b0 + warp) * A.ldflux + pt;
      const size_t stride = (size_t)nwarps * A.ldflux;
      if (fl == 0) {
        for (int i = warp; i < nb; i += nwarps, dst += stride)
          if (st) __stcs(dst, 1.0);
        continue;
      }
      double s[3][NB];
#pragma unroll
      for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int j = 0; j < NB; ++j) s[x][j] = S.S[x * NB + j][32 * q + lane];
      if (fl == 1) {
        for (int i = warp; i < nb; i += nwarps, dst += stride) {
          double v = 1.0;
#pragma unroll
          for (int j = 0; j < NB; ++j) v = __fma_rn(S.cin[i][j], s[0][j], v);
          if (st) __stcs(dst, act ? v : 1.0);
        }
      } else {
        for (int i = warp; i < nb; i += nwarps, dst += stride) {
          const double dk = S.dk[i];
          double v = 1.0;
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            if (fl & 1) v = __fma_rn(S.cin[i][j], s[0][j], v);
            v = __fma_rn(S.cout[i][j], __fma_rn(dk, s[2][j], s[1][j]), v);
          }
          if (st) __stcs(dst, act ? v : 1.0);
        }
      }
    }
  }
}

// The tiles of `reach` (bits from tile tb0 on) of pv by the whole block.
template <int NB>
__device__ __forceinline__ void ts64_tiles(const TsArgs<double>& A, int pv, int tb0, unsigned reach, const double* o,
                                           Ts64Smem& S) {
  __syncthreads();
  ts64_stage(A, o, S);
  for (unsigned m = reach; m; m &= m - 1u) {
    const int pt0 = (tb0 + __ffs(m) - 1) * TS_TILE;
    __syncthreads();   // the previous tile's sums and channels are consumed
    ts64_point<NB>(A, pv, pt0 + threadIdx.x, o, S);
    __syncthreads();
    ts64_channels<NB>(A, pv, pt0, o, S);
  }
}

}  // namespace rr
