// The full RoadRunner model (pytransit/models/roadrunner/model_full.py:9-100)
// on the GPU: per-parameter-vector prologue kernels (limb-darkening means,
// orbit + bounding box) and the per-point flux kernels, plain FP64 and split
// precision.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "rr_device.cuh"
#include "rr_f64_points.cuh"
#include "rr_internal.h"
#include "rr_ts.cuh"

namespace rr {

constexpr int LDM_PBB = 4;      // passbands per block of the LD-means kernel
constexpr int MAX_NZ = 64;      // radial grid points staged in shared memory
constexpr int LDM_SCRATCH = 512;   // FP64 areas of the 2D table per chunk of rows (FP32 tables)

// ---------------------------------------------------------------------------
// Limb-darkening means, model_full.py:43-55:
//   ldm[pv, pb, :] = (1-ak) W[ik] @ ldp[pv, pb] + ak W[ik+1] @ ldp[pv, pb]
// with k = kw[pv * kw_stride], or a table built at k (calculate_weights_2d,
// common.py:153-185) when k is outside [kmin, kmax] (mode 0) or when ik+1
// would run past the table.  mode 1: the transmission-spectroscopy rule
// kmin <= k <= kmax_pv[pv] (model_trspec.py:48); mode 2: always the 2D table.
// One block per (pv, share of the passband groups): the k-interpolated weight
// slab (or the 2D table, computed once per block) is staged in shared memory,
// then the block walks its groups of LDM_PBB passbands and every (pb, g) output
// is a dot product from shared memory: ldm[pv][pb][g].
//
// In FP32, with one passband, bound by the latency of the slab's loads, the issue
// of their index arithmetic and the FP64 divisions that place k in the table.  So
// where rows are whole 16-byte words (VEC: nz a multiple of 4 (FP32) or 2 (FP64),
// W aligned) both go by words, four pairs of loads in flight and rows unpadded (at
// nz = 40 a word-wise dot product meets two-way bank conflicts); else element by
// element, rows padded to nz + 1.  The divisions are one warp's, and the scratch
// of the 2D table is small, so that the shared memory leaves 9 blocks on an SM.
// 4096 pv, ng = 100, nz = 40: 55.4 us by elements, 35.5 by words, 26.1 with
// 4 KB of scratch instead of 16, 17.9 with one warp's divisions, 15.5 with products
// in their place.  In FP64 the pipe bounds it: 49 -> 39 us for 1500 pv.
// ---------------------------------------------------------------------------
// Shared memory: the slab [ng][nz + 1 at most], the LD profiles [LDM_PBB][MAX_NZ at
// most] at the next 16-byte boundary, and the FP64 scratch.  Byte offsets:
template <typename R>
__host__ __device__ inline size_t ldm_profile_offset(int ng, int ldw) {
  return (sizeof(R) * (size_t)ng * ldw + 15) & ~size_t(15);
}
template <typename R>
__host__ __device__ inline size_t ldm_scratch_offset(int ng, int nz) {
  return ldm_profile_offset<R>(ng, nz + 1) + sizeof(R) * (size_t)LDM_PBB * MAX_NZ;
}

template <typename R, bool VEC>
__global__ void __launch_bounds__(128)
ldm_kernel(const R* __restrict__ ldp, int npb, int nz, const double* __restrict__ kw, int kw_stride,
           const R* __restrict__ W, int nk, int ng, double dk, double inv_dk, double kmin, double kmax,
           const double* __restrict__ ze, int mode, const double* __restrict__ kmax_pv,
           R* __restrict__ ldm) {
  extern __shared__ __align__(16) unsigned char ldm_smem[];
  R* Wk = reinterpret_cast<R*>(ldm_smem);                  // [ng][nz + 1]
  using W16 = typename Word16<R>::T;
  constexpr int PER = 16 / sizeof(R);
  const int ldw = VEC ? nz : nz + 1;
  R* l = reinterpret_cast<R*>(ldm_smem + ldm_profile_offset<R>(ng, ldw));   // [LDM_PBB][nz]
  const int pv = blockIdx.x;

  overlap_next();
  // the block's place in the table, by one warp: FP64 work
  __shared__ int s_ik;
  __shared__ R s_ak;
  const double k = kw[(size_t)pv * kw_stride];
  if (threadIdx.x < 32) {
    int ik = -1;
    R ak = R(0);
    double kup = (mode == 1) ? kmax_pv[pv] : kmax;
    if (mode != 2 && W != nullptr && kmin <= k && k <= kup) table_place(k, kmin, dk, inv_dk, nk, ik, ak);
    if (threadIdx.x == 0) { s_ik = ik; s_ak = ak; }
  }
  __syncthreads();
  const int ik = s_ik;
  if (ik >= 0) {
    const R ak = s_ak;
    const R* W0 = W + (size_t)ik * ng * nz;
    const R* W1 = W0 + (size_t)ng * nz;
    const R a1 = ak, a0 = R(1) - ak;
    if constexpr (VEC) {
      const W16 *V0 = reinterpret_cast<const W16*>(W0), *V1 = reinterpret_cast<const W16*>(W1);
      W16* S = reinterpret_cast<W16*>(Wk);
      const int n = ng * nz / PER;
      for (int i0 = threadIdx.x; i0 < n; i0 += 4 * 128) {
        W16 u[4], v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = min(i0 + q * 128, n - 1);
          u[q] = __ldg(V0 + i);
          v[q] = __ldg(V1 + i);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (i0 + q * 128 < n) S[i0 + q * 128] = Word16<R>::lerp(a0, u[q], a1, v[q]);
      }
    } else {
      for (int i = threadIdx.x; i < ng * nz; i += blockDim.x)
        Wk[(i / nz) * ldw + (i % nz)] = a0 * __ldg(W0 + i) + a1 * __ldg(W1 + i);
    }
  } else {
    // 2D table at this k (calculate_weights_2d, common.py:153-185) in FP64:
    // the areas A(ze_z) at every (g, z) in parallel, then per row the
    // differences w_z = A(ze_z) - A(ze_{z-1}) and their sum, normalised.  The
    // areas go to the table itself (FP64) or, for an FP32 table, to an FP64
    // scratch in chunks of rows, each row's sum in the word after it.
    const double gstep = (1.0 - 1e-7) / (double)(ng - 1);
    double* A2 = (sizeof(R) == 8) ? reinterpret_cast<double*>(Wk)
                                  : reinterpret_cast<double*>(ldm_smem + ldm_scratch_offset<R>(ng, nz));
    const int rows = (sizeof(R) == 8) ? ng : LDM_SCRATCH / (nz + 1);
    const int lda = (sizeof(R) == 8) ? ldw : nz + 1;
    for (int g0 = 0; g0 < ng; g0 += rows) {
      const int nr = min(rows, ng - g0);
      for (int i = threadIdx.x; i < nr * nz; i += blockDim.x) {
        const int g = g0 + i / nz, z = i % nz;
        const double gg = (g == ng - 1) ? 1.0 - 1e-7 : (double)g * gstep;
        A2[(size_t)(i / nz) * lda + z] = cci_acos(ze[z], k, gg * (1.0 + k));
      }
      __syncthreads();
      for (int rr = threadIdx.x; rr < nr; rr += blockDim.x) {
        double* a = A2 + (size_t)rr * lda;
        double s = a[0];
        for (int z = 1; z < nz; ++z) s += a[z] - a[z - 1];
        if constexpr (sizeof(R) == 8) {
          // in place: walk down so a[z-1] is still the area
          R* row = Wk + (size_t)(g0 + rr) * ldw;
          for (int z = nz - 1; z >= 1; --z) row[z] = (a[z] - a[z - 1]) / s;
          row[0] = a[0] / s;
        } else {
          a[nz] = s;
        }
      }
      __syncthreads();
      if constexpr (sizeof(R) == 4) {
        for (int i = threadIdx.x; i < nr * nz; i += blockDim.x) {
          const int rr = i / nz, z = i % nz;
          const double* a = A2 + (size_t)rr * lda;
          Wk[(size_t)(g0 + rr) * ldw + z] = (R)((z ? a[z] - a[z - 1] : a[0]) / a[nz]);
        }
        __syncthreads();
      }
    }
  }
  const int ngroups = (npb + LDM_PBB - 1) / LDM_PBB;
  for (int grp = blockIdx.y; grp < ngroups; grp += gridDim.y) {
    const int pb0 = grp * LDM_PBB;
    const int nb = min(LDM_PBB, npb - pb0);
    __syncthreads();   // the slab is complete; the previous group's l is no longer read
    for (int i = threadIdx.x; i < nb * nz; i += blockDim.x)
      l[i] = ldp[((size_t)pv * npb + pb0) * nz + i];
    __syncthreads();
    for (int j = threadIdx.x; j < nb * ng; j += blockDim.x) {
      const int b = j / ng, g = j % ng;
      const R* row = Wk + (size_t)g * ldw;
      const R* lb = l + b * nz;
      R d = R(0);
      if constexpr (VEC) {
        const W16 *rw = reinterpret_cast<const W16*>(row), *lw = reinterpret_cast<const W16*>(lb);
#pragma unroll 5
        for (int z = 0; z < nz / PER; ++z) Word16<R>::dot(d, rw[z], lw[z]);
      } else {
        for (int z = 0; z < nz; ++z) d += row[z] * lb[z];
      }
      ldm[((size_t)pv * npb + pb0 + b) * ng + g] = d;
    }
  }
  overlap_end();
}

// Blocks per pv of the LD-means kernel: the 2D table (mode 2) is costly FP64
// work (GB300's FP64 rate is 1/64 of FP32), built once per block, so all of a
// pv's passbands share one block; the 3D slab is a cheap lerp.
static dim3 ldm_grid(int npv, int npb, int mode) {
  const int ngroups = (npb + LDM_PBB - 1) / LDM_PBB;
  const int want = (mode == 2) ? 1 : (4096 + npv - 1) / npv;
  return dim3(npv, (unsigned)std::max(1, std::min(ngroups, want)));
}

// Host launcher of the LD-means kernel; dynamic shared memory above the default
// 48 KB (large ng) opts in to the larger carve-out first.
template <typename R>
static void launch_ldm_impl(const R* ldp, int npv, int npb, int nz, const double* kw, int kw_stride, const R* W,
                            int nk, int ng, double dk, double kmin, double kmax, const double* ze, int mode,
                            const double* kmax_pv, R* ldm, cudaStream_t s, bool overlap = false) {
  const size_t scratch = (sizeof(R) == 8) ? 0 : sizeof(double) * LDM_SCRATCH;
  const size_t bytes = ldm_scratch_offset<R>(ng, nz) + scratch;
  const bool vec = W && nz % (16 / sizeof(R)) == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
  auto fn = vec ? ldm_kernel<R, true> : ldm_kernel<R, false>;
  if (bytes > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (overlap)
    launch_overlap(fn, ldm_grid(npv, npb, mode), 128, bytes, s, ldp, npb, nz, kw, kw_stride, W, nk, ng, dk, 1.0 / dk, kmin, kmax,
                   ze, mode, kmax_pv, ldm);
  else
    fn<<<ldm_grid(npv, npb, mode), 128, bytes, s>>>(ldp, npb, nz, kw, kw_stride, W, nk, ng, dk, 1.0 / dk, kmin, kmax, ze, mode,
                                                    kmax_pv, ldm);
}
void launch_ldm_f32(const float* ldp, int npv, int npb, int nz, const double* kw, int kw_stride, const float* W,
                    int nk, int ng, double dk, double kmin, double kmax, const double* ze, int mode,
                    const double* kmax_pv, float* ldm, cudaStream_t s) {
  launch_ldm_impl<float>(ldp, npv, npb, nz, kw, kw_stride, W, nk, ng, dk, kmin, kmax, ze, mode, kmax_pv, ldm, s);
}
void launch_ldm_f64(const double* ldp, int npv, int npb, int nz, const double* kw, int kw_stride, const double* W,
                    int nk, int ng, double dk, double kmin, double kmax, const double* ze, int mode,
                    const double* kmax_pv, double* ldm, cudaStream_t s) {
  launch_ldm_impl<double>(ldp, npv, npb, nz, kw, kw_stride, W, nk, ng, dk, kmin, kmax, ze, mode, kmax_pv, ldm, s);
}

// ---------------------------------------------------------------------------
// Basis tables of an affine law: B[ik][b][g] = sum_z W[ik][g][z] phi_b(mu_z),
// one thread per (ik, g), FP64 (and an FP32 copy).
// ---------------------------------------------------------------------------
__global__ void basis_tables_kernel(int law, int nb, const double* __restrict__ mu, int nz,
                                    const double* __restrict__ W, int nk, int ng, double* __restrict__ B64,
                                    float* __restrict__ B32) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= nk * ng) return;
  const int ik = row / ng, g = row % ng;
  const double* w = W + (size_t)row * nz;
  for (int b = 0; b < nb; ++b) {
    double acc = 0.0;
    for (int z = 0; z < nz; ++z) acc += w[z] * basis_value(law, b, mu[z]);
    const size_t o = ((size_t)ik * nb + b) * ng + g;
    B64[o] = acc;
    if (B32) B32[o] = (float)acc;
  }
}

// LD means of an affine law from the basis tables, one block per pv:
//   ldm[pv, pb, g] = sum_b coef_b(pv, pb) ((1-ak) B[ik][b][g] + ak B[ik+1][b][g]),
// k, ik, ak as model_full.py:46-51.  Outside the 3D table (k outside
// [kmin, kmax], or ik+1 == nk) the 2D table at k is built row by row in FP64
// and applied to ldp, as the generic kernel does.
constexpr int MAX_BASIS = 16;

// Row g of the LD means of one pv for every passband from the 2D weight table
// built at k in FP64 (calculate_weights_2d, common.py:153-185): the k-outside-
// the-tables case of the affine-law kernels.  ldp_pv = the pv's [npb][nz]
// profiles, out = its [npb][ng] means.
template <typename R>
__device__ inline void ldm_direct_g(double k, int g, int ng, int nz, const double* __restrict__ ze,
                                    const R* ldp_pv, int npb, R* out) {
  const double gstep = (1.0 - 1e-7) / (double)(ng - 1);
  double gg = (double)g * gstep;
  if (g == ng - 1) gg = 1.0 - 1e-7;
  const double bb = gg * (1.0 + k);
  double w[64];
  double a0 = cci_acos(ze[0], k, bb), s = a0;
  w[0] = a0;
  for (int z = 1; z < nz; ++z) {
    const double a1 = cci_acos(ze[z], k, bb);
    w[z] = a1 - a0;
    a0 = a1;
    s += w[z];
  }
  for (int pb = 0; pb < npb; ++pb) {
    const R* l = ldp_pv + (size_t)pb * nz;
    double acc = 0.0;
    for (int z = 0; z < nz; ++z) acc += (w[z] / s) * (double)l[z];
    out[(size_t)pb * ng + g] = (R)acc;
  }
}

template <typename R>
__global__ void __launch_bounds__(128)
ldm_basis_kernel(int law, const double* __restrict__ ldc, int npar, int npb, const double* __restrict__ kw,
                 int kw_stride, const R* __restrict__ B, int nb, int nk, int ng, double dk, double kmin,
                 double kmax, const R* __restrict__ ldp, int nz, const double* __restrict__ ze,
                 R* __restrict__ ldm) {
  extern __shared__ __align__(16) unsigned char bsm[];
  R* coef = reinterpret_cast<R*>(bsm);                    // [npb][nb]
  __shared__ int s_ik;
  __shared__ double s_ak;
  const int pv = blockIdx.x;
  overlap_next();
  if (threadIdx.x == 0) {
    const double k = kw[(size_t)pv * kw_stride];
    int ik = -1;
    double ak = 0.0;
    if (kmin <= k && k <= kmax) {
      ik = (int)floor((k - kmin) / dk);
      ak = (k - kmin - ik * dk) / dk;
      if (ik + 1 >= nk || ik < 0) ik = -1;
    }
    s_ik = ik;
    s_ak = ak;
  }
  for (int pb = threadIdx.x; pb < npb; pb += blockDim.x) {
    double c[MAX_BASIS];
    basis_coefs(law, ldc + ((size_t)pv * npb + pb) * npar, npar, c);
    for (int b = 0; b < nb; ++b) coef[pb * nb + b] = (R)c[b];
  }
  __syncthreads();
  const int ik = s_ik;
  R* out = ldm + (size_t)pv * npb * ng;
  if (ik >= 0) {
    const R a1 = (R)s_ak, a0 = R(1) - (R)s_ak;
    const R* B0 = B + (size_t)ik * nb * ng;
    const R* B1 = B0 + (size_t)nb * ng;
    for (int j = threadIdx.x; j < npb * ng; j += blockDim.x) {
      const int pb = j / ng, g = j % ng;
      R d0 = R(0), d1 = R(0);
      for (int b = 0; b < nb; ++b) {
        d0 += coef[pb * nb + b] * __ldg(B0 + b * ng + g);
        d1 += coef[pb * nb + b] * __ldg(B1 + b * ng + g);
      }
      out[j] = a0 * d0 + a1 * d1;
    }
  } else {
    const double k = kw[(size_t)pv * kw_stride];
    for (int g = threadIdx.x; g < ng; g += blockDim.x)
      ldm_direct_g(k, g, ng, nz, ze, ldp + (size_t)pv * npb * nz, npb, out);
  }
  overlap_end();
}

// ---------------------------------------------------------------------------
// Orbit prologue, model_full.py:39-42 and 56-71, one thread per pv:
// validity, Taylor coefficients (solve2d), contact points (bounding_box).
// ---------------------------------------------------------------------------
struct OrbitArgs {
  const double *k, *t0, *p, *a, *inc, *e, *w, *exptimes;
  const int32_t *pbids, *epids, *nsamples;
  int nkc, ldt0, nep, npv, nlc, npb, nz;
  const void* ldp;       // validity probe ldp[pv, 0, 0] (double or float)
  int ldp_is_f32;
  // plain FP64 path
  double* orb64;
  // split path
  float *orb32, *lc32;
  const float* istar32;
  double t_ref, t_absmax;
  // split path with the LD profile evaluated here rather than read from
  // ldp / istar32 (the fused prologue): the law's coefficients ldc[npv, npb,
  // npar] and the mu grid, taken as FP32 as ld_tables_kernel<float> takes them
  int ld_direct, law, npar;
  const double *ldc, *mu;
};

constexpr int ORB_MAX_LDPAR = 4;   // coefficients per passband of the fused prologue's laws

// FP32 coefficients of (pv, pb), as ld_tables_kernel<float> converts them.
__device__ inline void ld_coefs_f32(const OrbitArgs& A, int pv, int pb, float* c) {
  const double* src = A.ldc + ((size_t)pv * A.npb + pb) * A.npar;
#pragma unroll
  for (int i = 0; i < ORB_MAX_LDPAR; ++i) c[i] = i < A.npar ? (float)src[i] : 0.0f;
}

// Plain FP64 path: validity, the FP64 Taylor coefficients, the contact times
// and r^2(t) of one pv.
__device__ __forceinline__ void orbit_pv_f64(const OrbitArgs& A, int pv) {
  const double a = A.a[pv], e = A.e[pv], p = A.p[pv];
  bool ldbad;
  if (A.ld_direct) {
    double u[ORB_MAX_LDPAR];
#pragma unroll
    for (int i = 0; i < ORB_MAX_LDPAR; ++i) u[i] = i < A.npar ? A.ldc[(size_t)pv * A.npb * A.npar + i] : 0.0;
    ldbad = isnan(ld_value<double>(A.law, A.mu[0], u, A.npar));
  } else {
    ldbad = A.ldp_is_f32 ? isnan(((const float*)A.ldp)[(size_t)pv * A.npb * A.nz])
                         : isnan(((const double*)A.ldp)[(size_t)pv * A.npb * A.nz]);
  }
  const bool valid = !(isnan(a) || a <= 1.0 || e < 0.0 || ldbad);
  double c[10] = {}, d[R2_N] = {};
  double t1 = 0.0, t4 = 0.0;
  const double k0 = A.k[(size_t)pv * A.nkc];
  if (valid) {
    solve2d_conj(p, a, A.inc[pv], e, A.w[pv], c);
    r2_poly(c, d);
    contact_times(k0, c, d, t1, t4);
  }
  double* o = A.orb64 + (size_t)pv * ORB64;
  for (int i = 0; i < 10; ++i) o[i] = c[i];
  o[10] = t1;
  o[11] = t4;
  o[12] = valid ? 1.0 : 0.0;
  for (int i = 0; i < R2_N; ++i) o[ORB64_R2 + i] = d[i];
}

// Split path: the FP32 orbit record [ORB32] and the per-light-curve records
// [nlc][LC32] of one pv.  The pointers are restrict-qualified locals and the
// light curves go in groups of four with every load of a group issued before
// its records are stored, so the dependent loads (epoch id -> zero epoch,
// passband id -> coefficients) of different light curves overlap; both
// contact points are bisected in one loop; records are written 16 bytes at a
// time.
constexpr int ORB_LCG = 2;   // light curves per load group

__device__ __forceinline__ void orbit_pv_split(const OrbitArgs& A, int pv) {
  const double* __restrict__ t0v = A.t0 + (size_t)pv * A.ldt0;
  const double* __restrict__ kv = A.k + (size_t)pv * A.nkc;
  const double* __restrict__ exptimes = A.exptimes;
  const int32_t* __restrict__ epids = A.epids;
  const int32_t* __restrict__ pbids = A.pbids;
  const int32_t* __restrict__ nsamples = A.nsamples;
  float4* __restrict__ o4 = reinterpret_cast<float4*>(A.orb32 + (size_t)pv * ORB32);
  float4* __restrict__ q4 = reinterpret_cast<float4*>(A.lc32 + (size_t)pv * A.nlc * LC32);
  const double a = A.a[pv], e = A.e[pv], p = A.p[pv], inc = A.inc[pv], w = A.w[pv];
  const double k0 = kv[0];
  bool ldbad;
  if (A.ld_direct) {
    float c[ORB_MAX_LDPAR];
    ld_coefs_f32(A, pv, 0, c);
    ldbad = isnan(ld_value<float>(A.law, (float)A.mu[0], c, A.npar));
  } else {
    ldbad = isnan(((const float*)A.ldp)[(size_t)pv * A.npb * A.nz]);
  }
  double d0max = 0.0;
  for (int ep = 0; ep < A.nep; ++ep) d0max = fmax(d0max, fabs(t0v[ep] - A.t_ref));
  const bool valid = !(isnan(a) || a <= 1.0 || e < 0.0 || ldbad);
  float cf[10];
  float t1 = 0.0f, t4 = 0.0f;
  if (valid) {
    solve2d_conj_f32(p, a, inc, e, w, cf);
    contact_points14_f32((float)k0, cf, t1, t4);
  } else {
    for (int i = 0; i < 10; ++i) cf[i] = 0.0f;
  }
  const float p_hi = __double2float_rn(p);
  const float p_lo = __double2float_rn(p - (double)p_hi);
  // Bound of |fast-test tc - true tc|: 2^-24 (4 (T + |d0|) + 2 p), doubled.
  const double err = ldexp(1.0, -21) * (A.t_absmax + d0max + p) + 1e-9;
  int flags = (valid ? FLAG_VALID : 0) | FLAG_MULTI;
  for (int lc0 = 0; lc0 < A.nlc; lc0 += ORB_LCG) {
    double d0[ORB_LCG], kk[ORB_LCG], ex[ORB_LCG];
    int pb[ORB_LCG], ns[ORB_LCG];
    float is[ORB_LCG];
#pragma unroll
    for (int j = 0; j < ORB_LCG; ++j) {
      const int lc = min(lc0 + j, A.nlc - 1);
      pb[j] = pbids[lc];
      ns[j] = nsamples[lc];
      ex[j] = exptimes[lc];
      d0[j] = t0v[epids[lc]] - A.t_ref;
      kk[j] = kv[A.nkc == A.npb ? pb[j] : 0];
      // a non-finite disk integral makes every in-box point NaN, as (istar - I A)/istar does
      if (A.ld_direct) {
        float c[ORB_MAX_LDPAR];
        ld_coefs_f32(A, pv, pb[j], c);
        ld_integral<float>(A.law, c, is[j]);
      } else {
        is[j] = A.istar32[(size_t)pv * A.npb + pb[j]];
      }
    }
#pragma unroll
    for (int j = 0; j < ORB_LCG; ++j) {
      const int lc = lc0 + j;
      if (lc >= A.nlc) break;
      const double pad = 0.003 + ex[j];
      const double lo = (double)t1 - pad, hi = (double)t4 + pad;
      if (hi + 2 * err >= 0.5 * p || lo - 2 * err <= -0.5 * p) flags |= FLAG_WIDE;
      const float d0h = __double2float_rn(d0[j]);
      const float kf = (float)kk[j];
      if (ns[j] == 1) flags &= ~FLAG_MULTI;
      float4* q = q4 + (size_t)lc * (LC32 / 4);
      // LC_FLO, LC_FHI, LC_D0H, LC_D0L | LC_LO, LC_HI, LC_K, LC_INV1PK | LC_INVIS, LC_EXPT, LC_INVNS, LC_NS | LC_PB
      q[0] = make_float4((float)(lo - err), (float)(hi + err), d0h, __double2float_rn(d0[j] - (double)d0h));
      q[1] = make_float4((float)lo, (float)hi, kf, 1.0f / (1.0f + kf));
      q[2] = make_float4(isfinite(is[j]) ? 1.0f / is[j] : __int_as_float(0x7fc00000), (float)ex[j],
                         1.0f / (float)ns[j], __int_as_float(ns[j]));
      q[3] = make_float4(__int_as_float(pb[j]), 0.0f, 0.0f, 0.0f);
    }
  }
  o4[0] = make_float4(cf[0], cf[1], cf[2], cf[3]);
  o4[1] = make_float4(cf[4], cf[5], cf[6], cf[7]);
  o4[2] = make_float4(cf[8], cf[9], p_hi, p_lo);
  o4[3] = make_float4(1.0f / p_hi, (float)err, __int_as_float(flags), 0.0f);
}

template <bool SPLIT>
__device__ __forceinline__ void orbit_pv(const OrbitArgs& A, int pv) {
  if (SPLIT)
    orbit_pv_split(A, pv);
  else
    orbit_pv_f64(A, pv);
}

template <bool SPLIT>
__global__ void orbit_kernel(OrbitArgs A) {
  overlap_next();
  const int pv = blockIdx.x * blockDim.x + threadIdx.x;
  if (pv < A.npv) orbit_pv<SPLIT>(A, pv);
}

// ---------------------------------------------------------------------------
// Fused split prologue for the affine laws with an analytic disk integral
// (uniform, linear, quadratic, quadratic-tri): one launch does the work of
// ld_tables_kernel<float>, ldm_basis_kernel<float> and orbit_kernel<true>
// (rrmodel.py:212-227 and model_full.py:39-71).
//   blocks [0, norb): orbit blocks.  Their first warp takes 32 pvs, one per
//     lane: the FP64 orbit chain is latency-bound, so it is spread thin, and
//     the lane evaluates the disk integral and the profile's validity probe
//     itself instead of waiting for the LD tables.
//   blocks [norb, ...): LD blocks, one warp per pv: the profile on the mu
//     grid and its disk integral (written out as ld_tables_kernel<float> does),
//     then the LD means from the basis tables, in FP32 (FP64 only for a pv
//     whose k lies outside the tables).
// The orbit blocks come first in the grid, so their chains start at once and
// the LD blocks fill the SMs around them.
// ---------------------------------------------------------------------------
constexpr int PRO_THREADS = 128;
constexpr int PRO_WARPS = PRO_THREADS / 32;
constexpr int PRO_MAX_COEF = 128;   // npb * npar and npb * nb floats staged per warp

struct ProArgs {
  OrbitArgs orb;
  int npv, npb, npar, nz, nb, nk, ng, law, kw_stride;
  const double *ldc, *mu, *kw, *ze;
  double kmin, kmax, dk, inv_dk;
  const float* B;
  float *ldp, *istar, *ldm;
};

// Basis coefficients of one passband from its FP32 coefficients
// (basis_coefs on the FP32 values).
__device__ inline void basis_coefs_f32(int law, const float* c, int npar, float* coef) {
  switch (law) {
    case LD_QUADRATIC_TRI: {
      const float a = sqrtf(c[0]), b = 2.0f * c[1];
      coef[0] = 1.0f; coef[1] = a * b; coef[2] = a * (1.0f - b);
      return;
    }
    default:
      coef[0] = 1.0f;
      for (int i = 1; i < basis_count(law, npar); ++i) coef[i] = c[i - 1];
  }
}

template <int LAW>
__global__ void __launch_bounds__(PRO_THREADS, 8) prologue_split_kernel(ProArgs P, int norb) {
  constexpr int NB = LAW == LD_UNIFORM ? 1 : (LAW == LD_LINEAR ? 2 : 3);   // basis_count of the law
  __shared__ float s_mu[MAX_NZ];
  __shared__ float s_c[PRO_WARPS][PRO_MAX_COEF];
  __shared__ float s_coef[PRO_WARPS][PRO_MAX_COEF];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x < norb) {
    if (warp != 0) return;
    const int pv = blockIdx.x * 32 + lane;
    if (pv < P.npv) orbit_pv<true>(P.orb, pv);
    return;
  }
  for (int i = threadIdx.x; i < P.nz; i += PRO_THREADS) s_mu[i] = (float)P.mu[i];
  __syncthreads();
  const int pv = ((int)blockIdx.x - norb) * PRO_WARPS + warp;
  if (pv >= P.npv) return;   // warp-uniform; no block barrier follows
  const int npb = P.npb, npar = P.npar, nz = P.nz, ng = P.ng;
  float* sc = s_c[warp];
  float* scf = s_coef[warp];
  for (int i = lane; i < npb * npar; i += 32) sc[i] = (float)P.ldc[(size_t)pv * npb * npar + i];
  __syncwarp();
  // the profile and its disk integral (ld_tables_kernel<float>), lanes over the mu grid
  float* ldp_pv = P.ldp + (size_t)pv * npb * nz;
  for (int pb = 0; pb < npb; ++pb)
    for (int z = lane; z < nz; z += 32) ldp_pv[pb * nz + z] = ld_value<float>(LAW, s_mu[z], sc + pb * npar, npar);
  for (int pb = lane; pb < npb; pb += 32) {
    float is;
    ld_integral<float>(LAW, sc + pb * npar, is);
    P.istar[(size_t)pv * npb + pb] = is;
    basis_coefs_f32(LAW, sc + pb * npar, npar, scf + pb * NB);
  }
  __syncwarp();
  // the LD means (ldm_basis_kernel): per grid column g the two k rows' basis
  // columns are blended once, e_b = (1 - ak) B[ik][b][g] + ak B[ik+1][b][g],
  // then each passband is an NB-term dot product with its coefficients
  float* out = P.ldm + (size_t)pv * npb * ng;
  const double k = P.kw[(size_t)pv * P.kw_stride];
  int ik = -1;
  float a1 = 0.0f;
  if (P.kmin <= k && k <= P.kmax) {
    const double t = (k - P.kmin) * P.inv_dk;
    const double fl = floor(t);
    ik = (int)fl;
    a1 = (float)(t - fl);
    if (ik + 1 >= P.nk || ik < 0) ik = -1;
  }
  if (ik >= 0) {
    const float a0 = 1.0f - a1;
    const float* B0 = P.B + (size_t)ik * NB * ng;
    const float* B1 = B0 + (size_t)NB * ng;
    for (int g = lane; g < ng; g += 32) {
      float eb[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) eb[b] = a0 * __ldg(B0 + b * ng + g) + a1 * __ldg(B1 + b * ng + g);
      for (int pb = 0; pb < npb; ++pb) {
        float d = 0.0f;
#pragma unroll
        for (int b = 0; b < NB; ++b) d = fmaf(scf[pb * NB + b], eb[b], d);
        out[(size_t)pb * ng + g] = d;
      }
    }
  } else {
    for (int g = lane; g < ng; g += 32) ldm_direct_g(k, g, ng, nz, P.ze, (const float*)ldp_pv, npb, out);
  }
}

// ---------------------------------------------------------------------------
// The same for the plain FP64 path: ld_tables_kernel<double>,
// ldm_basis_kernel<double> and orbit_kernel<false> in one launch.  The three
// took 74 + 63 + 53 us for 8192 pv x 4 passbands, each bound by the FP64 pipe
// or by one thread's chain of FP64 instructions; this one takes 54 us (77 pv
// x 1: 12 us, against 4 + 4 + 51).  Here the chains run beside
// the LD blocks; the two k rows of a basis column are blended once for all
// passbands (2 NB + NB npb FP64 instructions per column instead of
// 2 (NB + 1) npb); and the profile on the mu grid is evaluated only for a k
// outside the tables, which alone reads it.
// ---------------------------------------------------------------------------
struct Pro64Args {
  OrbitArgs orb;
  int npv, npb, npar, nz, nk, ng, kw_stride;
  const double *ldc, *mu, *kw, *ze;
  double kmin, kmax, dk;
  const double* B;
  double *ldp, *istar, *ldm;
};

template <int LAW>
__global__ void __launch_bounds__(PRO_THREADS) prologue_f64_kernel(Pro64Args P, int norb) {
  constexpr int NB = LAW == LD_UNIFORM ? 1 : (LAW == LD_LINEAR ? 2 : 3);   // basis_count of the law
  __shared__ double s_coef[PRO_WARPS][PRO_MAX_COEF];
  overlap_next();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x < norb) {
    if (warp != 0) return;
    const int pv = blockIdx.x * 32 + lane;
    if (pv < P.npv) orbit_pv<false>(P.orb, pv);
    return;
  }
  const int pv = ((int)blockIdx.x - norb) * PRO_WARPS + warp;
  if (pv >= P.npv) return;   // warp-uniform; no block barrier follows
  const int npb = P.npb, ng = P.ng;
  double* coef = s_coef[warp];
  const double* ldc = P.ldc + (size_t)pv * npb * P.npar;
  for (int pb = lane; pb < npb; pb += 32) {
    double is;
    ld_integral<double>(LAW, ldc + pb * P.npar, is);
    P.istar[(size_t)pv * npb + pb] = is;
    basis_coefs(LAW, ldc + pb * P.npar, P.npar, coef + pb * NB);
  }
  __syncwarp();
  double* out = P.ldm + (size_t)pv * npb * ng;
  const double k = P.kw[(size_t)pv * P.kw_stride];
  int ik = -1;
  double ak = 0.0;
  if (P.kmin <= k && k <= P.kmax) {   // model_full.py:46-51
    ik = (int)floor((k - P.kmin) / P.dk);
    ak = (k - P.kmin - ik * P.dk) / P.dk;
    if (ik + 1 >= P.nk || ik < 0) ik = -1;
  }
  if (ik >= 0) {
    const double a0 = 1.0 - ak;
    const double* B0 = P.B + (size_t)ik * NB * ng;
    const double* B1 = B0 + (size_t)NB * ng;
    for (int g = lane; g < ng; g += 32) {
      double eb[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) eb[b] = fma(ak, __ldg(B1 + b * ng + g), a0 * __ldg(B0 + b * ng + g));
      for (int pb = 0; pb < npb; ++pb) {
        double d = coef[pb * NB] * eb[0];
#pragma unroll
        for (int b = 1; b < NB; ++b) d = fma(coef[pb * NB + b], eb[b], d);
        out[(size_t)pb * ng + g] = d;
      }
    }
  } else {
    double* ldp_pv = P.ldp + (size_t)pv * npb * P.nz;
    for (int i = lane; i < npb * P.nz; i += 32)
      ldp_pv[i] = ld_value<double>(LAW, P.mu[i % P.nz], ldc + (i / P.nz) * P.npar, P.npar);
    __syncwarp();
    for (int g = lane; g < ng; g += 32) ldm_direct_g(k, g, ng, P.nz, P.ze, (const double*)ldp_pv, npb, out);
  }
}

// Parameter vector of a flux block: grid.y x grid.z cover npv beyond 65535.
__device__ __forceinline__ int block_pv() { return blockIdx.z * 65535 + blockIdx.y; }

struct FluxF64Args : F64Args {
  double* flux;
  int ldflux;
};

// The flux of one point at tc from conjunction, in or out of the box, by one
// thread.
__device__ __noinline__ double f64_point(const F64Args& A, int pv, int lc, double tc, const double* o) {
  const double pad = __dadd_rn(A.pad0, A.exptimes[lc]);
  if (!(__dsub_rn(o[10], pad) <= tc && tc <= __dadd_rn(o[11], pad))) return 1.0;
  F64Orbit P;
  f64_orbit(o, P);
  F64Lc R;
  f64_lc(A, pv, lc, P, R);
  return f64_point_value(R, P, F64Transit{o, A.ldm + ((size_t)pv * A.npb + R.pb) * A.ng, A.ng, A.dg}, tc);
}

// The plain FP64 flux: one thread per point, every point through the
// reference's fold.
__global__ void __launch_bounds__(256) flux_f64_kernel(const __grid_constant__ FluxF64Args A) {
  const int pv = block_pv();
  const int pt = blockIdx.x * blockDim.x + threadIdx.x;
  if (pt >= A.npt || pv >= A.npv) return;
  const double* o = A.orb64 + (size_t)pv * ORB64;
  double f = CUDART_NAN;
  if (o[12] != 0.0) {
    const int lc = A.lcids[pt];
    const double t = A.times[pt], p = A.p[pv];
    f = f64_point(A, pv, lc, __dsub_rn(t, f64_conjunction(t, A.t0[(size_t)pv * A.ldt0 + A.epids[lc]], p,
                                                          1.0f / (float)p)), o);
  }
  A.flux[(size_t)pv * A.ldflux + pt] = f;
}

// ---------------------------------------------------------------------------
// The FP64 flux with the fold once per 128-point tile and full warps on the
// in-transit samples.
//
// The reference's epoch and tc = t - (t0 + epoch p), each step rounded as in
// f64_conjunction, are non-decreasing in t.  So when a tile of one light curve
// has the same epoch at its earliest and latest time (tiles64: the FP64
// summaries of rr_time_tiles_f64), every point of it has that epoch and a tc
// between the two ends' tc: a range that misses the box makes every point 1.0
// without per-point work, and otherwise a point's tc is one subtraction.  A
// warp tests 32 tiles at once, one per lane, and writes the missed ones first.
//
// The kernel is bound by the FP64 pipe, where an instruction costs the same
// for 1 and for 32 active lanes.  So the in-box points of a warp's tiles are
// collected in shared memory (F64Queue), their samples are classified in FP32
// (f64_class), and full warps run the inner samples (16 FP64 instructions, 13
// for a circular orbit) and the limb samples (21 more) from two lists.  The
// terms of a point are then added in sample order by one lane: the same bits
// as flux_f64_kernel.  Blocks are single warps: warps of one block would wait
// for the one that holds the transits.
// ---------------------------------------------------------------------------
constexpr int F64_BLOCKS = 24;    // warps per SM: registers for 16, 20, 24, 28 give 532, 518, 499, 498 us on the
                                  // 8192 x 19,700 population

// The flux of the n queued points, all of light curve lc.  One copy of the
// code: inlined at the walk's call sites it does not fit the instruction cache.
static __device__ __noinline__ void f64_flux_flush(const FluxF64Args& A, const F64Orbit& P, F64Lc* recs, F64Queue& Q,
                                                   const double* o, int pv, int lc, int n) {
  const int nrec = min(A.nlc, F64_LC_SMEM);
  if (lc >= F64_LC_SMEM) {
    if ((threadIdx.x & 31) == 0) f64_lc(A, pv, lc, P, recs[nrec]);
    __syncwarp();
  }
  const F64Lc& R = recs[min(lc, nrec)];
  const F64Transit T{o, A.ldm + ((size_t)pv * A.npb + R.pb) * A.ng, A.ng, A.dg};
  double* row = A.flux + (size_t)pv * A.ldflux;
  f64_sums(R, P, T, Q, n,
           [&](int i, double D) {
             __stcs(row + Q.pt[i], f64_in_box(A, P, R, Q.tc[i]) ? T.value(R, D) : 1.0);
           },
           [](int, int) {});
}

struct F64FluxSink {
  static constexpr bool BY_LIGHT_CURVE = false;
  const FluxF64Args& A;
  const F64Orbit& P;
  F64Lc* recs;
  F64Queue& Q;
  const double* o;
  double* row;
  int pv;
  double fill;
  bool vec;

  __device__ __forceinline__ void tile(int p0, int q0, int q1) const {
    f64_fill_tile(row, A.npt, p0, q0, q1, fill, vec);
  }
  __device__ __forceinline__ void outside(int pt) const { __stcs(row + pt, 1.0); }
  __device__ __forceinline__ void flush(int lc, int n) const { f64_flux_flush(A, P, recs, Q, o, pv, lc, n); }
};

__global__ void __launch_bounds__(32, F64_BLOCKS)
flux_f64_culled_kernel(const __grid_constant__ FluxF64Args A, const double* tiles64, int slots) {
  __shared__ double o[ORB64];
  __shared__ F64Orbit P;
  __shared__ F64Queue Q;
  extern __shared__ __align__(16) unsigned char f64_smem[];
  F64Lc* recs = reinterpret_cast<F64Lc*>(f64_smem);   // [min(nlc, F64_LC_SMEM)], then one for a further light curve
  const int pv = block_pv();
  if (pv >= A.npv) return;
  const int lane = threadIdx.x;
  if (lane < ORB64) o[lane] = A.orb64[(size_t)pv * ORB64 + lane];
  __syncwarp();
  if (lane == 0) f64_orbit(o, P);
  __syncwarp();
  const bool valid = o[12] != 0.0;
  if (valid)
    for (int lc = lane; lc < min(A.nlc, F64_LC_SMEM); lc += 32) f64_lc(A, pv, lc, P, recs[lc]);
  __syncwarp();
  const F64FluxSink sink{A, P, recs, Q, o, A.flux + (size_t)pv * A.ldflux, pv, valid ? 1.0 : CUDART_NAN,
                   ((A.ldflux & 1) == 0) && ((reinterpret_cast<uintptr_t>(A.flux) & 15) == 0)};
  f64_walk(A, pv, tiles64, slots, valid, P, recs, Q, sink);
}

// ---------------------------------------------------------------------------
// Split-precision flux.  The output row of a pv is cut into warp tiles of
// 128 consecutive points.  A block stages the pv's orbit record and its
// per-light-curve records in shared memory, so the per-point work has no
// dependent global loads, and its warps take a range of tiles.  A warp tests
// 32 of its tiles at once against the precomputed tile summaries (one lane
// per tile): a tile of one light curve whose time range misses every box
// copy is one 16-byte store of ones per lane.  The other tiles load their
// FP32-pair times (slot q of lane l holds point q * 32 + l) and take the
// per-point path: the phase-folded time exact in FP32 pairs (error-free
// transformations) and the box test; then, in FP32, z, the LD-table lerp and
// the kite area on the limb; points with several samples go through the warp's
// queue (split_flush).  Output F = 1 - deficit.
// ---------------------------------------------------------------------------
constexpr int SPLIT_WARPS = 8;                // warps per block of the serving kernel
constexpr int SPLIT_PTS = 4;                 // points per lane
constexpr int WARP_TILE = 32 * SPLIT_PTS;    // points per warp tile

struct FluxSplitArgs {
  const float2* times_ff;
  const int32_t* lcids;
  const float *orb32, *lc32, *ldm;
  int npt, npv, npb, nlc, ng, ldflux;
  float inv_dg;
  void* flux;          // float or double rows (the kernel's OutT)
  int transits_only;   // store only the tiles that reach a transit (and invalid rows); the rest holds 1
};

// Output rows of the split flux kernels: FP32 (the split path's own type), or
// FP64 (the reference's output type, each FP32 result widened exactly).  A
// culled tile is one 16-byte store of the fill value per lane (FP32) or two
// (FP64).
template <typename OutT>
struct TileOut;

template <>
struct TileOut<float> {
  static __device__ __forceinline__ void fill(float* row, int tile, int lane, float v) {
    __stcs(reinterpret_cast<float4*>(row) + lane + (size_t)tile * (32 * 4 / 4), make_float4(v, v, v, v));
  }
};

template <>
struct TileOut<double> {
  static __device__ __forceinline__ void fill(double* row, int tile, int lane, float v) {
    const double d = v;
    double2* q = reinterpret_cast<double2*>(row) + (size_t)tile * 64 + 2 * lane;
    __stcs(q, make_double2(d, d));
    __stcs(q + 1, make_double2(d, d));
  }
};

constexpr int LC_SMEM = 64;                  // light-curve records staged in shared memory

struct WarpList {
  float tc[WARP_TILE];
  int lc[WARP_TILE];
  int off[WARP_TILE + 1];
  float acc[WARP_TILE], sum[WARP_TILE];
};

// Points of supersampled light curves that the fast fold puts in the box, kept
// by a warp over its tiles until they fill whole warps: at a 30-min cadence a
// tile that reaches a transit holds ~10 of them.
constexpr int SPLIT_Q = 160;       // points: what a tile adds to a queue of whole warps' remainder, and a warp
constexpr int SPLIT_ROWS = 10;     // rows of 32 samples evaluated at once
struct SplitQueue {
  int pt[SPLIT_Q];
  float term[SPLIT_ROWS * 32], z[SPLIT_ROWS * 32];
  unsigned short list[SPLIT_ROWS * 32];
};

// An output row of either type: one copy of the evaluating code serves both,
// so their values are the same bits.
struct SplitRow {
  char* p;
  bool f64;
  __device__ __forceinline__ void put(int pt, float v) const {
    if (f64) __stcs(reinterpret_cast<double*>(p) + pt, (double)v);
    else __stcs(reinterpret_cast<float*>(p) + pt, v);
  }
  __device__ __forceinline__ void fill(int tile, int lane, float v) const {
    if (f64) TileOut<double>::fill(reinterpret_cast<double*>(p), tile, lane, v);
    else TileOut<float>::fill(reinterpret_cast<float*>(p), tile, lane, v);
  }
};

// 1 / sqrt(x) of a normal x, without the scaling around it for denormals.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Evaluates and stores queued points, all of the light curve record R: whole
// warps of them, or, with all set, every one.  Returns the points left, moved
// to the front.
//
// The kernel is bound by instruction issue.  A lane takes a point, folds its
// time exactly and walks its samples, so that no index arithmetic is needed
// per sample; the samples of up to SPLIT_ROWS rows (32 points x 1 sample) get
// their separation and LD mean first, which finishes those inside the star,
// and the overlap area of the samples on the limb (about a third) follows in
// full warps from a list.  A point's terms are added as a tree within SPLIT_ROWS
// samples, and the sums of more rounds (each folds its points again) with their
// rounding errors.  4096 pv
// x 118,526 times x 10 samples: 2682 us with each tile's (point, sample) pairs
// by themselves (a binary search for a pair's point, the full area for every
// pair, a segmented shuffle sum), 1672 us.  Ranges of 64, 128 and 256 tiles per
// block instead of 32: 5, 8 and 14 % slower.
// MANY: more samples than SPLIT_ROWS, so that a point's sum so far and its error live across
// rounds (two registers that the common case does without).
template <bool MANY>
__device__ __forceinline__ int split_flush(const float2* __restrict__ times, const float* orb, const float* R,
                                           const float* ldm_pv, int ng, float inv_dg, SplitQueue& Q, int n, bool all,
                                           const SplitRow& row) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  __syncwarp();
  const float k = R[LC_K], ex = R[LC_EXPT], inv_ns = R[LC_INVNS], gsc = R[LC_INV1PK] * inv_dg, step = ex * inv_ns;
  const int ns_all = __float_as_int(R[LC_NS]);
  const float invis = R[LC_INVIS];
  const float* lda = ldm_pv + __float_as_int(R[LC_PB]) * ng;
  const float lim_out = 1.0f + k, lim_in = (k < 1.0f) ? 1.0f - k : -1.0f, area_in = float(PI) * k * k;
  const float4 ca = *reinterpret_cast<const float4*>(orb);
  const float4 cb = *reinterpret_cast<const float4*>(orb + 4);
  const float2 cc = *reinterpret_cast<const float2*>(orb + 8);
  const float4 fold = *reinterpret_cast<const float4*>(R), box = *reinterpret_cast<const float4*>(R + 4);
  const int take = all ? n : n & ~31;
  const int sc = MANY ? SPLIT_ROWS : max(ns_all, 1), nb = MANY ? 1 : SPLIT_ROWS / sc;   // samples, batches of 32 points at once
  for (int i0 = 0; i0 < take; i0 += 32 * nb) {
    float Dh = 0.0f, Dl = 0.0f;
    for (int s0 = 0; s0 < (MANY ? ns_all : 1); s0 += sc) {
      const int ns = MANY ? min(sc, ns_all - s0) : ns_all;
      int nlimb = 0, r = 0;
      for (int b = i0; b < min(take, i0 + 32 * nb); b += 32) {
        // time_offset = exptime ((isample - 0.5)/ns - 0.5), isample = s0 + s + 1
        float tb = 1e30f;   // no overlap past the last point and out of the box
        if (b + lane < take) {
          const float2 tt = __ldg(times + Q.pt[b + lane]);
          const float ne = floorf(fmaf(tt.x - fold.z, orb[12], 0.5f));
          const float tc = exact_tc(tt.x, tt.y, fold.z, fold.w, ne, orb[10], orb[11]);
          if (box.x <= tc && tc <= box.y) tb = fmaf(-0.5f, ex, tc);
        }
        float sf = (float)s0 + 0.5f;
#pragma unroll 2
        for (int s = 0; s < ns; ++s, r += 32, sf += 1.0f) {
          const float t = fmaf(sf, step, tb);
          const float x = fmaf(t, fmaf(t, fmaf(t, fmaf(t, cb.x, ca.w), ca.z), ca.y), ca.x);
          const float y = fmaf(t, fmaf(t, fmaf(t, fmaf(t, cc.y, cc.x), cb.w), cb.z), cb.y);
          const float r2 = fmaf(x, x, y * y);
          const float z = r2 * rsqrt_ftz(fmaxf(r2, 1e-30f));
          const bool ovl = z < lim_out, limb = ovl && !(z <= lim_in);
          const float gg = fminf(z, lim_out) * gsc;
          const int i = min(max((int)gg, 0), ng - 2);
          const float l0 = __ldg(lda + i), l1 = __ldg(lda + i + 1);
          const float mean = fmaf(gg - (float)i, l1 - l0, l0);
          Q.term[r + lane] = ovl ? (limb ? mean : mean * area_in) : 0.0f;
          const unsigned m = __ballot_sync(FULL, limb);
          if (limb) {
            const int at = nlimb + __popc(m & below);
            Q.z[at] = z;
            Q.list[at] = (unsigned short)(r + lane);
          }
          nlimb += __popc(m);
        }
      }
      __syncwarp();
      for (int j = lane; j < nlimb; j += 32) {
        const int f = Q.list[j];
        const float z = Q.z[j];
        float a;
        if (k <= 0.25f) {          // uniform over the warp
          a = kite_star_f32_smallk(k, z);
        } else if (k < 1.0f) {
          a = kite_star_f32(k, z);
        } else {
          float kap;
          a = ccia_star<float>(k, z, kap);
        }
        Q.term[f] *= a;
      }
      __syncwarp();
      const bool last = !MANY || s0 + ns >= ns_all;
      r = 0;
      for (int b = i0; b < min(take, i0 + 32 * nb); b += 32) {
        float D = 0.0f;
        const float* q = Q.term + r + lane;
        int s = 0;
        for (; s + 4 <= ns; s += 4) D += (q[32 * s] + q[32 * (s + 1)]) + (q[32 * (s + 2)] + q[32 * (s + 3)]);
        if (s < ns) {
          float rest = q[32 * s];
          if (s + 1 < ns) rest += q[32 * (s + 1)];
          if (s + 2 < ns) rest += q[32 * (s + 2)];
          D += rest;
        }
        r += 32 * max(ns, 0);
        if constexpr (MANY) {
          float sum, err;
          two_sum(Dh, D, sum, err);
          Dh = sum;
          Dl += err;
          D = Dh + Dl;
        }
        // in the box without overlap: 1, or NaN with a NaN disk integral
        const float f = 1.0f - D * invis * inv_ns;
        if (last && b + lane < take) {
          if (D != 0.0f) {
            row.put(Q.pt[b + lane], f);
          } else {
            const float2 tt = __ldg(times + Q.pt[b + lane]);
            const float ne = floorf(fmaf(tt.x - fold.z, orb[12], 0.5f));
            const float tc = exact_tc(tt.x, tt.y, fold.z, fold.w, ne, orb[10], orb[11]);
            row.put(Q.pt[b + lane], box.x <= tc && tc <= box.y ? f : 1.0f);
          }
        }
      }
      __syncwarp();
    }
  }
  const int left = n - take;
  if (take > 0 && lane < left) Q.pt[lane] = Q.pt[take + lane];
  __syncwarp();
  return left;
}

static __device__ __noinline__ int split_flush_many(const float2* __restrict__ times, const float* orb, const float* R,
                                                    const float* ldm_pv, int ng, float inv_dg, SplitQueue& Q, int n,
                                                    bool all, const SplitRow& row) {
  __builtin_assume(__isShared(&Q));
  __builtin_assume(__isShared(orb));
  return split_flush<true>(times, orb, R, ldm_pv, ng, inv_dg, Q, n, all, row);
}

union SplitSmem {   // a warp's lists: one of the two per pv
  WarpList l;
  SplitQueue q;
};
struct ListSmem {   // without the queue
  WarpList l;
};

// The cull test of one tile: its time range (from its summary) misses every
// box copy, the rounding of t - d0 and of j p covered by the error bound in
// the box (flo, fhi).  Tiles of several light curves never miss.
__device__ __forceinline__ bool split_tile_misses(const float4 tm, const float* LCR, float p_hi, float inv_p) {
  const int tlc = __float_as_int(tm.z);
  if (tlc < 0) return false;
  const float4 f = *reinterpret_cast<const float4*>(LCR + tlc * LC32);  // flo, fhi, d0h, d0l
  const float smin = tm.x - f.z, smax = tm.y - f.z;
  const float j0f = ceilf((smin - f.y) * inv_p);
  bool hit = false;
#pragma unroll
  for (int dj = -1; dj <= 1; ++dj) {
    const float jj = j0f + (float)dj;
    hit = hit || (fmaf(jj, p_hi, f.x) <= smax && fmaf(jj, p_hi, f.y) >= smin);
  }
  return !hit;
}

// The points of a tile of several light curves, a lane per point.
__device__ __noinline__ void split_mixed_tile(const float2* __restrict__ times, const int32_t* __restrict__ lcids,
                                              int npt, const float* orb, const float* LCR, const float* ldm_pv,
                                              int ng, float inv_dg, int pt0, const SplitRow& row) {
  const bool wide = __float_as_int(orb[14]) & FLAG_WIDE;
  for (int q = 0; q < SPLIT_PTS; ++q) {
    const int pt = pt0 + 32 * q;
    if (pt >= npt) continue;
    const float2 tt = __ldg(times + pt);
    const float* R = LCR + __ldg(lcids + pt) * LC32;
    const float sv = tt.x - R[LC_D0H], ne = floorf(fmaf(sv, orb[12], 0.5f)), r = fmaf(-ne, orb[10], sv);
    float f = 1.0f;
    if (wide || (r >= R[LC_FLO] && r <= R[LC_FHI])) {
      const float tc = exact_tc(tt.x, tt.y, R[LC_D0H], R[LC_D0L], ne, orb[10], orb[11]);
      if (R[LC_LO] <= tc && tc <= R[LC_HI]) {
        const float* lda = ldm_pv + __float_as_int(R[LC_PB]) * ng;
        const float k = R[LC_K];
        const int ns = __float_as_int(R[LC_NS]);
        float D = 0.0f, low = 0.0f;   // the sum and its error
        for (int s = 0; s < ns; ++s) {
          const float z = sep_c_f32(tc + R[LC_EXPT] * fmaf((float)s + 0.5f, R[LC_INVNS], -0.5f), orb);
          if (!(z < 1.0f + k)) continue;
          const float gg = z * R[LC_INV1PK] * inv_dg;
          const int i = min(max((int)gg, 0), ng - 2);
          const float l0 = __ldg(lda + i), l1 = __ldg(lda + i + 1);
          float kap;
          const float term = fmaf(gg - (float)i, l1 - l0, l0) * ccia_star<float>(k, z, kap);
          float sum, err;
          two_sum(D, term, sum, err);
          D = sum;
          low += err;
        }
        D += low;
        f = 1.0f - D * R[LC_INVIS] * R[LC_INVNS];
      }
    }
    row.put(pt, f);
  }
}

// A warp's tiles of a valid pv with supersampled light curves: the same cull
// test, every tile filled with 1, and of the tiles that reach a box the points
// that the fast FP32 fold (its error allowed for in flo, fhi) puts in it to the
// queue; their values overwrite the 1.  The queue is emptied at one place,
// before a tile, so that no values of a tile live across it.
__device__ __noinline__ void split_pv_multi(const FluxSplitArgs& A, int pv, int t_first, int t_step, int t_end,
                                            const float* orb, const float* LCR, SplitQueue& Q, bool out_f64) {
  const unsigned FULL = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __builtin_assume(__isShared(&Q));
  __builtin_assume(__isShared(orb));
  // locals: a field of A would be read again after every store to the row
  const int npt = A.npt, ng = A.ng;
  const float inv_dg = A.inv_dg;
  const float2* __restrict__ times = A.times_ff;
  const bool wide = __float_as_int(orb[14]) & FLAG_WIDE;
  const float p_hi = orb[10], inv_p = orb[12];
  const float* __restrict__ ldm_pv = A.ldm + (size_t)pv * A.npb * ng;
  const SplitRow row{static_cast<char*>(A.flux) + (size_t)pv * A.ldflux * (out_f64 ? 8 : 4), out_f64};
  const bool row_vec = ((A.ldflux & 3) == 0) && ((reinterpret_cast<uintptr_t>(A.flux) & 15) == 0);
  const bool fill = !A.transits_only;
  const float4* meta = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(times) + time_meta_offset(npt));
  const int tw0 = t_first + warp;
  const int ntl = tw0 < t_end ? (t_end - tw0 + t_step - 1) / t_step : 0;
  int n = 0, qlc = -1;   // queued points and their light curve
  int j0 = -32, mylc = 0;
  unsigned m = 0;        // tiles of the current group of 32 still to do
  for (;;) {
    while (m == 0 && j0 + 32 < ntl) {
      j0 += 32;
      const int jn = min(32, ntl - j0);
      bool cull = false;
      if (lane < jn) {
        const float4 tm = __ldg(meta + tw0 + (j0 + lane) * t_step);
        mylc = __float_as_int(tm.z);
        cull = !wide && split_tile_misses(tm, LCR, p_hi, inv_p);
      }
      const unsigned jmask = jn == 32 ? FULL : (1u << jn) - 1u;
      const unsigned cmask = __ballot_sync(FULL, cull) & jmask;
      m = ~cmask & jmask;
      for (unsigned c = fill ? jmask : m; c; c &= c - 1u) {
        const int tile = tw0 + (j0 + __ffs(c) - 1) * t_step;
        if (row_vec && (tile + 1) * WARP_TILE <= npt) {
          row.fill(tile, lane, 1.0f);
        } else {
          for (int q = 0; q < SPLIT_PTS; ++q)
            if (tile * WARP_TILE + 32 * q + lane < npt) row.put(tile * WARP_TILE + 32 * q + lane, 1.0f);
        }
      }
    }
    const bool done = m == 0;
    const int j = done ? 0 : __ffs(m) - 1;
    const int tlc = __shfl_sync(FULL, mylc, j);
    const bool all = done || tlc != qlc;
    if (n > 0 && (all || n > SPLIT_Q - WARP_TILE)) {
      const float* R = LCR + qlc * LC32;
      n = __float_as_int(R[LC_NS]) <= SPLIT_ROWS ? split_flush<false>(times, orb, R, ldm_pv, ng, inv_dg, Q, n, all, row)
                                                 : split_flush_many(times, orb, R, ldm_pv, ng, inv_dg, Q, n, all, row);
    }
    if (done) return;
    m &= m - 1u;
    const int p0 = (tw0 + (j0 + j) * t_step) * WARP_TILE;
    if (tlc < 0) {
      __syncwarp();   // after the fill
      split_mixed_tile(times, A.lcids, npt, orb, LCR, ldm_pv, ng, inv_dg, p0 + lane, row);
      continue;
    }
    qlc = tlc;
    // points p0 + 4 lane + q
    const float* R = LCR + tlc * LC32;
    const float4 f = *reinterpret_cast<const float4*>(R);       // flo, fhi, d0h, d0l
    const float lo = wide ? -INFINITY : f.x, hi = wide ? INFINITY : f.y;
    const int pt = p0 + SPLIT_PTS * lane;
    float t[SPLIT_PTS];
    if (p0 + WARP_TILE <= npt) {
      const float4 u = __ldg(reinterpret_cast<const float4*>(times + pt));
      const float4 v = __ldg(reinterpret_cast<const float4*>(times + pt) + 1);
      t[0] = u.x; t[1] = u.z; t[2] = v.x; t[3] = v.z;
    } else {
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q)
        t[q] = pt + q < npt ? __ldg(times + pt + q).x : __int_as_float(0x7fc00000);   // NaN: in no box
    }
    unsigned mask[SPLIT_PTS];
    unsigned in = 0;
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q) {
      const float sv = t[q] - f.z;
      const float r = fmaf(-floorf(fmaf(sv, inv_p, 0.5f)), p_hi, sv);
      const bool b = r >= lo && r <= hi;
      in |= b ? 1u << q : 0u;
      mask[q] = __ballot_sync(FULL, b);
    }
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q) {
      if (in >> q & 1u) Q.pt[n + __popc(mask[q] & ((1u << lane) - 1u))] = pt + q;
      n += __popc(mask[q]);
    }
  }
}

// Per-point path for one warp tile of one pv (slot q of lane l = the tile's
// point q * 32 + l).  Phase-folded times: for a tile of one light curve whose
// span plus box half-width is below p/2, the exact time of the tile's first
// point plus each point's (exact, small) offset from it; otherwise a fast
// FP32 test per point and the exact reduction for candidates.  Then the
// flux of the in-box points in place, skipping slots without an in-box point as a whole warp.  res[] holds
// 1.0 on entry and the flux of in-box points on exit.  With several samples per point
// the in-box points' (point, sample) pairs are spread over the lanes, whatever each light
// curve's count, and summed by a segmented shuffle reduction, over groups of 32 pairs and
// over 16 of those at a time, so that the error grows little with the samples.
__device__ __forceinline__ void split_tile_points(const float* __restrict__ orb, const float* __restrict__ LCR,
                                                  const float* __restrict__ ldm_pv, int ng, float inv_dg,
                                                  bool wide, float4 tm, const float* hi, const float* lo,
                                                  const int* lcv, WarpList& L, int lane, float* res) {
  const unsigned FULL = 0xffffffffu;
  const float p_hi = orb[10], p_lo = orb[11], inv_p = orb[12];
  const int tlc = __float_as_int(tm.z);
  float tcq[SPLIT_PTS];
  unsigned inb = 0;
  // Tile-relative times are exact whenever no point of the tile can fold onto
  // another box copy: span + |box| < p/2 (points whose offset crosses p/2 are
  // then out of box in both foldings).
  const float* RT = LCR + (tlc >= 0 ? tlc : 0) * LC32;
  if (!wide && tlc >= 0 && (tm.y - tm.x) + fmaxf(-RT[LC_LO], RT[LC_HI]) < 0.5f * p_hi) {
    const float* R = RT;
    const float h0 = __shfl_sync(FULL, hi[0], 0), l0 = __shfl_sync(FULL, lo[0], 0);
    const float n0 = floorf(fmaf(h0 - R[LC_D0H], inv_p, 0.5f));
    float tail0;
    const float s0 = exact_tc_pair(h0, l0, R[LC_D0H], R[LC_D0L], n0, p_hi, p_lo, tail0);
    const float blo = R[LC_LO], bhi = R[LC_HI];
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q) {
      // s0 + (hi - h0) is exact (Sterbenz) near the transit, where the two
      // nearly cancel; the small terms go in last: one rounding at |tc| scale
      tcq[q] = (s0 + (hi[q] - h0)) + ((lo[q] - l0) + tail0);
      if (lcv[q] >= 0 && blo <= tcq[q] && tcq[q] <= bhi) inb |= 1u << q;
    }
  } else {
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q) {
      tcq[q] = 0.0f;
      if (lcv[q] < 0) continue;
      const float4 f = *reinterpret_cast<const float4*>(LCR + lcv[q] * LC32);  // flo, fhi, d0h, d0l
      const float sv = hi[q] - f.z;
      const float n = floorf(fmaf(sv, inv_p, 0.5f));
      const float r = fmaf(-n, p_hi, sv);
      if (wide || (r >= f.x && r <= f.y)) {
        const float t = exact_tc(hi[q], lo[q], f.z, f.w, n, p_hi, p_lo);
        const float* R = LCR + lcv[q] * LC32;
        tcq[q] = t;
        if (R[LC_LO] <= t && t <= R[LC_HI]) inb |= 1u << q;
      }
    }
  }
  if (!__ballot_sync(FULL, inb != 0)) return;
  // Slot q of the lanes holds the tile's 32 consecutive points q*32 .. q*32+31:
  // a slot without an in-box point skips the per-point work as a whole warp.
  unsigned act = 0;
#pragma unroll
  for (int q = 0; q < SPLIT_PTS; ++q) act |= (__ballot_sync(FULL, inb >> q & 1u) ? 1u : 0u) << q;
  bool single;
  if (tlc >= 0) {
    single = __float_as_int(RT[LC_NS]) == 1;   // one light curve: warp-uniform
  } else {
    single = true;
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q)
      if (inb >> q & 1u) single = single && (__float_as_int(LCR[lcv[q] * LC32 + LC_NS]) == 1);
    single = __all_sync(FULL, single);
  }
  if (single) {
    // One sample per point.  A point whose planet disk is fully inside the
    // star (area pi k^2) is finished in place; points on the limb (kite area,
    // two atan2) are gathered into the warp's list and evaluated 32 at a time,
    // so that the costly branch runs with full lanes.
    unsigned limb = 0;
    float zq[SPLIT_PTS];
    if (tlc >= 0) {
      // one light curve in the tile: its record in registers, the orbit
      // polynomial from vector loads, z = r2 rsqrt(r2) (2 ulp)
      const float k = RT[LC_K], gsc = RT[LC_INV1PK] * inv_dg, invis = RT[LC_INVIS];
      const float* lda = ldm_pv + __float_as_int(RT[LC_PB]) * ng;
      const float lim_out = 1.0f + k, lim_in = (k < 1.0f) ? 1.0f - k : -1.0f;
      const float area_in = float(PI) * k * k * invis;
      const float4 ca = *reinterpret_cast<const float4*>(orb);
      const float4 cb = *reinterpret_cast<const float4*>(orb + 4);
      const float2 cc = *reinterpret_cast<const float2*>(orb + 8);
      // the active slots side by side, without per-lane branches until the
      // loads are issued, so that their dependent chains overlap
      float frq[SPLIT_PTS], l0q[SPLIT_PTS], l1q[SPLIT_PTS];
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q) {
        zq[q] = 0.0f;
        frq[q] = l0q[q] = l1q[q] = 0.0f;
        if (!(act >> q & 1u)) continue;   // warp-uniform
        const float t = tcq[q];
        const float x = fmaf(t, fmaf(t, fmaf(t, fmaf(t, cb.x, ca.w), ca.z), ca.y), ca.x);
        const float y = fmaf(t, fmaf(t, fmaf(t, fmaf(t, cc.y, cc.x), cb.w), cb.z), cb.y);
        const float r2 = fmaf(x, x, y * y);
        zq[q] = r2 > 0.0f ? r2 * rsqrtf(r2) : 0.0f;
        const float gg = fminf(zq[q], lim_out) * gsc;
        const int i = min(max((int)gg, 0), ng - 2);
        frq[q] = gg - (float)i;
        const bool need = (inb >> q & 1u) && zq[q] < lim_out;   // inner and limb points
        l0q[q] = need ? __ldg(lda + i) : 0.0f;
        l1q[q] = need ? __ldg(lda + i + 1) : 0.0f;
      }
      // classification by selects: no overlap (1 - 0 / istar, NaN with a NaN
      // istar), fully inside (the lerp times pi k^2 / istar) or on the limb
      const float res_out = 1.0f - 0.0f * invis;
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q) {
        if (!(act >> q & 1u)) continue;   // warp-uniform
        const bool in = inb >> q & 1u;
        const bool ovl = zq[q] < lim_out, inner = zq[q] <= lim_in;
        const float r_in = 1.0f - fmaf(frq[q], l1q[q] - l0q[q], l0q[q]) * area_in;
        res[q] = in ? (ovl ? (inner ? r_in : res[q]) : res_out) : res[q];
        limb |= (in && ovl && !inner) ? 1u << q : 0u;
      }
      // Limb points (kite area, two atan2) in place, slot by slot: the limb
      // points of a slot are consecutive in time (an ingress or an egress),
      // so one or two slots of a tile hold them all, and their table values
      // came with the loads above.  For k < 1 every limb point is in the kite
      // case, evaluated on all lanes of the slot without branches and kept
      // where the lane's point is on the limb.
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q) {
        if (!(act >> q & 1u)) continue;                    // warp-uniform
        if (!__ballot_sync(FULL, limb >> q & 1u)) continue;  // warp-uniform
        const bool lm = limb >> q & 1u;
        const float lerp = fmaf(frq[q], l1q[q] - l0q[q], l0q[q]);
        if (k <= 0.25f) {                                  // tile-uniform
          const float zz = lm ? zq[q] : 1.0f;              // an in-range z for the other lanes
          const float a = kite_star_f32_smallk(k, zz);
          res[q] = lm ? 1.0f - (lerp * a) * invis : res[q];
        } else if (k < 1.0f) {                             // tile-uniform
          const float zz = lm ? zq[q] : 1.0f;
          const float a = kite_star_f32(k, zz);
          res[q] = lm ? 1.0f - (lerp * a) * invis : res[q];
        } else if (lm) {
          float kap;
          res[q] = 1.0f - (lerp * ccia_star<float>(k, zq[q], kap)) * invis;
        }
      }
      return;
    } else {
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q) {
        zq[q] = 0.0f;
        if (!(inb >> q & 1u)) continue;
        const float* R = LCR + lcv[q] * LC32;
        const float k = R[LC_K];
        const float z = sep_c_f32(tcq[q], orb);
        zq[q] = z;
        if (!(z < 1.0f + k)) {                         // no overlap: 1 - 0 / istar (NaN with a NaN istar)
          res[q] = 1.0f - 0.0f * R[LC_INVIS];
          continue;
        }
        if (k < 1.0f && z <= 1.0f - k) {
          const float gg = z * R[LC_INV1PK] * inv_dg;
          int i = (int)gg;
          i = min(max(i, 0), ng - 2);
          const float fr = gg - (float)i;
          const float* lda = ldm_pv + __float_as_int(R[LC_PB]) * ng;
          const float l0 = __ldg(lda + i), l1 = __ldg(lda + i + 1);
          res[q] = 1.0f - fmaf(fr, l1 - l0, l0) * (float(PI) * k * k) * R[LC_INVIS];
        } else {
          limb |= 1u << q;
        }
      }
    }
    if (!__ballot_sync(FULL, limb != 0)) return;
    int nl = 0;
    int posq[SPLIT_PTS];
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q) {
      posq[q] = -1;
      if (!(act >> q & 1u)) continue;   // warp-uniform
      const bool in = limb >> q & 1u;
      const unsigned m = __ballot_sync(FULL, in);
      if (in) {
        const int pos = nl + __popc(m & ((1u << lane) - 1u));
        L.tc[pos] = zq[q];
        L.lc[pos] = lcv[q];
        posq[q] = pos;
      }
      nl += __popc(m);
    }
    __syncwarp();
    for (int i0 = 0; i0 < nl; i0 += 32) {
      const int it = i0 + lane;
      if (it < nl) {
        const float z = L.tc[it];
        const float* R = LCR + L.lc[it] * LC32;
        const float k = R[LC_K];
        const float gg = z * R[LC_INV1PK] * inv_dg;
        int i = (int)gg;
        i = min(max(i, 0), ng - 2);
        const float fr = gg - (float)i;
        const float* lda = ldm_pv + __float_as_int(R[LC_PB]) * ng;
        const float l0 = __ldg(lda + i), l1 = __ldg(lda + i + 1);
        float kap;
        L.acc[it] = fmaf(fr, l1 - l0, l0) * ccia_star<float>(k, z, kap);
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < SPLIT_PTS; ++q)
      if (posq[q] >= 0) res[q] = 1.0f - L.acc[posq[q]] * LCR[lcv[q] * LC32 + LC_INVIS];
    __syncwarp();
    return;
  }
  int nitems = 0;
  int posq[SPLIT_PTS];
#pragma unroll
  for (int q = 0; q < SPLIT_PTS; ++q) {
    const bool in = inb >> q & 1u;
    const unsigned m = __ballot_sync(FULL, in);
    posq[q] = -1;
    if (in) {
      const int pos = nitems + __popc(m & ((1u << lane) - 1u));
      L.tc[pos] = tcq[q];
      L.lc[pos] = lcv[q];
      L.acc[pos] = L.sum[pos] = 0.0f;
      posq[q] = pos;
    }
    nitems += __popc(m);
  }
  __syncwarp();
  // exclusive prefix sum of the sample counts -> L.off
  int total = 0;
  for (int c0 = 0; c0 < nitems; c0 += 32) {
    const int it = c0 + lane;
    const int v = (it < nitems) ? max(__float_as_int(LCR[L.lc[it] * LC32 + LC_NS]), 0) : 0;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(FULL, incl, d);
      if (lane >= d) incl += u;
    }
    if (it < nitems) L.off[it] = total + incl - v;
    total += __shfl_sync(FULL, incl, 31);
  }
  __syncwarp();
  for (int f0 = 0; f0 < total; f0 += 32) {
    const int f = f0 + lane;
    float d = 0.0f;
    int item = -1;
    if (f < total) {
      int lo_i = 0, hi_i = nitems - 1;   // largest item with off[item] <= f
      while (lo_i < hi_i) {
        const int mid = (lo_i + hi_i + 1) >> 1;
        if (L.off[mid] <= f) lo_i = mid; else hi_i = mid - 1;
      }
      item = lo_i;
      const int smp = f - L.off[item];
      const float* R = LCR + L.lc[item] * LC32;
      const float k = R[LC_K];
      // time_offset = exptime ((isample - 0.5)/ns - 0.5), isample = smp + 1
      const float t = L.tc[item] + R[LC_EXPT] * fmaf((float)smp + 0.5f, R[LC_INVNS], -0.5f);
      const float z = sep_c_f32(t, orb);
      if (z < 1.0f + k) {
        const float gg = z * R[LC_INV1PK] * inv_dg;
        const int i = min(max((int)gg, 0), ng - 2);
        const float* lda = ldm_pv + __float_as_int(R[LC_PB]) * ng;
        const float l0 = __ldg(lda + i), l1 = __ldg(lda + i + 1);
        float kap;
        d = fmaf(gg - (float)i, l1 - l0, l0) * ccia_star<float>(k, z, kap);
      }
    }
    // segmented sum over lanes holding the same item
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
      const float dv = __shfl_down_sync(FULL, d, dd);
      const int iv = __shfl_down_sync(FULL, item, dd);
      if (lane + dd < 32 && iv == item) d += dv;
    }
    const int before = __shfl_up_sync(FULL, item, 1);
    if (item >= 0 && (lane == 0 || before != item)) L.acc[item] += d;
    __syncwarp();
    if ((f0 & 511) == 480) {   // after 16 groups of pairs
      for (int it = lane; it < nitems; it += 32) {
        L.sum[it] += L.acc[it];
        L.acc[it] = 0.0f;
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int q = 0; q < SPLIT_PTS; ++q)
    if (posq[q] >= 0) {
      const float* R = LCR + lcv[q] * LC32;
      res[q] = 1.0f - (L.sum[posq[q]] + L.acc[posq[q]]) * R[LC_INVIS] * R[LC_INVNS];
    }
  __syncwarp();
}

// One block's share of one parameter vector: stage the pv's orbit and
// light-curve records in shared memory, then the warps loop over the tiles
// t_first + warp, + t_step, ... below t_end, 32 at a time: the cull tests,
// the stores of the culled tiles (walking the set bits of the cull mask),
// then the per-point path of the others.  Ends without a barrier: the caller
// synchronises before staging another pv.
template <typename OutT, bool QUEUE, typename Smem>
__device__ __forceinline__ void split_pv_tiles(const FluxSplitArgs& A, int pv, int t_first, int t_step, int t_end,
                                               float* recs, bool lc_in_smem, Smem* lists) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* lcg = A.lc32 + (size_t)pv * A.nlc * LC32;
  if (threadIdx.x < ORB32) recs[threadIdx.x] = __ldg(A.orb32 + (size_t)pv * ORB32 + threadIdx.x);
  if (lc_in_smem)
    for (int i = threadIdx.x; i < A.nlc * LC32; i += blockDim.x) recs[ORB32 + i] = __ldg(lcg + i);
  __syncthreads();
  const float* orb = recs;
  const float* LCR = lc_in_smem ? recs + ORB32 : lcg;
  const int flags = __float_as_int(orb[14]);
  const bool valid = flags & FLAG_VALID;
  const bool wide = flags & FLAG_WIDE;
  // Which way a pv's tiles go (block-uniform): through the queue over tiles where every
  // light curve is supersampled and most tiles are of one (light curves of two tiles
  // on average), else each tile by itself, which keeps tiles of single samples, or of
  // several light curves with counts of any kind, at their own cost.  Flux kernel, us,
  // queue / by itself: 4096 pv x 118,526 30-min times x 10 samples 1672 / 2682; a 30-min
  // light curve x 10 beside three 2-min ones (4096 x 21,015) 136 / 118; 60 light
  // curves of 73 points x 5 (1024 pv) 140 / 111; points of four interleaved, x 10,
  // (1024 x 19,700) 164 / 181.
  if constexpr (QUEUE) {
    if (valid && (flags & FLAG_MULTI) && A.npt >= 2LL * WARP_TILE * A.nlc) {
      split_pv_multi(A, pv, t_first, t_step, t_end, orb, LCR, lists[warp].q, sizeof(OutT) == 8);
      return;
    }
  }
  const float p_hi = orb[10], inv_p = orb[12];
  const float* ldm_pv = A.ldm + (size_t)pv * A.npb * A.ng;
  OutT* row = static_cast<OutT*>(A.flux) + (size_t)pv * A.ldflux;
  const bool row_vec = ((A.ldflux & 3) == 0) && ((reinterpret_cast<uintptr_t>(A.flux) & 15) == 0);
  const float4* meta = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(A.times_ff) +
                                                       time_meta_offset(A.npt));
  WarpList& L = lists[warp].l;
  const unsigned FULL = 0xffffffffu;
  // The warp's tiles are t_first + warp + j t_step, j < ntl.  A culled tile is
  // one 16-byte store of the fill value per lane (ones; NaN for an invalid
  // pv, whose tiles are all "culled"); only the row's last tile can be
  // partial, and it is stored point by point.
  const int tw0 = t_first + warp;
  const int ntl = tw0 < t_end ? (t_end - tw0 + t_step - 1) / t_step : 0;
  const int tile_part = (A.npt % WARP_TILE) ? A.npt / WARP_TILE : -1;
  const float fill = valid ? 1.0f : __int_as_float(0x7fc00000);
  for (int j0 = 0; j0 < ntl; j0 += 32) {
    const int tl = tw0 + (j0 + lane) * t_step;
    const bool cull = !valid || (!wide && j0 + lane < ntl && split_tile_misses(__ldg(meta + tl), LCR, p_hi, inv_p));
    const int jn = min(32, ntl - j0);
    const unsigned jmask = jn == 32 ? 0xffffffffu : (1u << jn) - 1u;
    const unsigned cmask = __ballot_sync(FULL, cull) & jmask;
    // the culled tiles first, walking the set bits of the mask (none when the
    // caller has already set the row to 1; an invalid pv's NaN always)
    for (unsigned m = (A.transits_only && valid) ? 0u : cmask; m; m &= m - 1u) {
      const int tile = tw0 + (j0 + __ffs(m) - 1) * t_step;
      if (row_vec && tile != tile_part) {
        TileOut<OutT>::fill(row, tile, lane, fill);
      } else {
        const int pt0 = tile * WARP_TILE + lane * SPLIT_PTS;
        for (int q = 0; q < SPLIT_PTS; ++q)
          if (pt0 + q < A.npt) __stcs(row + pt0 + q, (OutT)fill);
      }
    }
    // then the tiles that reach a box copy
    for (unsigned m = ~cmask & jmask; m; m &= m - 1u) {
      const int tile = tw0 + (j0 + __ffs(m) - 1) * t_step;
      // The tile reaches a box copy (the cull test above said so).  Slot q of
      // lane l holds point tile * 128 + q * 32 + l: each slot is 32
      // consecutive points, coalesced in its loads and stores.
      const float4 tm = __ldg(meta + tile);                 // tmin, tmax, lc
      const int ps0 = tile * WARP_TILE + lane;
      float res[SPLIT_PTS] = {1.0f, 1.0f, 1.0f, 1.0f};
      float hi[SPLIT_PTS], lo[SPLIT_PTS];
      int lcv[SPLIT_PTS];
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q) {
        const int pt = ps0 + 32 * q;
        if (pt < A.npt) {
          const float2 tt = __ldg(A.times_ff + pt);
          hi[q] = tt.x; lo[q] = tt.y; lcv[q] = __ldg(A.lcids + pt);
        } else {
          hi[q] = 0.0f; lo[q] = 0.0f; lcv[q] = -1;
        }
      }
      split_tile_points(orb, LCR, ldm_pv, A.ng, A.inv_dg, wide, tm, hi, lo, lcv, L, lane, res);
#pragma unroll
      for (int q = 0; q < SPLIT_PTS; ++q)
        if (ps0 + 32 * q < A.npt) __stcs(row + ps0 + 32 * q, (OutT)res[q]);
    }
  }
}

// Flux launch shape: blocks of FLUX_NW warps, each block one range of at
// most FLUX_CHUNK consecutive warp tiles of one pv (its warps interleaved over
// the range).  Grid: x = tile ranges, y/z = parameter vectors.  A small block
// gives its registers back as soon as its own tiles are done, so a range that
// holds a transit keeps no finished warps resident, and the hardware block
// scheduler balances the ranges over the SMs.  The pv's records are staged in
// dynamic shared memory sized to the light-curve count.
constexpr int FLUX_NW = 2;
constexpr int FLUX_CHUNK = 32;

// QUEUE: with the queue over tiles, whose call and shared memory cost the tiles by
// themselves 2 %: 117.4 us for 8192 x 19,700 points of single samples, 115.3 without.
template <bool LC_IN_SMEM, typename OutT, bool QUEUE>
__global__ void __launch_bounds__(FLUX_NW * 32, 16)
flux_split_kernel(const __grid_constant__ FluxSplitArgs A, int chunk) {
  __shared__ typename std::conditional<QUEUE, SplitSmem, ListSmem>::type lists[FLUX_NW];
  extern __shared__ __align__(16) float flux_recs[];
  const int pv = block_pv();
  if (pv >= A.npv) return;  // block-uniform
  const int ntiles = (A.npt + WARP_TILE - 1) / WARP_TILE;
  const int t0 = blockIdx.x * chunk;
  const int t1 = t0 + chunk < ntiles ? t0 + chunk : ntiles;
  split_pv_tiles<OutT, QUEUE>(A, pv, t0, FLUX_NW, t1, flux_recs, LC_IN_SMEM, lists);
}

// ---------------------------------------------------------------------------
// Serving: one persistent launch over the work items of many requests.  Each
// block takes the next item (request, pv range, tile range) from a device
// counter and runs split_pv_tiles for it with that request's tables; the
// item list is complete at launch, so no block ever waits for work.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SPLIT_WARPS * 32, 3)
serve_split_kernel(const rr_serve_request* __restrict__ reqs, const rr_serve_item* __restrict__ items,
                   const int* __restrict__ nitems_p, int* __restrict__ counter) {
  // the per-warp lists of the RoadRunner tiles and the tile state of the
  // transmission-spectroscopy tiles share the block's shared memory
  __shared__ union ServeSmem {
    SplitSmem lists[SPLIT_WARPS];
    TsSmem<float> ts;
  } U;
  __shared__ __align__(16) float recs[ORB32 + LC_SMEM * LC32];
  __shared__ int s_item;
  const int nitems = *nitems_p;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int it = s_item;
    __syncthreads();
    if (it >= nitems) return;
    const rr_serve_item w = items[it];
    const rr_serve_request& r = reqs[w.req];
    if (r.kind == 1) {
      // transmission spectroscopy (rr_ts.cuh): items span at most 32 tiles
      TsArgs<float> T{};
      T.times_ff = reinterpret_cast<const float2*>(r.times_ff);
      T.orb = r.orb32; T.ch = r.lc32; T.ldm = r.ldm; T.flux = r.flux;
      T.ldflux = r.ldflux; T.npt = r.npt; T.npb = r.npb; T.ng = r.ng; T.nsamples0 = r.nsamples0;
      T.exptime0 = (double)r.exptime0; T.dg = r.dg;
      for (int pv = w.pv0; pv < w.pv1; ++pv) {
        __syncthreads();   // the previous pv's record is consumed
        if (threadIdx.x < TS_ORB) recs[threadIdx.x] = __ldg(r.orb32 + (size_t)pv * TS_ORB + threadIdx.x);
        __syncthreads();
        ts_range<float, true>(T, pv, w.tile0, w.tile1, recs, U.ts);
      }
      __syncthreads();
      continue;
    }
    FluxSplitArgs A{};
    A.times_ff = reinterpret_cast<const float2*>(r.times_ff);
    A.lcids = r.lcids;
    A.orb32 = r.orb32; A.lc32 = r.lc32; A.ldm = r.ldm;
    A.npt = r.npt; A.npv = r.npv; A.npb = r.npb; A.nlc = r.nlc; A.ng = r.ng; A.ldflux = (int)r.ldflux;
    A.inv_dg = r.inv_dg; A.flux = r.flux;
    const bool lc_smem = r.nlc <= LC_SMEM;
    for (int pv = w.pv0; pv < w.pv1; ++pv) {
      split_pv_tiles<float, true>(A, pv, w.tile0, SPLIT_WARPS, w.tile1, recs, lc_smem, U.lists);
      __syncthreads();
    }
  }
}

bool prepare_f64_fused(int law, int npar, int npb, const double* ldc, const double* mu, const double* basis, int nb) {
  const bool analytic = law == LD_UNIFORM || law == LD_LINEAR || law == LD_QUADRATIC || law == LD_QUADRATIC_TRI;
  return analytic && basis && ldc && mu && nb > 0 && nb <= MAX_BASIS && nb == basis_count(law, npar) && npar >= 0 &&
         npar <= ORB_MAX_LDPAR && npb * nb <= PRO_MAX_COEF;
}

}  // namespace rr

using namespace rr;

extern "C" {

size_t rr_full_f64_workspace_bytes(int npv, int npb, int ng) {
  Carve c(nullptr);
  c.take<double>((size_t)npv * ORB64);
  c.take<double>((size_t)npv * npb * ng);
  return c.used + 256;
}

size_t rr_full_split_workspace_bytes(int npv, int npb, int nlc, int nep, int ng) {
  (void)nep;
  Carve c(nullptr);
  c.take<float>((size_t)npv * ORB32);
  c.take<float>((size_t)npv * nlc * LC32);
  c.take<float>((size_t)npv * npb * ng);
  return c.used + 256;
}

static int check_common(int npt, int nkc, int npv, int nlc, int npb, int nk, int ng, int nz, int ldflux) {
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npt < 0 || npv < 0 || nlc < 1 || npb < 1 || nk < 2 || ng < 2 || nz < 1 || nz > MAX_NZ ||
      nkc < 1 || ldflux < npt)
    return RR_ERR_ARG;
  return RR_OK;
}

struct SplitTables {
  float *orb, *lc, *ldm;
};

static SplitTables carve_split(void* ws, int npv, int npb, int nlc, int ng) {
  Carve cv(ws);
  SplitTables t;
  t.orb = cv.take<float>((size_t)npv * ORB32);
  t.lc = cv.take<float>((size_t)npv * nlc * LC32);
  t.ldm = cv.take<float>((size_t)npv * npb * ng);
  return t;
}

int rr_prepare_f64(const double* k, int nkc, const double* p, const double* a, const double* inc,
                   const double* e, const double* w, int npv, int npb, const double* ldp,
                   const double* weights, int nk, int ng, int nz, double dk, double kmin, double kmax,
                   const double* z_edges, void* workspace, size_t workspace_bytes, void* stream,
                   int law, const double* ldc, int npar, const double* basis, int nb) {
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npv < 0 || npb < 1 || nk < 2 || ng < 2 || nz < 1 || nz > MAX_NZ || nkc < 1) return RR_ERR_ARG;
  if (npv == 0) return RR_OK;
  if (workspace_bytes < rr_full_f64_workspace_bytes(npv, npb, ng)) return RR_ERR_WORKSPACE;
  cudaStream_t s = as_stream(stream);
  Carve cv(workspace);
  double* orb = cv.take<double>((size_t)npv * ORB64);
  double* ldm = cv.take<double>((size_t)npv * npb * ng);
  OrbitArgs oa{};
  oa.k = k; oa.p = p; oa.a = a; oa.inc = inc; oa.e = e; oa.w = w;
  oa.nkc = nkc; oa.npv = npv; oa.npb = npb; oa.nz = nz;
  oa.ldp = ldp; oa.ldp_is_f32 = 0; oa.orb64 = orb;
  orbit_kernel<false><<<(npv + 31) / 32, 32, 0, s>>>(oa);
  // beside the orbits' chains
  if (basis && nb > 0 && nb <= MAX_BASIS && ldc) {
    launch_overlap(ldm_basis_kernel<double>, npv, 128, sizeof(double) * npb * nb, s, law, ldc, npar, npb, k, nkc, basis, nb,
                   nk, ng, dk, kmin, kmax, ldp, nz, z_edges, ldm);
  } else {
    launch_ldm_impl<double>(ldp, npv, npb, nz, k, nkc, weights, nk, ng, dk, kmin, kmax, z_edges, 0, nullptr, ldm, s,
                            true);
  }
  return check_launch("rr_prepare_f64");
}

int rr_flux_f64_range(const double* times, int npt, const double* k, int nkc, const double* t0, int ldt0,
                      const double* p, int npv, int nlc, int npb, const int32_t* lcids, const int32_t* pbids,
                      const int32_t* epids, const int32_t* nsamples, const double* exptimes,
                      const double* istar, int ng, double dg, const void* workspace, int pv0, int pv1,
                      double* flux, int ldflux, void* stream) {
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npt < 0 || npv < 0 || nlc < 1 || npb < 1 || ng < 2 || nkc < 1 || ldflux < npt) return RR_ERR_ARG;
  if (pv0 < 0 || pv1 > npv || pv0 > pv1) return RR_ERR_ARG;
  if (pv1 == pv0 || npt == 0) return RR_OK;
  Carve cv(const_cast<void*>(workspace));
  double* orb = cv.take<double>((size_t)npv * ORB64);
  double* ldm = cv.take<double>((size_t)npv * npb * ng);
  // the range's parameters and records: the kernel indexes pv from 0 within it
  FluxF64Args fa{};
  fa.times = times; fa.k = k + (size_t)pv0 * nkc; fa.t0 = t0 + (size_t)pv0 * ldt0; fa.p = p + pv0;
  fa.exptimes = exptimes; fa.istar = istar + (size_t)pv0 * npb;
  fa.ldm = ldm + (size_t)pv0 * npb * ng; fa.orb64 = orb + (size_t)pv0 * ORB64;
  fa.lcids = lcids; fa.pbids = pbids; fa.epids = epids;
  fa.nsamples = nsamples; fa.npt = npt; fa.npv = pv1 - pv0; fa.nkc = nkc; fa.ldt0 = ldt0; fa.npb = npb;
  fa.nlc = nlc; fa.ng = ng; fa.ldflux = ldflux; fa.dg = dg; fa.nan_istar = true; fa.flux = flux;
  const int n = pv1 - pv0;
  dim3 fg((npt + 255) / 256, n < 65535 ? n : 65535, (n + 65534) / 65535);
  flux_f64_kernel<<<fg, 256, 0, as_stream(stream)>>>(fa);
  return check_launch("rr_flux_f64");
}

int rr_flux_f64_culled_range(const double* times, const double* tiles64, int npt, const double* k, int nkc,
                             const double* t0, int ldt0, const double* p, int npv, int nlc, int npb,
                             const int32_t* lcids, const int32_t* pbids, const int32_t* epids,
                             const int32_t* nsamples, const double* exptimes, const double* istar, int ng,
                             double dg, const void* workspace, int pv0, int pv1, double* flux, int ldflux,
                             void* stream) {
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npt < 0 || npv < 0 || nlc < 1 || npb < 1 || ng < 2 || nkc < 1 || ldflux < npt) return RR_ERR_ARG;
  if (pv0 < 0 || pv1 > npv || pv0 > pv1) return RR_ERR_ARG;
  if (pv1 == pv0 || npt == 0) return RR_OK;
  if (!tiles64) return RR_ERR_ARG;
  Carve cv(const_cast<void*>(workspace));
  double* orb = cv.take<double>((size_t)npv * ORB64);
  double* ldm = cv.take<double>((size_t)npv * npb * ng);
  FluxF64Args fa{};
  fa.times = times; fa.k = k + (size_t)pv0 * nkc; fa.t0 = t0 + (size_t)pv0 * ldt0; fa.p = p + pv0;
  fa.exptimes = exptimes; fa.istar = istar + (size_t)pv0 * npb;
  fa.ldm = ldm + (size_t)pv0 * npb * ng; fa.orb64 = orb + (size_t)pv0 * ORB64;
  fa.lcids = lcids; fa.pbids = pbids; fa.epids = epids;
  fa.nsamples = nsamples; fa.npt = npt; fa.npv = pv1 - pv0; fa.nkc = nkc; fa.ldt0 = ldt0; fa.npb = npb;
  fa.nlc = nlc; fa.ng = ng; fa.ldflux = ldflux; fa.dg = dg; fa.nan_istar = true; fa.flux = flux;
  const int n = pv1 - pv0;
  const int slots = f64_slots(npt, n, sm_count());
  dim3 fg(f64_warps(npt, slots), n < 65535 ? n : 65535, (n + 65534) / 65535);
  const size_t smem = sizeof(F64Lc) * (std::min(nlc, F64_LC_SMEM) + 1);
  flux_f64_culled_kernel<<<fg, 32, smem, as_stream(stream)>>>(fa, tiles64, slots);
  return check_launch("rr_flux_f64_culled");
}

int rr_flux_f64(const double* times, int npt, const double* k, int nkc, const double* t0, int ldt0,
                const double* p, int npv, int nlc, int npb, const int32_t* lcids, const int32_t* pbids,
                const int32_t* epids, const int32_t* nsamples, const double* exptimes,
                const double* istar, int ng, double dg, const void* workspace, double* flux, int ldflux,
                void* stream) {
  return rr_flux_f64_range(times, npt, k, nkc, t0, ldt0, p, npv, nlc, npb, lcids, pbids, epids, nsamples, exptimes,
                           istar, ng, dg, workspace, 0, npv, flux, ldflux, stream);
}

int rr_full_f64(const double* times, int npt, const double* k, int nkc, const double* t0, int ldt0,
                const double* p, const double* a, const double* inc, const double* e, const double* w,
                int npv, int nlc, int npb, const int32_t* lcids, const int32_t* pbids,
                const int32_t* epids, const int32_t* nsamples, const double* exptimes,
                const double* ldp, const double* istar, const double* weights, int nk, int ng, int nz,
                double dk, double kmin, double kmax, double dg, const double* z_edges, void* workspace,
                size_t workspace_bytes, double* flux, int ldflux, void* stream) {
  int st = check_common(npt, nkc, npv, nlc, npb, nk, ng, nz, ldflux);
  if (st) return st;
  if (npv == 0 || npt == 0) return RR_OK;
  if (workspace_bytes < rr_full_f64_workspace_bytes(npv, npb, ng)) return RR_ERR_WORKSPACE;
  st = rr_prepare_f64(k, nkc, p, a, inc, e, w, npv, npb, ldp, weights, nk, ng, nz, dk, kmin, kmax, z_edges,
                      workspace, workspace_bytes, stream, 0, nullptr, 0, nullptr, 0);
  if (st) return st;
  return rr_flux_f64(times, npt, k, nkc, t0, ldt0, p, npv, nlc, npb, lcids, pbids, epids, nsamples, exptimes,
                     istar, ng, dg, workspace, flux, ldflux, stream);
}

int rr_prepare_split(double t_ref, double t_absmax, const double* k, int nkc, const double* t0, int ldt0,
                     int nep, const double* p, const double* a, const double* inc, const double* e,
                     const double* w, int npv, int nlc, int npb, const int32_t* pbids, const int32_t* epids,
                     const int32_t* nsamples, const double* exptimes, const float* ldp, const float* istar,
                     const float* weights, int nk, int ng, int nz, double dk, double kmin, double kmax,
                     const double* z_edges, void* workspace, size_t workspace_bytes, void* stream, int law,
                     const double* ldc, int npar, const float* basis, int nb) {
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npv < 0 || nlc < 1 || npb < 1 || nk < 2 || ng < 2 || nz < 1 || nz > MAX_NZ || nkc < 1 || nep < 1 ||
      nep > ldt0)
    return RR_ERR_ARG;
  if (npv == 0) return RR_OK;
  if (workspace_bytes < rr_full_split_workspace_bytes(npv, npb, nlc, nep, ng)) return RR_ERR_WORKSPACE;
  cudaStream_t s = as_stream(stream);
  SplitTables t = carve_split(workspace, npv, npb, nlc, ng);
  OrbitArgs oa{};
  oa.k = k; oa.t0 = t0; oa.p = p; oa.a = a; oa.inc = inc; oa.e = e; oa.w = w; oa.exptimes = exptimes;
  oa.pbids = pbids; oa.epids = epids; oa.nsamples = nsamples;
  oa.nkc = nkc; oa.ldt0 = ldt0; oa.nep = nep; oa.npv = npv; oa.nlc = nlc; oa.npb = npb; oa.nz = nz;
  oa.ldp = ldp; oa.ldp_is_f32 = 1; oa.orb32 = t.orb; oa.lc32 = t.lc;
  oa.istar32 = istar; oa.t_ref = t_ref; oa.t_absmax = t_absmax;
  orbit_kernel<true><<<(npv + 31) / 32, 32, 0, s>>>(oa);
  // beside the orbits' chains
  if (basis && nb > 0 && nb <= MAX_BASIS && ldc) {
    launch_overlap(ldm_basis_kernel<float>, npv, 128, sizeof(float) * npb * nb, s, law, ldc, npar, npb, k, nkc, basis, nb,
                   nk, ng, dk, kmin, kmax, ldp, nz, z_edges, t.ldm);
  } else {
    launch_ldm_impl<float>(ldp, npv, npb, nz, k, nkc, weights, nk, ng, dk, kmin, kmax, z_edges, 0, nullptr, t.ldm, s,
                            true);
  }
  return check_launch("rr_prepare_split");
}

int rr_prepare_split_ld(double t_ref, double t_absmax, const double* k, int nkc, const double* t0, int ldt0,
                        int nep, const double* p, const double* a, const double* inc, const double* e,
                        const double* w, int npv, int nlc, int npb, const int32_t* pbids, const int32_t* epids,
                        const int32_t* nsamples, const double* exptimes, int law, const double* ldc, int npar,
                        const double* mu, int nz, const float* basis, int nb, const float* weights, int nk, int ng,
                        double dk, double kmin, double kmax, const double* z_edges, float* ldp, float* istar,
                        void* workspace, size_t workspace_bytes, void* stream) {
  const bool analytic = law == LD_UNIFORM || law == LD_LINEAR || law == LD_QUADRATIC || law == LD_QUADRATIC_TRI;
  const bool fused = analytic && basis && ldc && mu && nb > 0 && nb <= MAX_BASIS && nb == basis_count(law, npar) &&
                     npar >= 0 && npar <= ORB_MAX_LDPAR && npb * npar <= PRO_MAX_COEF && npb * nb <= PRO_MAX_COEF;
  if (!fused) {
    int st = rr_ld_tables_f32(law, ldc, npv, npb, npar, mu, nz, ldp, istar, stream);
    if (st) return st;
    return rr_prepare_split(t_ref, t_absmax, k, nkc, t0, ldt0, nep, p, a, inc, e, w, npv, nlc, npb, pbids, epids,
                            nsamples, exptimes, ldp, istar, weights, nk, ng, nz, dk, kmin, kmax, z_edges, workspace,
                            workspace_bytes, stream, law, ldc, npar, basis, nb);
  }
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npv < 0 || nlc < 1 || npb < 1 || nk < 2 || ng < 2 || nz < 1 || nz > MAX_NZ || nkc < 1 || nep < 1 ||
      nep > ldt0 || !ldp || !istar)
    return RR_ERR_ARG;
  if (npv == 0) return RR_OK;
  if (workspace_bytes < rr_full_split_workspace_bytes(npv, npb, nlc, nep, ng)) return RR_ERR_WORKSPACE;
  SplitTables t = carve_split(workspace, npv, npb, nlc, ng);
  ProArgs P{};
  OrbitArgs& oa = P.orb;
  oa.k = k; oa.t0 = t0; oa.p = p; oa.a = a; oa.inc = inc; oa.e = e; oa.w = w; oa.exptimes = exptimes;
  oa.pbids = pbids; oa.epids = epids; oa.nsamples = nsamples;
  oa.nkc = nkc; oa.ldt0 = ldt0; oa.nep = nep; oa.npv = npv; oa.nlc = nlc; oa.npb = npb; oa.nz = nz;
  oa.ldp = nullptr; oa.ldp_is_f32 = 1; oa.orb32 = t.orb; oa.lc32 = t.lc;
  oa.istar32 = nullptr; oa.t_ref = t_ref; oa.t_absmax = t_absmax;
  oa.ld_direct = 1; oa.law = law; oa.npar = npar; oa.ldc = ldc;
  P.npv = npv; P.npb = npb; P.npar = npar; P.nz = nz; P.nb = nb; P.nk = nk; P.ng = ng; P.law = law;
  P.kw_stride = nkc; P.ldc = ldc; P.mu = mu; P.kw = k; P.ze = z_edges;
  P.kmin = kmin; P.kmax = kmax; P.dk = dk; P.inv_dk = 1.0 / dk;
  P.B = basis; P.ldp = ldp; P.istar = istar; P.ldm = t.ldm;
  oa.mu = mu;
  cudaStream_t s = as_stream(stream);
  const int norb = (npv + 31) / 32;
  const int nld = (npv + PRO_WARPS - 1) / PRO_WARPS;
  switch (law) {
    case LD_UNIFORM: prologue_split_kernel<LD_UNIFORM><<<norb + nld, PRO_THREADS, 0, s>>>(P, norb); break;
    case LD_LINEAR: prologue_split_kernel<LD_LINEAR><<<norb + nld, PRO_THREADS, 0, s>>>(P, norb); break;
    case LD_QUADRATIC: prologue_split_kernel<LD_QUADRATIC><<<norb + nld, PRO_THREADS, 0, s>>>(P, norb); break;
    default: prologue_split_kernel<LD_QUADRATIC_TRI><<<norb + nld, PRO_THREADS, 0, s>>>(P, norb); break;
  }
  return check_launch("rr_prepare_split_ld");
}

int rr_prepare_f64_ld(const double* k, int nkc, const double* p, const double* a, const double* inc, const double* e,
                      const double* w, int npv, int npb, int law, const double* ldc, int npar, const double* mu,
                      int nz, const double* basis, int nb, const double* weights, int nk, int ng, double dk,
                      double kmin, double kmax, const double* z_edges, double* ldp, double* istar, void* workspace,
                      size_t workspace_bytes, void* stream) {
  if (!prepare_f64_fused(law, npar, npb, ldc, mu, basis, nb)) {
    const int st = rr_ld_tables_f64(law, ldc, npv, npb, npar, mu, nz, ldp, istar, stream);
    if (st) return st;
    return rr_prepare_f64(k, nkc, p, a, inc, e, w, npv, npb, ldp, weights, nk, ng, nz, dk, kmin, kmax, z_edges,
                          workspace, workspace_bytes, stream, law, ldc, npar, basis, nb);
  }
  if (nkc > 1 && nkc != npb) return RR_ERR_SHAPE;
  if (npv < 0 || npb < 1 || nk < 2 || ng < 2 || nz < 1 || nz > MAX_NZ || nkc < 1 || !ldp || !istar) return RR_ERR_ARG;
  if (npv == 0) return RR_OK;
  if (workspace_bytes < rr_full_f64_workspace_bytes(npv, npb, ng)) return RR_ERR_WORKSPACE;
  Carve cv(workspace);
  Pro64Args P{};
  OrbitArgs& oa = P.orb;
  oa.orb64 = cv.take<double>((size_t)npv * ORB64);
  P.ldm = cv.take<double>((size_t)npv * npb * ng);
  oa.k = k; oa.p = p; oa.a = a; oa.inc = inc; oa.e = e; oa.w = w;
  oa.nkc = nkc; oa.npv = npv; oa.npb = npb; oa.nz = nz;
  oa.ld_direct = 1; oa.law = law; oa.npar = npar; oa.ldc = ldc; oa.mu = mu;
  P.npv = npv; P.npb = npb; P.npar = npar; P.nz = nz; P.nk = nk; P.ng = ng; P.kw_stride = nkc;
  P.ldc = ldc; P.mu = mu; P.kw = k; P.ze = z_edges; P.kmin = kmin; P.kmax = kmax; P.dk = dk;
  P.B = basis; P.ldp = ldp; P.istar = istar;
  cudaStream_t s = as_stream(stream);
  const int norb = (npv + 31) / 32, nblk = norb + (npv + PRO_WARPS - 1) / PRO_WARPS;
  switch (law) {
    case LD_UNIFORM: prologue_f64_kernel<LD_UNIFORM><<<nblk, PRO_THREADS, 0, s>>>(P, norb); break;
    case LD_LINEAR: prologue_f64_kernel<LD_LINEAR><<<nblk, PRO_THREADS, 0, s>>>(P, norb); break;
    case LD_QUADRATIC: prologue_f64_kernel<LD_QUADRATIC><<<nblk, PRO_THREADS, 0, s>>>(P, norb); break;
    default: prologue_f64_kernel<LD_QUADRATIC_TRI><<<nblk, PRO_THREADS, 0, s>>>(P, norb); break;
  }
  return check_launch("rr_prepare_f64_ld");
}

int rr_flux_split(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb, int ng,
                  double dg, const void* workspace, float* flux, int ldflux, void* stream) {
  return rr_flux_split_range(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, 0, npv, flux, ldflux, stream);
}

static int flux_split_args(int npt, int npv, int nlc, int npb, int ng, int pv0, int pv1, int ldflux) {
  if (npt < 0 || npv < 0 || nlc < 1 || npb < 1 || ng < 2 || ldflux < npt) return RR_ERR_ARG;
  if (pv0 < 0 || pv1 > npv || pv0 > pv1) return RR_ERR_ARG;
  return RR_OK;
}

static int flux_split_launch(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb,
                             int ng, double dg, const void* workspace, int pv0, int pv1, void* flux, int ldflux,
                             void* stream, int kind) {
  const bool transits_only = kind & RR_ROWS_TRANSITS, out_f64 = kind & RR_ROWS_F64;
  const int st = flux_split_args(npt, npv, nlc, npb, ng, pv0, pv1, ldflux);
  if (st != RR_OK) return st;
  if (pv1 == pv0 || npt == 0) return RR_OK;
  SplitTables t = carve_split(const_cast<void*>(workspace), npv, npb, nlc, ng);
  FluxSplitArgs fa{};
  fa.times_ff = reinterpret_cast<const float2*>(times_ff);
  fa.lcids = lcids;
  // the range's records: the kernel indexes pv from 0 within the range
  fa.orb32 = t.orb + (size_t)pv0 * ORB32;
  fa.lc32 = t.lc + (size_t)pv0 * nlc * LC32;
  fa.ldm = t.ldm + (size_t)pv0 * npb * ng;
  npv = pv1 - pv0;
  fa.npt = npt; fa.npv = npv; fa.npb = npb; fa.nlc = nlc; fa.ng = ng; fa.ldflux = ldflux;
  fa.inv_dg = (float)(1.0 / dg); fa.flux = flux; fa.transits_only = transits_only;
  // tile ranges of FLUX_CHUNK tiles, shorter when the launch would otherwise
  // have fewer than about four blocks per resident warp slot (SMs x 32)
  const int ntiles = (npt + WARP_TILE - 1) / WARP_TILE;
  long long chunk = (long long)ntiles * npv / (4LL * sm_count() * 32);
  chunk = chunk < 1 ? 1 : (chunk > FLUX_CHUNK ? FLUX_CHUNK : chunk);
  const int bx = (int)((ntiles + chunk - 1) / chunk);
  dim3 fg((unsigned)bx, npv < 65535 ? npv : 65535, (npv + 65534) / 65535);
  const bool lc_smem = nlc <= LC_SMEM;
  const size_t smem = sizeof(float) * (ORB32 + (lc_smem ? (size_t)nlc * LC32 : 0));
  cudaStream_t s = as_stream(stream);
  const bool queue = !(kind & RR_ROWS_TILES) && npt >= 2LL * WARP_TILE * nlc;
  auto fn = flux_split_kernel<false, float, false>;
  if (queue)
    fn = out_f64 ? (lc_smem ? flux_split_kernel<true, double, true> : flux_split_kernel<false, double, true>)
                 : (lc_smem ? flux_split_kernel<true, float, true> : flux_split_kernel<false, float, true>);
  else
    fn = out_f64 ? (lc_smem ? flux_split_kernel<true, double, false> : flux_split_kernel<false, double, false>)
                 : (lc_smem ? flux_split_kernel<true, float, false> : flux_split_kernel<false, float, false>);
  fn<<<fg, FLUX_NW * 32, smem, s>>>(fa, (int)chunk);
  return check_launch("rr_flux_split");
}

// The device address of output rows given as device memory or page-locked
// host memory; NULL for anything else (pageable host memory).
static void* device_rows(void* flux, int* status) {
  *status = RR_OK;
  if (!flux) {
    *status = RR_ERR_ARG;
    return nullptr;
  }
  cudaPointerAttributes at{};
  const cudaError_t e = cudaPointerGetAttributes(&at, flux);
  if (e != cudaSuccess) {
    set_cuda_error(e, "rr_flux_split_transits (pointer)");
    *status = RR_ERR_CUDA;
    return nullptr;
  }
  void* dst = nullptr;
  if (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged)
    dst = flux;
  else if (at.type == cudaMemoryTypeHost)
    dst = at.devicePointer;
  if (!dst) *status = RR_ERR_ARG;   // pageable host memory: not reachable by the kernel here
  return dst;
}

int rr_flux_split_rows(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb, int ng,
                       double dg, const void* workspace, int pv0, int pv1, void* flux, int ldflux, int kind,
                       void* stream) {
  if (kind & ~(RR_ROWS_F64 | RR_ROWS_TRANSITS | RR_ROWS_TILES)) return RR_ERR_ARG;
  int st = flux_split_args(npt, npv, nlc, npb, ng, pv0, pv1, ldflux);
  if (st != RR_OK || pv1 == pv0 || npt == 0) return st;
  if (kind & RR_ROWS_TRANSITS) {
    flux = device_rows(flux, &st);
    if (!flux) return st;
  }
  return flux_split_launch(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, pv0, pv1, flux, ldflux, stream, kind);
}

int rr_flux_split_range(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb, int ng,
                        double dg, const void* workspace, int pv0, int pv1, float* flux, int ldflux,
                        void* stream) {
  return rr_flux_split_rows(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, pv0, pv1, flux, ldflux, 0, stream);
}

int rr_flux_split_range_f64(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb,
                            int ng, double dg, const void* workspace, int pv0, int pv1, double* flux, int ldflux,
                            void* stream) {
  return rr_flux_split_rows(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, pv0, pv1, flux, ldflux,
                            RR_ROWS_F64, stream);
}

int rr_flux_split_transits(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb, int ng,
                           double dg, const void* workspace, int pv0, int pv1, float* flux, int ldflux,
                           void* stream) {
  return rr_flux_split_rows(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, pv0, pv1, flux, ldflux,
                            RR_ROWS_TRANSITS, stream);
}

int rr_flux_split_transits_f64(const float* times_ff, int npt, const int32_t* lcids, int npv, int nlc, int npb,
                               int ng, double dg, const void* workspace, int pv0, int pv1, double* flux,
                               int ldflux, void* stream) {
  return rr_flux_split_rows(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, pv0, pv1, flux, ldflux,
                            RR_ROWS_TRANSITS | RR_ROWS_F64, stream);
}

int rr_full_split(const float* times_ff, double t_ref, double t_absmax, int npt, const double* k, int nkc,
                  const double* t0, int ldt0, int nep, const double* p, const double* a, const double* inc,
                  const double* e, const double* w, int npv, int nlc, int npb, const int32_t* lcids,
                  const int32_t* pbids, const int32_t* epids, const int32_t* nsamples,
                  const double* exptimes, const float* ldp, const float* istar, const float* weights,
                  int nk, int ng, int nz, double dk, double kmin, double kmax, double dg,
                  const double* z_edges, void* workspace, size_t workspace_bytes, float* flux,
                  int ldflux, void* stream) {
  int st = check_common(npt, nkc, npv, nlc, npb, nk, ng, nz, ldflux);
  if (st) return st;
  if (nep < 1 || nep > ldt0) return RR_ERR_ARG;
  if (npv == 0 || npt == 0) return RR_OK;
  if (workspace_bytes < rr_full_split_workspace_bytes(npv, npb, nlc, nep, ng)) return RR_ERR_WORKSPACE;
  st = rr_prepare_split(t_ref, t_absmax, k, nkc, t0, ldt0, nep, p, a, inc, e, w, npv, nlc, npb, pbids, epids,
                        nsamples, exptimes, ldp, istar, weights, nk, ng, nz, dk, kmin, kmax, z_edges, workspace,
                        workspace_bytes, stream, 0, nullptr, 0, nullptr, 0);
  if (st) return st;
  return rr_flux_split(times_ff, npt, lcids, npv, nlc, npb, ng, dg, workspace, flux, ldflux, stream);
}

void rr_full_split_tables(void* workspace, int npv, int npb, int nlc, int nep, int ng, const float** orb32,
                          const float** lc32, const float** ldm) {
  (void)nep;
  SplitTables t = carve_split(workspace, npv, npb, nlc, ng);
  if (orb32) *orb32 = t.orb;
  if (lc32) *lc32 = t.lc;
  if (ldm) *ldm = t.ldm;
}

void rr_serve_struct_sizes(int* request_size, int* item_size) {
  if (request_size) *request_size = (int)sizeof(rr_serve_request);
  if (item_size) *item_size = (int)sizeof(rr_serve_item);
}

int rr_serve_flux_split(const rr_serve_request* reqs, const rr_serve_item* items, const int* nitems, int* counter,
                        int nblocks, void* stream) {
  if (!reqs || !items || !nitems || !counter || nblocks < 1) return RR_ERR_ARG;
  serve_split_kernel<<<nblocks, SPLIT_WARPS * 32, 0, as_stream(stream)>>>(reqs, items, nitems, counter);
  return check_launch("rr_serve_flux_split");
}

int rr_basis_count(int law, int npar) {
  if (law < 0 || law >= LD_NLAWS) return 0;
  return basis_count(law, npar);
}

int rr_basis_tables(int law, int npar, const double* mu, int nz, const double* W64, int nk, int ng, double* B64,
                    float* B32, void* stream) {
  const int nb = rr_basis_count(law, npar);
  if (nb <= 0 || nb > MAX_BASIS || nk < 2 || ng < 2 || nz < 1 || !mu || !W64 || !B64) return RR_ERR_ARG;
  basis_tables_kernel<<<(nk * ng + 127) / 128, 128, 0, as_stream(stream)>>>(law, nb, mu, nz, W64, nk, ng, B64, B32);
  return check_launch("rr_basis_tables");
}

}  // extern "C"
