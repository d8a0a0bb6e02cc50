// Short-range direct sum over warp groups (every pair once for the built-in
// kernels, one-sided otherwise), the pair count and the exact
// O(N^2) sum.
//
// Direct sum (src/PotentialLaplace.cpp:201-264 and the pair kernels cited in
// common.cuh): V_i = sum_{j != i, r_ij <= Rdir} q_j f_SR(r_ij),
// dV_i/dx = sum q_j f1_SR(r_ij) (x_i - x_j).  Targets are grouped by 32 in
// z-sorted coarse columns and every group owns a list of source segments
// (built on the device at set-up, setup.cu); one warp walks one group in both
// precisions.  In the pair-once walk the target-side sums stay in registers
// and each output row is written once, while the source-side sums are added
// with float (FP32) or double (FP64) atomics into a per-source buffer that a
// merge kernel folds into V: results are reproducible only up to the order
// of those atomic additions.  The one-sided walk uses no atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "bodies.cuh"
#include "internal.h"

namespace npme {

// Original Ewald split in FP32: erfcx(x) = 1 + v sum_n e_n v^n with v = x / (x +
// 2), a fit of degree 9 over 0 <= x <= 12 (error 2e-09, below FP32 rounding;
// beyond x = 10.2 exp(-x^2) is zero in FP32).  In v the value at x = 0 is exact
// and the rounding errors near it, where the pairs that matter most are, grow
// with v: 2e-08 RMS for x < 0.3.
constexpr double kErfcxFit[10] = {
    -2.2567580482e+00, 1.7432280943e+00, -2.7456315043e-01,
    -3.1246204138e-01, 1.2640637311e-02, 7.3816158880e-02,
    3.7015627549e-02, 2.7656030148e-02, -8.1190085803e-02,
    3.0625252134e-02};

double dm_taylor(const npme_params &p, double (&c)[kMaxDeriv + 1], double (&ca)[kMaxDeriv + 1]) {
  const double al = p.funcType == NPME_FUNC_RALPHA ? p.alpha : -1.0, a = 0.5 * al;
  for (int i = 0; i <= kMaxDeriv; i++) {
    if (i < 2) ca[i] = i;
    else ca[i] = i <= p.nDeriv ? ca[i - 1] * (i - 1 - a) / i : 0.0;
    c[i] = i == 0 ? 1.0 : -a * ca[i];
  }
  return std::pow(p.Rdir, al);
}

template <typename T>
PairCoef<T> make_pair_coef(const npme_handle *h) {
  PairCoef<T> k;
  memset(&k, 0, sizeof(k));
  const double R = h->p.Rdir, R2 = R * R;
  k.func = h->p.funcType;
  k.split = h->p.EwaldSplit;
  k.nder = h->p.nDeriv;
  k.R2 = (T)R2;
  k.invR2 = (T)(1.0 / R2);
  k.alpha = (T)h->p.alpha;
  k.half_alpha = (T)(0.5 * h->p.alpha);
  k.beta = (T)h->beta;
  k.beta2 = (T)(h->beta * h->beta);
  k.two_beta_rpi = (T)(2.0 * h->beta / std::sqrt(M_PI));
  k.k0r = (T)h->p.k0_r;
  k.k0i = (T)h->p.k0_i;
  double s = 1.0;  // R^(2n)
  for (int i = 0; i <= k.nder && i <= kMaxDeriv; i++) {
    k.ar[i] = (T)(h->a_r[i] * s);
    k.ai[i] = (T)(h->a_i[i] * s);
    k.br[i] = (T)(h->b_r[i] * s);
    k.bi[i] = (T)(h->b_i[i] * s);
    k.nac2[i].x = (T)(-h->a_r[i] * s), k.nac2[i].y = (T)(-h->a_i[i] * s);
    k.nbc2[i].x = (T)(-h->b_r[i] * s), k.nbc2[i].y = (T)(-h->b_i[i] * s);
    s *= R2;
  }
  // the radial-derivative polynomials have degree nder - 1: their entry nder
  // is zero, as are all entries above nder (the zero-padded evaluation of
  // the packed bodies relies on it)
  if (k.nder >= 0 && k.nder <= kMaxDeriv) {
    k.br[k.nder] = k.bi[k.nder] = (T)0;
    k.nbc2[k.nder].x = k.nbc2[k.nder].y = (T)0;
  }
  {
    const double al = h->p.funcType == NPME_FUNC_RALPHA ? h->p.alpha : -1.0;
    // the matched polynomial (zero above the order)
    const double a = 0.5 * al;
    double c[kMaxDeriv + 1], ca[kMaxDeriv + 1];
    const double Ral = dm_taylor(h->p, c, ca);
    for (int i = 0; i <= k.nder && i <= kMaxDeriv; i++) {
      k.nc2[i].x = k.nc2[i].y = (T)-c[i];
      if (i > 0) k.nq2[i - 1].x = k.nq2[i - 1].y = (T)(-i * ca[i]);
      if (i == k.nder) k.kn2.x = k.kn2.y = (T)((k.nder - a) * ca[i]);
      if (h->p.funcType != NPME_FUNC_HELMHOLTZ) {
        k.ar[i] = (T)(Ral * c[i]), k.ai[i] = (T)0;
        if (i > 0) k.br[i - 1] = (T)(-2.0 * i * c[i] * Ral / R2), k.bi[i - 1] = (T)0;
      }
    }
    if (k.split == NPME_SPLIT_LAPLACE_ORIG) {  // dm_eval2<2, 0>: coefficients and constants
      const double b = h->beta * R;
      for (int i = 0; i < 10; i++) k.nc2[i].x = k.nc2[i].y = (T)kErfcxFit[i];
      k.nq2[0].x = k.nq2[0].y = (T)b;
      k.nq2[1].x = k.nq2[1].y = (T)(-b * b / std::log(2.0));
      k.kn2.x = k.kn2.y = (T)(2.0 * b / std::sqrt(M_PI));
    }
    k.invR = 1.0 / R;
    if constexpr (sizeof(T) == 8) {
      if (h->p.funcType == NPME_FUNC_HELMHOLTZ) {
        // the unit of length is the greatest power of two <= Rdir, so that scaling by
        // it rounds nothing and the cutoff is in [1, 2)
        const double unit = std::exp2(std::ilogb(R));
        const double S2 = (R / unit) * (R / unit);
        int64_t bits;
        std::memcpy(&bits, &S2, sizeof(bits));
        k.cut_bits = (unsigned long long)bits - kMinNormal64;
        k.cut2 = S2;
        k.invR = 1.0 / unit;
        k.kapr = h->p.k0_r * unit, k.kapi = h->p.k0_i * unit;
        // the polynomial that the smooth part carries (its coefficients of r^2n,
        // rounded, magnify their rounding by their cancellation, 1e3 at |k0| Rdir = 8),
        // expanded in u = S2 - s, so that what one part adds the other takes away:
        // with the exact coefficients the sum is off by 2e-14 at |k0| Rdir = 10
        typedef long double ld;
        ld cr[kMaxDeriv + 1] = {}, ci[kMaxDeriv + 1] = {}, scale = unit;  // unit^(2n + 1)
        for (int n = 0; n <= k.nder && n <= kMaxDeriv; n++, scale *= (ld)unit * unit) {
          ld binom = scale * std::pow((ld)S2, n);  // (-1)^m n over m, S2^(n - m)
          for (int m = 0; m <= n; m++) {
            cr[m] += binom * (ld)h->a_r[n];
            ci[m] += binom * (ld)h->a_i[n];
            binom *= -(ld)(n - m) / ((m + 1) * (ld)S2);
          }
        }
        for (int m = 0; m <= k.nder && m <= kMaxDeriv; m++) {
          k.hc[m].x = (T)-cr[m], k.hc[m].y = (T)-ci[m];
          if (m > 0) k.hd[m - 1].x = (T)(2 * m * cr[m]), k.hd[m - 1].y = (T)(2 * m * ci[m]);
        }
      }
    }
    k.vscale = Ral;
    // the real walks scale FP32 coordinates by 1/Rdir, those of FP64 not
    k.gscale = (k.split == NPME_SPLIT_LAPLACE_ORIG ? 1.0 : -al) *
               std::pow(R, al - (sizeof(T) == 4 ? 1.0 : 2.0));
  }
  return k;
}
template PairCoef<float> make_pair_coef<float>(const npme_handle *);
template PairCoef<double> make_pair_coef<double>(const npme_handle *);

// ---------------------------------------------------------------------------
// FP32 bulk direct sum over warp groups.
// One warp owns one group of <= 32 targets (one per lane) and walks the
// group's source segments in chunks of 32 that run across segment
// boundaries: every lane loads one source (FP64 position), the warp stages
// the chunk in shared memory as float coordinates relative to the group
// centre and every lane then sweeps the staged chunk for its target.  The next
// chunk's loads are issued before the sweep, so global latency hides behind the
// arithmetic.  Warps are independent: only __syncwarp, no block barrier.
//
// Coordinates: each FP64 offset from the group centre is split into a float
// head and the float residual (hi + lo).  The distance test and the pair
// arithmetic use the heads; for the rare close pairs (r^2 < refine2) the
// difference is recomputed as (t_hi - s_hi) + (t_lo - s_lo), which is exact
// to ~1e-15 because the heads of two close points subtract exactly.  Without
// this, a pair at r ~ 0.01 in a group of radius ~2 carries a ~1e-5 relative
// error that dominates the gradient.

template <bool CPLX, int FUNC, int SPLIT, int ND>
__global__ void __launch_bounds__(32 * kGroupWarps, kGroupMinBlocks) direct_groups_kernel(
    PairCoef<float> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const uint32_t *__restrict__ perm, long ngroups,
    float refine2, double fself_r, double fself_i, double *__restrict__ V) {
  __shared__ float4 sp[kGroupWarps][32];   // (x_hi, y_hi, z_hi, q) / q.re
  __shared__ float4 slo[kGroupWarps][32];  // (x_lo, y_lo, z_lo, q.im)
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long g = (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform; nothing below synchronises the block
  direct_group_body<CPLX, FUNC, SPLIT, ND>(k, gpos, spos, qs, qcaller, groups[g], gcen[g], segs,
                                           perm, refine2, fself_r, fself_i, V, sp[wid], slo[wid],
                                           lane);
}


template <bool CPLX, int FUNC, int SPLIT, int ND>
static void groups_launch_nd(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  const long blocks = (h->n_groups + kGroupWarps - 1) / kGroupWarps;
  if (blocks == 0) return;
  direct_groups_kernel<CPLX, FUNC, SPLIT, ND><<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
      make_pair_coef<float>(h), h->d_gpos, h->d_spos, (const float *)a.q, a.qcaller, h->d_groups,
      h->d_gcen, h->d_segs, h->d_cperm, h->n_groups, (float)h->refine2, a.fself_r, a.fself_i,
      a.V);
}

// After a pair-once launch: the source-side sums are merged into V now, or,
// when CalcV asked for it, left for the interpolation (which visits every
// point in brick order and folds its slot in, saving a pass over V).
static void merge_or_defer(npme_handle *h, const DirectArgs &a, cudaStream_t s, double vs,
                           double gs) {
  if (a.defer_merge) {
    h->merge_pending = true;
    h->merge_vs = vs, h->merge_gs = gs;
  } else {
    launch_merge_source(h, a.V, s, vs, gs);
    h->launches++;
  }
}

// Warps per group of a pair-once launch with ngroups groups.  The SMs hold
// 16 warps each (128 registers a thread), 2,368 in all, and a group is one
// serial walk of its half-shell list, so with few groups the launch lasts as
// long as one walk with most of the chip idle, and with about one round of
// them as long as the heaviest: the walk is split over the warps of a CTA.
// Measured, whole against split walks: 141 groups (4,000 points) 92 / 26 us
// with 16 warps, 28 with 8; 1,062 groups (30,000 points in a flat box) 110 /
// 82 us with 4 warps, 96 with 2, 98 with 8; 2,000 groups (FP64 Helmholtz,
// 62,500 points) 1,530 / 1,098 us with 4.  From about two rounds on the
// splitting's own work (every warp stages the targets and walks all segments)
// costs more than it gives: 3,300 groups 137 / 139 us, 31,700 groups +10 %.
constexpr int kMaxSplit = 16;
static int split_warps(long ngroups) {
  if (ngroups <= 148) return 16;
  if (ngroups <= 4 * 148) return 8;
  if (ngroups <= 20 * 148) return 4;
  return 1;
}

// FP32 real-DM direct sum with every pair evaluated once (direct_group_sym),
// then the source-side sums folded into V.
template <int FUNC, int ND>
__global__ void __launch_bounds__(32 * kGroupWarps, 4) direct_sym_kernel(
    PairCoef<float> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const int2 *__restrict__ zones,
    const uint32_t *__restrict__ perm, long ngroups, float refine2, double fself_r,
    double *__restrict__ V, float4 *__restrict__ vsrc) {
  __shared__ SymWarp W[kGroupWarps];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long g = (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform; nothing below synchronises the block
  direct_group_sym<FUNC, ND>(k, gpos, spos, qs, qcaller, groups[g], gcen[g], segs, zones[g], perm,
                             refine2, vsrc, W[wid], lane, 0, 1);
  sym_store(k, groups[g], perm, qcaller, fself_r, V, lane, &W[wid], 1);
}

// The same with a CTA of blockDim.x / 32 warps per group (split_warps).
template <int FUNC, int ND>
__global__ void __launch_bounds__(32 * kMaxSplit) direct_sym_split_kernel(
    PairCoef<float> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const int2 *__restrict__ zones,
    const uint32_t *__restrict__ perm, float refine2, double fself_r, double *__restrict__ V,
    float4 *__restrict__ vsrc) {
  __shared__ SymWarp W[kMaxSplit];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nsplit = blockDim.x >> 5;
  const long g = blockIdx.x;
  const int4 G = groups[g];
  direct_group_sym<FUNC, ND>(k, gpos, spos, qs, qcaller, G, gcen[g], segs, zones[g], perm, refine2,
                             vsrc, W[wid], lane, wid, nsplit);
  __syncthreads();
  if (wid == 0) sym_store(k, G, perm, qcaller, fself_r, V, lane, W, nsplit);
}

// V[caller(i)] += scale * vsrc[i] for every brick-order slot i, then
// vsrc[i] = 0 for the next call.
__global__ void merge_source_kernel(float4 *__restrict__ vsrc, const uint32_t *__restrict__ bperm,
                                    long n, double vs, double gs, double *__restrict__ V) {
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const float4 a = vsrc[s];
  vsrc[s] = make_float4(0.f, 0.f, 0.f, 0.f);
  double4 *o = reinterpret_cast<double4 *>(V) + bperm[s];
  double4 v = *o;
  v.x += vs * (double)a.x;
  v.y += gs * (double)a.y;
  v.z += gs * (double)a.z;
  v.w += gs * (double)a.w;
  *o = v;
}

// FP32 Helmholtz DM form (direct_group_sym_helm): CTAs of kGroupWarps groups, or
// (SPLIT) of one group.
template <int ND, bool SPLIT>
__global__ void __launch_bounds__(32 * (SPLIT ? kMaxSplit : kGroupWarps), SPLIT ? 1 : 4)
    direct_sym_helm_kernel(
    PairCoef<float> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const int2 *__restrict__ zones,
    const uint32_t *__restrict__ perm, long ngroups, float refine2, double fself_r,
    double fself_i, double *__restrict__ V, float4 *__restrict__ vsrc) {
  constexpr int W = SPLIT ? kMaxSplit : kGroupWarps;
  __shared__ float4 th[W][32];  // group targets: heads, Re q
  __shared__ float4 tl[W][32];  // residuals, Im q
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsplit = SPLIT ? blockDim.x >> 5 : 1, part = SPLIT ? wid : 0;
  const long g = SPLIT ? (long)blockIdx.x : (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform (SPLIT: no CTA is past the end)
  double acc[4] = {0, 0, 0, 0}, acci[4] = {0, 0, 0, 0};
  const int4 G = groups[g];
  direct_group_sym_helm<ND>(k, gpos, spos, qs, qcaller, G, gcen[g], segs, zones[g], perm, refine2,
                            vsrc, th[wid], tl[wid], lane, part, nsplit, acc, acci);
  if constexpr (SPLIT) {
    __shared__ double red[kMaxSplit][32][4];
    reduce_parts(acc, red, wid, nsplit, lane);
    __syncthreads();
    reduce_parts(acci, red, wid, nsplit, lane);
    if (wid > 0) return;
  }
  store_targets_cplx(G, perm, qcaller, fself_r, fself_i, 1.0, 1.0, V, lane, acc, acci);
}

// Complex V[caller(i)][0..3] += vsrc[2i], vsrc[2i + 1] (re, im pairs), then zero.
__global__ void merge_source_cplx_kernel(float4 *__restrict__ vsrc,
                                         const uint32_t *__restrict__ bperm, long n,
                                         double *__restrict__ V) {
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const float4 a = vsrc[2 * s], b = vsrc[2 * s + 1];
  vsrc[2 * s] = vsrc[2 * s + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  double4 *o = reinterpret_cast<double4 *>(V) + 2 * (long)bperm[s];
  double4 u = o[0], w = o[1];
  u.x += a.x, u.y += a.y, u.z += a.z, u.w += a.w;
  w.x += b.x, w.y += b.y, w.z += b.z, w.w += b.w;
  o[0] = u, o[1] = w;
}

template <int ND>
static void sym_helm_launch_nd(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  const long blocks = (h->n_hgroups + kGroupWarps - 1) / kGroupWarps;
  if (blocks == 0) return;
  const PairCoef<float> k = make_pair_coef<float>(h);
  const int split = split_warps(h->n_hgroups);
  if (split > 1)
    direct_sym_helm_kernel<ND, true><<<(unsigned)h->n_hgroups, 32 * split, 0, s>>>(
        k, h->d_gpos, h->d_spos, (const float *)a.q, a.qcaller, h->d_hgroups, h->d_hcen,
        h->d_hsegs, h->d_hzones, h->d_cperm, h->n_hgroups, (float)h->refine2, a.fself_r,
        a.fself_i, a.V, h->d_vsrc);
  else
    direct_sym_helm_kernel<ND, false><<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
        k, h->d_gpos, h->d_spos, (const float *)a.q, a.qcaller, h->d_hgroups, h->d_hcen,
        h->d_hsegs, h->d_hzones, h->d_cperm, h->n_hgroups, (float)h->refine2, a.fself_r,
        a.fself_i, a.V, h->d_vsrc);
  merge_or_defer(h, a, s, 1.0, 1.0);
}

template <int FUNC, int ND>
static void sym_launch_nd(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  if (h->n_hgroups == 0) return;
  const PairCoef<float> k = make_pair_coef<float>(h);
  const int split = split_warps(h->n_hgroups);
  if (split > 1) {
    direct_sym_split_kernel<FUNC, ND><<<(unsigned)h->n_hgroups, 32 * split, 0, s>>>(
        k, h->d_gpos, h->d_spos, (const float *)a.q, a.qcaller, h->d_hgroups, h->d_hcen,
        h->d_hsegs, h->d_hzones, h->d_cperm, (float)h->refine2, a.fself_r, a.V, h->d_vsrc);
  } else {
    const long blocks = (h->n_hgroups + kGroupWarps - 1) / kGroupWarps;
    direct_sym_kernel<FUNC, ND><<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
        k, h->d_gpos, h->d_spos, (const float *)a.q, a.qcaller, h->d_hgroups, h->d_hcen,
        h->d_hsegs, h->d_hzones, h->d_cperm, h->n_hgroups, (float)h->refine2, a.fself_r, a.V,
        h->d_vsrc);
  }
  merge_or_defer(h, a, s, k.vscale, k.gscale);
}

// FP64 form for the real built-in kernels (DM and original Ewald).
template <int FUNC, int SPLIT, int ND>
__global__ void __launch_bounds__(32 * kGroupWarps) direct_sym64_kernel(
    PairCoef<double> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const double *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const int2 *__restrict__ zones,
    const uint32_t *__restrict__ perm, long ngroups,
    double fself_r, double *__restrict__ V, double *__restrict__ vsrc) {
  __shared__ double4 tsm[kGroupWarps][32];  // group targets (x, y, z, q)
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long g = (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform
  if constexpr (SPLIT == 0) {
    double acc[4] = {0, 0, 0, 0};
    const int4 G = groups[g];
    direct_group_sym64_dm<FUNC, ND>(k, gpos, spos, qs, qcaller, G, gcen[g], segs, zones[g], perm,
                                    vsrc,
                                    tsm[wid], lane, 0, 1, acc);
    store_targets64(G, perm, qcaller, fself_r, k.vscale, k.gscale, V, lane, acc);
  } else
    direct_group_sym64<FUNC, SPLIT, ND>(k, gpos, spos, qs, qcaller, groups[g], gcen[g], segs,
                                        perm, fself_r, V, vsrc, tsm[wid], lane);
}

// The DM form with a CTA of blockDim.x / 32 warps per group (split_warps).
template <int FUNC, int ND>
__global__ void __launch_bounds__(32 * kMaxSplit) direct_sym64_split_kernel(
    PairCoef<double> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const double *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const int2 *__restrict__ zones,
    const uint32_t *__restrict__ perm, double fself_r,
    double *__restrict__ V, double *__restrict__ vsrc) {
  __shared__ double4 tsm[kMaxSplit][32];
  __shared__ double red[kMaxSplit][32][4];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nsplit = blockDim.x >> 5;
  const long g = blockIdx.x;
  double acc[4] = {0, 0, 0, 0};
  const int4 G = groups[g];
  direct_group_sym64_dm<FUNC, ND>(k, gpos, spos, qs, qcaller, G, gcen[g], segs, zones[g], perm,
                                  vsrc,
                                  tsm[wid], lane, wid, nsplit, acc);
  reduce_parts(acc, red, wid, nsplit, lane);
  if (wid == 0) store_targets64(G, perm, qcaller, fself_r, k.vscale, k.gscale, V, lane, acc);
}

// V[caller(i)][m] += vsrc[i][m], then vsrc[i] = 0 for the next call.
__global__ void merge_source64_kernel(double4 *__restrict__ vsrc,
                                      const uint32_t *__restrict__ bperm, long n,
                                      double *__restrict__ V) {
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const double4 a = vsrc[s];
  vsrc[s] = make_double4(0, 0, 0, 0);
  double4 *o = reinterpret_cast<double4 *>(V) + bperm[s];
  double4 v = *o;
  v.x += a.x, v.y += a.y, v.z += a.z, v.w += a.w;
  *o = v;
}

template <int FUNC, int SPLIT, int ND>
static void sym64_launch_nd(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  const long blocks = (h->n_hgroups + kGroupWarps - 1) / kGroupWarps;
  if (blocks == 0) return;
  if constexpr (SPLIT == 0) {
    const int split = split_warps(h->n_hgroups);
    if (split > 1) {
      direct_sym64_split_kernel<FUNC, ND><<<(unsigned)h->n_hgroups, 32 * split, 0, s>>>(
          make_pair_coef<double>(h), h->d_gpos, h->d_spos, (const double *)a.q, a.qcaller,
          h->d_hgroups, h->d_hcen, h->d_hsegs, h->d_hzones, h->d_cperm, a.fself_r, a.V,
          h->d_vsrc64);
      merge_or_defer(h, a, s, 1.0, 1.0);
      return;
    }
  }
  direct_sym64_kernel<FUNC, SPLIT, ND><<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
      make_pair_coef<double>(h), h->d_gpos, h->d_spos, (const double *)a.q, a.qcaller,
      h->d_hgroups, h->d_hcen, h->d_hsegs, h->d_hzones, h->d_cperm, h->n_hgroups, a.fself_r, a.V,
      h->d_vsrc64);
  merge_or_defer(h, a, s, 1.0, 1.0);
}

// FP64 Helmholtz form: CTAs of kGroupWarps groups (split = 1) or of one group.
template <int ND, bool SPLIT>
__global__ void __launch_bounds__(32 * (SPLIT ? kMaxSplit : kGroupWarps), SPLIT ? 1 : 4)
    direct_sym64_helm_kernel(
    PairCoef<double> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const double *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const int2 *__restrict__ zones,
    const uint32_t *__restrict__ perm, long ngroups,
    double fself_r, double fself_i, double *__restrict__ V, double *__restrict__ vsrc) {
  constexpr int W = SPLIT ? kMaxSplit : kGroupWarps;
  __shared__ double tsm[W][5][32];  // group targets: x, y, z, q
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsplit = SPLIT ? blockDim.x >> 5 : 1, part = SPLIT ? wid : 0;
  const long g = SPLIT ? (long)blockIdx.x : (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform (SPLIT: no CTA is past the end)
  double acc[4] = {0, 0, 0, 0}, acci[4] = {0, 0, 0, 0};
  const int4 G = groups[g];
  direct_group_sym64_helm<ND>(k, gpos, spos, qs, qcaller, G, gcen[g], segs, zones[g], perm, vsrc,
                              tsm[wid],
                              lane, part, nsplit, acc, acci);
  if constexpr (SPLIT) {
    __shared__ double red[kMaxSplit][32][4];
    reduce_parts(acc, red, wid, nsplit, lane);
    __syncthreads();
    reduce_parts(acci, red, wid, nsplit, lane);
    if (wid > 0) return;
  }
  store_targets_cplx(G, perm, qcaller, fself_r, fself_i, k.invR, k.invR * k.invR, V, lane, acc,
                     acci);
}

// Complex V[caller(i)][0..3] += vsrc[i] (re, im pairs), then zero.
__global__ void merge_source64_cplx_kernel(double4 *__restrict__ vsrc,
                                           const uint32_t *__restrict__ bperm, long n,
                                           double *__restrict__ V) {
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const double4 a = vsrc[2 * s], b = vsrc[2 * s + 1];
  vsrc[2 * s] = vsrc[2 * s + 1] = make_double4(0, 0, 0, 0);
  double4 *o = reinterpret_cast<double4 *>(V) + 2 * (long)bperm[s];
  double4 u = o[0], w = o[1];
  u.x += a.x, u.y += a.y, u.z += a.z, u.w += a.w;
  w.x += b.x, w.y += b.y, w.z += b.z, w.w += b.w;
  o[0] = u, o[1] = w;
}

template <int ND>
static void sym64_helm_launch_nd(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  const long blocks = (h->n_hgroups + kGroupWarps - 1) / kGroupWarps;
  if (blocks == 0) return;
  const PairCoef<double> k = make_pair_coef<double>(h);
  const int split = split_warps(h->n_hgroups);
  if (split > 1)
    direct_sym64_helm_kernel<ND, true><<<(unsigned)h->n_hgroups, 32 * split, 0, s>>>(
        k, h->d_gpos, h->d_spos, (const double *)a.q, a.qcaller, h->d_hgroups, h->d_hcen,
        h->d_hsegs, h->d_hzones, h->d_cperm, h->n_hgroups, a.fself_r, a.fself_i, a.V, h->d_vsrc64);
  else
    direct_sym64_helm_kernel<ND, false><<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
        k, h->d_gpos, h->d_spos, (const double *)a.q, a.qcaller, h->d_hgroups, h->d_hcen,
        h->d_hsegs, h->d_hzones, h->d_cperm, h->n_hgroups, a.fself_r, a.fself_i, a.V, h->d_vsrc64);
  merge_or_defer(h, a, s, 1.0, 1.0);
}

template <int FUNC, int SPLIT>
static void sym64_launch(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  switch (SPLIT == 1 || (FUNC == 1 && h->p.alpha >= 0) ? 0 : h->p.nDeriv) {
    case 3: sym64_launch_nd<FUNC, SPLIT, 3>(h, a, s); break;
    case 6: sym64_launch_nd<FUNC, SPLIT, 6>(h, a, s); break;
    case 8: sym64_launch_nd<FUNC, SPLIT, 8>(h, a, s); break;
    default: sym64_launch_nd<FUNC, SPLIT, 0>(h, a, s); break;
  }
}

void launch_merge_source(npme_handle *h, double *V, cudaStream_t s, double vs, double gs) {
  const long n = (long)h->n;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (!h->fp32 && h->complex_kernel)
    merge_source64_cplx_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<double4 *>(h->d_vsrc64),
                                                      h->d_bperm, n, V);
  else if (!h->fp32)
    merge_source64_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<double4 *>(h->d_vsrc64),
                                                 h->d_bperm, n, V);
  else if (h->complex_kernel)
    merge_source_cplx_kernel<<<blocks, 256, 0, s>>>(h->d_vsrc, h->d_bperm, n, V);
  else
    merge_source_kernel<<<blocks, 256, 0, s>>>(h->d_vsrc, h->d_bperm, n, vs, gs, V);
}

void clear_source_sums(npme_handle *h, cudaStream_t s) {
  const size_t b =
      (h->fp32 ? sizeof(float) : sizeof(double)) * 4 * (h->complex_kernel ? 2 : 1) * h->n;
  cudaMemsetAsync(h->fp32 ? (void *)h->d_vsrc : (void *)h->d_vsrc64, 0, b, s);
}

// The pair-once form applies to all built-in kernels (derivative orders 3, 6 and 8
// compiled with the order fixed, the others by one instance at degree kMaxDeriv
// with zero-padded coefficients) and to real caller-defined ones.  FP64 Helmholtz
// with |k0| Rdir >= kMaxHelmArg, complex caller-defined kernels and handles set up
// under NPME_PAIRS_ONCE=0 walk the full segments.
bool needs_full_lists(const npme_handle *h) {
  if (!h->use_sym) return true;
  if (h->user_kernel) return h->complex_kernel;  // real: the functor's scalar pair kernel
  // FP64 Helmholtz: its argument reduction holds for moderate arguments
  return h->p.funcType == NPME_FUNC_HELMHOLTZ && !h->fp32 &&
         !(std::fabs(h->p.k0_r) * h->p.Rdir < kMaxHelmArg);
}

bool pairs_once(const npme_handle *h) { return h->n_hgroups > 0 && !needs_full_lists(h); }

static bool sym_launch(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  if (!pairs_once(h)) return false;
  const int f = h->p.funcType, nd = h->p.nDeriv;
  if (f == NPME_FUNC_HELMHOLTZ && !h->fp32) {
    if (nd == 3) sym64_helm_launch_nd<3>(h, a, s);
    else if (nd == 6) sym64_helm_launch_nd<6>(h, a, s);
    else if (nd == 8) sym64_helm_launch_nd<8>(h, a, s);
    else sym64_helm_launch_nd<0>(h, a, s);
    return true;
  }
  if (f == NPME_FUNC_HELMHOLTZ) {
    if (nd == 3) sym_helm_launch_nd<3>(h, a, s);
    else if (nd == 6) sym_helm_launch_nd<6>(h, a, s);
    else if (nd == 8) sym_helm_launch_nd<8>(h, a, s);
    else sym_helm_launch_nd<0>(h, a, s);
    return true;
  }
  if (h->fp32 && h->p.EwaldSplit == NPME_SPLIT_LAPLACE_ORIG) {
    sym_launch_nd<2, 0>(h, a, s);
    return true;
  }
  if (!h->fp32) {
    if (h->p.EwaldSplit == NPME_SPLIT_LAPLACE_ORIG) sym64_launch<0, 1>(h, a, s);
    else if (f == NPME_FUNC_RALPHA) sym64_launch<1, 0>(h, a, s);
    else sym64_launch<0, 0>(h, a, s);
    return true;
  }
  if (f == NPME_FUNC_LAPLACE) {
    if (nd == 3) sym_launch_nd<0, 3>(h, a, s);
    else if (nd == 6) sym_launch_nd<0, 6>(h, a, s);
    else if (nd == 8) sym_launch_nd<0, 8>(h, a, s);
    else sym_launch_nd<0, 0>(h, a, s);
  } else {
    // the fixed-order instances hold for alpha < 0 (dm_eval2)
    if (h->p.alpha >= 0) sym_launch_nd<1, 0>(h, a, s);
    else if (nd == 3) sym_launch_nd<1, 3>(h, a, s);
    else if (nd == 6) sym_launch_nd<1, 6>(h, a, s);
    else if (nd == 8) sym_launch_nd<1, 8>(h, a, s);
    else sym_launch_nd<1, 0>(h, a, s);
  }
  return true;
}

template <bool CPLX, int FUNC, int SPLIT, int ND>
__global__ void __launch_bounds__(32 * kGroupWarps) direct_groups64_kernel(
    PairCoef<double> k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const double *__restrict__ qs, const double *__restrict__ qcaller,
    const int4 *__restrict__ groups, const double4 *__restrict__ gcen,
    const int2 *__restrict__ segs, const uint32_t *__restrict__ perm, long ngroups,
    double fself_r, double fself_i, double *__restrict__ V) {
  __shared__ double4 sp[kGroupWarps][32];
  __shared__ double sqi[kGroupWarps][32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long g = (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform
  direct_group_fp64<CPLX, FUNC, SPLIT, ND>(k, gpos, spos, qs, qcaller, groups[g], gcen[g], segs,
                                           perm, fself_r, fself_i, V, sp[wid], sqi[wid], lane);
}

template <bool CPLX, int FUNC, int SPLIT, int ND>
static void groups64_launch_nd(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  const long blocks = (h->n_groups + kGroupWarps - 1) / kGroupWarps;
  if (blocks == 0) return;
  direct_groups64_kernel<CPLX, FUNC, SPLIT, ND><<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
      make_pair_coef<double>(h), h->d_gpos, h->d_spos, (const double *)a.q, a.qcaller,
      h->d_groups, h->d_gcen, h->d_segs, h->d_cperm, h->n_groups, a.fself_r, a.fself_i, a.V);
}

template <bool CPLX, int FUNC, int SPLIT>
static void groups_launch(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  if (!h->fp32) {
    switch (SPLIT == 1 ? 0 : h->p.nDeriv) {
      case 3: groups64_launch_nd<CPLX, FUNC, SPLIT, 3>(h, a, s); break;
      case 6: groups64_launch_nd<CPLX, FUNC, SPLIT, 6>(h, a, s); break;
      case 8: groups64_launch_nd<CPLX, FUNC, SPLIT, 8>(h, a, s); break;
      default: groups64_launch_nd<CPLX, FUNC, SPLIT, 0>(h, a, s); break;
    }
    return;
  }
  switch (SPLIT == 1 || (FUNC == 1 && h->p.alpha >= 0) ? 0 : h->p.nDeriv) {
    case 3: groups_launch_nd<CPLX, FUNC, SPLIT, 3>(h, a, s); break;
    case 6: groups_launch_nd<CPLX, FUNC, SPLIT, 6>(h, a, s); break;
    case 8: groups_launch_nd<CPLX, FUNC, SPLIT, 8>(h, a, s); break;
    default: groups_launch_nd<CPLX, FUNC, SPLIT, 0>(h, a, s); break;
  }
}

int launch_direct_args(npme_handle *h, const DirectArgs &a, cudaStream_t s) {
  int rc = NPME_OK;
  if (h->user_kernel) {
    rc = h->uops.direct(h, &a, s);
  } else if (!sym_launch(h, a, s)) {  // both precisions walk warp groups
    const int f = h->p.funcType, sp = h->p.EwaldSplit;
    if (f == NPME_FUNC_HELMHOLTZ) groups_launch<true, 2, 0>(h, a, s);
    else if (sp == NPME_SPLIT_LAPLACE_ORIG) groups_launch<false, 0, 1>(h, a, s);
    else if (f == NPME_FUNC_RALPHA) groups_launch<false, 1, 0>(h, a, s);
    else groups_launch<false, 0, 0>(h, a, s);
  }
  h->launches++;
  return rc;
}

int launch_direct(npme_handle *h, const double *d_q, double *d_V, cudaStream_t s) {
  DirectArgs a{h->d_qc, d_q, h->fself_r, h->fself_i, d_V};
  a.defer_merge = true;  // CalcV: the interpolation folds the source-side sums in
  return launch_direct_args(h, a, s);
}

// Unordered pairs with 0 < r <= Rdir (FP64 distances) over the pair-once
// lists: every target of a group against the later ones of its group and every
// source of its half-shell segments: the work count of the roofline report
// (not on the CalcV path).
__global__ void __launch_bounds__(32 * kGroupWarps) count_pairs_kernel(
    const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const int4 *__restrict__ groups, const int2 *__restrict__ segs, long ngroups, double R2,
    unsigned long long *__restrict__ count) {
  __shared__ double4 sp[kGroupWarps][32];
  const unsigned FULL = 0xffffffffu;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long g = (long)blockIdx.x * kGroupWarps + wid;
  if (g >= ngroups) return;  // warp-uniform
  const int4 G = groups[g];
  const double4 t = lane < G.y ? gpos[G.x + lane] : make_double4(1e150, 1e150, 1e150, 0.0);
  unsigned long long mine = 0;
  auto count_chunk = [&](int from, int cnt) {
    for (int s = from; s < cnt; s++) {
      const double4 q = sp[wid][s];
      const double x = t.x - q.x, y = t.y - q.y, z = t.z - q.z;
      const double r2 = x * x + y * y + z * z;
      mine += (r2 <= R2 && r2 > 0.0) ? 1ull : 0ull;
    }
  };
  sp[wid][lane] = t;
  __syncwarp();
  if (lane < G.y) count_chunk(lane + 1, G.y);
  SrcCursor cur{G.z, lane};
  cur.normalize(segs, G.w);
  while (__any_sync(FULL, cur.seg < G.w)) {
    const bool v = cur.seg < G.w;
    const int cnt = __popc(__ballot_sync(FULL, v));  // valid lanes form a prefix
    __syncwarp();
    if (v) sp[wid][lane] = spos[(long)segs[cur.seg].x + cur.off];
    __syncwarp();
    count_chunk(0, cnt);
    cur.off += 32;
    cur.normalize(segs, G.w);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(FULL, mine, o);
  if (lane == 0) atomicAdd(count, mine);
}

void launch_count_pairs(npme_handle *h, unsigned long long *d_count, cudaStream_t s) {
  const long blocks = (h->n_hgroups + kGroupWarps - 1) / kGroupWarps;
  if (blocks == 0) return;
  count_pairs_kernel<<<(unsigned)blocks, 32 * kGroupWarps, 0, s>>>(
      h->d_gpos, h->d_spos, h->d_hgroups, h->d_hsegs, h->n_hgroups, h->p.Rdir * h->p.Rdir,
      d_count);
}

// ---------------------------------------------------------------------------
// Exact sum (src/PotentialLaplace.cpp:40-132, src/PotentialHelmholtz.cpp:41,
// src/PotentialGenFunc.cpp:321): all pairs j != i with the full kernel, FP64,
// no self term.  A CTA of 128 targets walks its share of the sources (blockIdx.y
// of gridDim.y) in shared-memory tiles; with more than one share the partial
// sums go to scratch and exact_reduce_kernel adds them in order.  Bound by the
// FP64 pipe: 18 operations per ordered pair for 1/r.

constexpr int kExactBS = 128;

struct ExactArgs {
  const double *coord, *q;
  long n;
  double alpha, k0r, k0i;
  const uint32_t *tidx;
  long nt, share;  // targets, sources per share
  double *out;     // V, or the partial sums [share][target][4 or 8]
};

// 1/sqrt(r2) of any r2 >= 0: the iteration where it holds, the hardware's 0
// or infinity elsewhere (coincident points give infinity, as rsqrt does).
__device__ __forceinline__ double rsqrt_any(double r2) {
  const double y = rsqrt_iter(r2);
  const bool normal = (unsigned)__double2hiint(r2) - 0x00100000u < 0x7fe00000u;
  return normal ? y : rsqrt(r2);
}

// One ordered pair added to the target's sums.  FUNC as in npme_params; 3:
// Helmholtz with arguments beyond kMaxHelmArg.
template <int FUNC>
__device__ __forceinline__ void exact_pair(const ExactArgs &A, double x, double y, double z,
                                           double r2, double qr, double qi, double (&a)[4],
                                           double (&ai)[4]) {
  const double ri = rsqrt_any(r2), ri2 = ri * ri;
  if constexpr (FUNC < 2) {
    const double f = FUNC == 0 ? qr * ri : qr * pow(r2, 0.5 * A.alpha);
    const double g = (FUNC == 0 ? -f : A.alpha * f) * ri2;
    a[0] += f;
    a[1] = fma(g, x, a[1]);
    a[2] = fma(g, y, a[2]);
    a[3] = fma(g, z, a[3]);
  } else {
    const double r = r2 * ri;
    double sn, cs;
    if (FUNC == 2) sincos_taylor(A.k0r * r, sn, cs);
    else sincos(A.k0r * r, &sn, &cs);
    const double d = A.k0i != 0.0 ? exp(-A.k0i * r) * ri : ri;
    const double er = cs * d, ei = sn * d;
    // f1 = f0 (i k0 / r - 1 / r^2)
    const double u = fma(-A.k0i, ri, -ri2), v = A.k0r * ri;
    const double f1r = fma(u, er, -v * ei), f1i = fma(u, ei, v * er);
    a[0] = fma(er, qr, fma(-ei, qi, a[0]));
    ai[0] = fma(er, qi, fma(ei, qr, ai[0]));
    const double gr = fma(f1r, qr, -f1i * qi), gi = fma(f1r, qi, f1i * qr);
    a[1] = fma(gr, x, a[1]), a[2] = fma(gr, y, a[2]), a[3] = fma(gr, z, a[3]);
    ai[1] = fma(gi, x, ai[1]), ai[2] = fma(gi, y, ai[2]), ai[3] = fma(gi, z, ai[3]);
  }
}

template <int FUNC>
__global__ void __launch_bounds__(kExactBS) exact_kernel(const __grid_constant__ ExactArgs A) {
  constexpr bool CPLX = FUNC >= 2;
  __shared__ double4 sp[kExactBS];  // x, y, z, Re q
  __shared__ double sqi[CPLX ? kExactBS : 1];
  // output row t holds target tidx[t] (every point when tidx is null)
  const long t = blockIdx.x * (long)kExactBS + threadIdx.x;
  const bool active = t < A.nt;
  const long i = active ? (A.tidx ? (long)A.tidx[t] : t) : -1;
  double xi = 0, yi = 0, zi = 0;
  if (active) xi = A.coord[3 * i], yi = A.coord[3 * i + 1], zi = A.coord[3 * i + 2];
  double a[4] = {0, 0, 0, 0}, ai[4] = {0, 0, 0, 0};
  const long first = blockIdx.y * A.share, last = min(A.n, first + A.share);
  for (long j0 = first; j0 < last; j0 += kExactBS) {
    __syncthreads();
    const long j = j0 + threadIdx.x;
    if (j < last) {
      sp[threadIdx.x] = make_double4(A.coord[3 * j], A.coord[3 * j + 1], A.coord[3 * j + 2],
                                     CPLX ? A.q[2 * j] : A.q[j]);
      if (CPLX) sqi[threadIdx.x] = A.q[2 * j + 1];
    }
    __syncthreads();
    const int cnt = (int)min((long)kExactBS, last - j0);
    auto sweep = [&](bool own) {  // own: the target itself may be in the tile
#pragma unroll 4
      for (int s = 0; s < cnt; s++) {
        if (own && j0 + s == i) continue;
        const double4 S = sp[s];
        const double x = xi - S.x, y = yi - S.y, z = zi - S.z;
        exact_pair<FUNC>(A, x, y, z, fma(x, x, fma(y, y, z * z)), S.w, CPLX ? sqi[s] : 0.0, a, ai);
      }
    };
    if (__any_sync(0xffffffffu, i >= j0 && i < j0 + cnt)) sweep(true);
    else sweep(false);
  }
  if (active) {
    const long row = (long)blockIdx.y * A.nt + t;
    if (CPLX) {
      double2 *Vo = reinterpret_cast<double2 *>(A.out) + 4 * row;
      for (int m = 0; m < 4; m++) Vo[m] = make_double2(a[m], ai[m]);
    } else {
      reinterpret_cast<double4 *>(A.out)[row] = make_double4(a[0], a[1], a[2], a[3]);
    }
  }
}

// V[i] = sum of the shares' partial sums, in order.
__global__ void exact_reduce_kernel(const double *__restrict__ part, long m, int shares,
                                    double *__restrict__ V) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= m) return;
  double v = part[i];
  for (int s = 1; s < shares; s++) v += part[(long)s * m + i];
  V[i] = v;
}

int launch_exact(npme_handle *h, const double *d_q, double *d_V, cudaStream_t s,
                 const uint32_t *d_tidx, long nt) {
  const long n = (long)h->n;
  if (!d_tidx) nt = n;
  const int blocks = (int)((nt + kExactBS - 1) / kExactBS);
  if (blocks == 0) return NPME_OK;
  if (h->user_kernel) {
    h->launches++;
    return h->uops.exact(h, d_q, d_V, s, d_tidx, nt);
  }
  // Shares of the sources: about 16 CTAs per SM (two rounds of the 8 that are
  // resident), so that a few thousand targets fill the chip and the last round
  // of a larger set is short; at least 1,024 sources each.  Without memory
  // for the partial sums: one share.
  const int C = h->complex_kernel ? 2 : 1;
  long shares = std::min<long>((148L * 16 + blocks - 1) / blocks, (n + 1023) / 1024);
  shares = std::max<long>(1, shares);
  if (shares > 1 && handle_buffer(h, (void **)&h->d_part, sizeof(double) * 4 * C * nt * shares))
    shares = 1;
  ExactArgs A{h->d_coord, d_q, n, h->p.alpha, h->p.k0_r, h->p.k0_i, d_tidx, nt, 0, d_V};
  A.share = ((n + shares - 1) / shares + kExactBS - 1) / kExactBS * kExactBS;
  shares = (n + A.share - 1) / A.share;
  if (shares > 1) A.out = h->d_part;
  const int f = h->p.funcType;
  double diag2 = 0;
  for (int d = 0; d < 3; d++) diag2 += std::pow(h->bmax[d] - h->bmin[d], 2);
  const bool near = std::fabs(h->p.k0_r) * std::sqrt(diag2) < kMaxHelmArg;
  const dim3 grid((unsigned)blocks, (unsigned)shares);
  if (f == 0) exact_kernel<0><<<grid, kExactBS, 0, s>>>(A);
  else if (f == 1) exact_kernel<1><<<grid, kExactBS, 0, s>>>(A);
  else if (near) exact_kernel<2><<<grid, kExactBS, 0, s>>>(A);
  else exact_kernel<3><<<grid, kExactBS, 0, s>>>(A);
  h->launches++;
  if (shares > 1) {
    const long m = nt * 4 * C;
    exact_reduce_kernel<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(h->d_part, m, (int)shares,
                                                                    d_V);
    h->launches++;
  }
  return NPME_OK;
}

}  // namespace npme
