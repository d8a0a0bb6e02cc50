// Direct sums of a batched CalcV: one launch per class of systems with
// identical pair-kernel coefficients, warp groups of all of them concatenated.
#include <cuda_runtime.h>

#include "batch.cuh"
#include "bodies.cuh"
#include "internal.h"

namespace npme {

template <bool CPLX, int FUNC, int SPLIT, int ND>
__global__ void __launch_bounds__(32 * kGroupWarps, kGroupMinBlocks) batch_direct_kernel(
    PairCoef<float> k, const BatchSys *__restrict__ sys, const long long *__restrict__ off,
    int count) {
  __shared__ float4 sp[kGroupWarps][32];
  __shared__ float4 slo[kGroupWarps][32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long u = (long long)blockIdx.x * kGroupWarps + wid;
  if (u >= off[count]) return;  // warp-uniform
  const int s = find_sys(off, count, u);
  const BatchSys &S = sys[s];
  const long g = (long)(u - off[s]);
  direct_group_body<CPLX, FUNC, SPLIT, ND>(k, S.gpos, S.spos, S.qc, S.q, S.groups[g], S.gcen[g],
                                           S.segs, S.cperm, S.refine2, S.fself_r, S.fself_i, S.V,
                                           sp[wid], slo[wid], lane);
}

// Pair-once direct sums of a batch: KIND 0 the packed real body
// (direct_group_sym), 1 Helmholtz DM.
// SPLIT: a CTA of kGroupWarps warps per group, for classes with few groups
// (split_warps in direct.cu).
template <int KIND, int FUNC, int ND, bool SPLIT>
__global__ void __launch_bounds__(32 * kGroupWarps, 4) batch_sym_kernel(
    PairCoef<float> k, const BatchSys *__restrict__ sys, const long long *__restrict__ off,
    int count) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = SPLIT ? wid : 0, nsplit = SPLIT ? kGroupWarps : 1;
  const long long u = SPLIT ? (long long)blockIdx.x : (long long)blockIdx.x * kGroupWarps + wid;
  if (u >= off[count]) return;  // warp-uniform (SPLIT: no CTA is past the end)
  const int s = find_sys(off, count, u);
  const BatchSys &S = sys[s];
  const long g = (long)(u - off[s]);
  if constexpr (KIND == 0) {
    __shared__ SymWarp W[kGroupWarps];
    direct_group_sym<FUNC, ND>(k, S.gpos, S.spos, S.qc, S.q, S.hgroups[g], S.hcen[g], S.hsegs,
                               S.hzones[g], S.cperm, S.refine2, S.vsrc, W[wid], lane, part,
                               nsplit);
    if (SPLIT) __syncthreads();
    if (!SPLIT || wid == 0)
      sym_store(k, S.hgroups[g], S.cperm, S.q, S.fself_r, S.V, lane, &W[wid], nsplit);
  } else {
    __shared__ float4 ta[kGroupWarps][32], tb[kGroupWarps][32];
    double acc[4] = {0, 0, 0, 0}, acci[4] = {0, 0, 0, 0};
    const int4 G = S.hgroups[g];
    direct_group_sym_helm<ND>(k, S.gpos, S.spos, S.qc, S.q, G, S.hcen[g], S.hsegs, S.hzones[g],
                              S.cperm, S.refine2, S.vsrc, ta[wid], tb[wid], lane, part, nsplit,
                              acc, acci);
    if constexpr (SPLIT) {
      __shared__ double red[kGroupWarps][32][4];
      reduce_parts(acc, red, wid, kGroupWarps, lane);
      __syncthreads();
      reduce_parts(acci, red, wid, kGroupWarps, lane);
      if (wid > 0) return;
    }
    store_targets_cplx(G, S.cperm, S.q, S.fself_r, S.fself_i, 1.0, 1.0, S.V, lane, acc, acci);
  }
}

void launch_batch_direct(const PairCoef<float> &k, bool once, bool alpha_positive,
                         const BatchSys *sys, const long long *off, int count, long long ng,
                         cudaStream_t s) {
  const unsigned g = (unsigned)((ng + kGroupWarps - 1) / kGroupWarps);
  const int f = k.func, sp = k.split;
  // fixed-order instances: see dm_eval2 for alpha
  const int nd = sp == 1 || (f == NPME_FUNC_RALPHA && alpha_positive) ? 0 : k.nder;
  // four warps per group up to 20 groups per SM (split_warps); a class of a
  // batch runs beside other launches, so fewer groups take no more warps
  const bool split = ng <= 20 * 148;
#define NPME_BSYM(KD, FN, ND)                                                              \
  if (split)                                                                               \
    batch_sym_kernel<KD, FN, ND, true>                                                     \
        <<<(unsigned)ng, 32 * kGroupWarps, 0, s>>>(k, sys, off, count);                     \
  else                                                                                     \
    batch_sym_kernel<KD, FN, ND, false><<<g, 32 * kGroupWarps, 0, s>>>(k, sys, off, count)
#define NPME_BSYM_ND(KD, FN)                \
  switch (nd) {                             \
    case 3: NPME_BSYM(KD, FN, 3); break;    \
    case 6: NPME_BSYM(KD, FN, 6); break;    \
    case 8: NPME_BSYM(KD, FN, 8); break;    \
    default: NPME_BSYM(KD, FN, 0); break;   \
  }
  if (once) {  // the source-side sums are folded into V by the interpolation
    if (f == NPME_FUNC_HELMHOLTZ) {
      NPME_BSYM_ND(1, 2);
    } else if (sp == NPME_SPLIT_LAPLACE_ORIG) {
      NPME_BSYM(0, 2, 0);
    } else if (f == NPME_FUNC_RALPHA) {
      NPME_BSYM_ND(0, 1);
    } else {
      NPME_BSYM_ND(0, 0);
    }
    return;
  }
#undef NPME_BSYM_ND
#undef NPME_BSYM
#define NPME_BD(CX, FN, SL, ND) \
  batch_direct_kernel<CX, FN, SL, ND><<<g, 32 * kGroupWarps, 0, s>>>(k, sys, off, count)
#define NPME_BD_ND(CX, FN, SL)               \
  switch (nd) {                              \
    case 3: NPME_BD(CX, FN, SL, 3); break;   \
    case 6: NPME_BD(CX, FN, SL, 6); break;   \
    case 8: NPME_BD(CX, FN, SL, 8); break;   \
    default: NPME_BD(CX, FN, SL, 0); break;  \
  }
  if (f == NPME_FUNC_HELMHOLTZ) { NPME_BD_ND(true, 2, 0); }
  else if (sp == NPME_SPLIT_LAPLACE_ORIG) { NPME_BD(false, 0, 1, 0); }
  else if (f == NPME_FUNC_RALPHA) { NPME_BD_ND(false, 1, 0); }
  else { NPME_BD_ND(false, 0, 0); }
#undef NPME_BD_ND
#undef NPME_BD
}

}  // namespace npme
