// Per-system descriptors of a batched CalcV (batch.cu) and its direct sums
// (batch_direct.cu).
#pragma once

#include "internal.h"

namespace npme {

struct BatchSys {
  const double *q;  // caller charges (device)
  double *V;        // caller output (device)
  const BrickPoint<float> *bpts;
  const uint32_t *cperm;  // targets: group order -> caller index
  const uint32_t *dperm;  // direct-sum sources: source order -> caller index
  float *qc;
  const int *brick_list, *odd_list, *brick_start;
  int nb2, nb3;
  int apart;  // odd bricks go by themselves
  float *grid;    // real N1 N2 N3 (real kernels) or complex (Helmholtz)
  float2 *kgrid;  // R2C half spectrum (real kernels)
  const float *G;
  long N1, N2, N3;  // FFT box
  long g1, g2, g3;  // dimensions the grid is stored with
  float c1, c2, c3;
  const double4 *gpos, *spos;
  const int4 *groups;
  const double4 *gcen;
  const int2 *segs;
  // pair-once walk: half-shell groups and segments, source-side sums
  const int4 *hgroups;
  const int2 *hzones;
  const double4 *hcen;
  const int2 *hsegs;
  float4 *vsrc;            // source-side sums, slot = brick-order position
  const uint32_t *bperm;   // brick-order position -> caller index
  float refine2;
  double fself_r, fself_i;
  // pair-once systems: the interpolation adds the source-side sums into V
  // (potential times vs, gradient times gs) and clears them
  int fold;
  double vs, gs;
};

// The system that owns work unit u of a class (off: prefix sums of the units).
__device__ __forceinline__ int find_sys(const long long *__restrict__ off, int count,
                                        long long u) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= u) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// The direct sums of one class (the pair-once walk or the one-sided one) with
// ng groups in all: one launch.
void launch_batch_direct(const PairCoef<float> &k, bool once, bool alpha_positive,
                         const BatchSys *sys, const long long *off, int count, long long ng,
                         cudaStream_t s);

}  // namespace npme
