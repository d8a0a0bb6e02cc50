// Device bodies of the per-call kernels, shared by the single-system kernels
// (recsum.cu, direct.cu) and the multi-system batch kernels (batch.cu).  Each
// body processes one unit of work (one point, one brick, one spectrum
// element, one warp group) of one system; the kernels only map threads to
// (system, unit).
#pragma once

#include "internal.h"

namespace npme {

#ifndef NPME_GROUP_MIN_BLOCKS
#define NPME_GROUP_MIN_BLOCKS 1
#endif
constexpr int kGroupMinBlocks = NPME_GROUP_MIN_BLOCKS;  // resident CTAs asked of ptxas
#ifndef NPME_DIRECT_UNROLL
#define NPME_DIRECT_UNROLL 8
#endif
constexpr int kDirectUnroll = NPME_DIRECT_UNROLL;  // pair-loop unroll factor

// Charges into the direct sum's source order (dperm: source slot -> caller
// index) and the bulk precision; the spread reads the caller's charges itself.
template <typename T, bool CPLX>
__device__ __forceinline__ void gather_body(const double *__restrict__ q,
                                            const uint32_t *__restrict__ dperm,
                                            T *__restrict__ qc, long i) {
  const long o = dperm[i];
  if (CPLX) {
    qc[2 * i] = (T)q[2 * o];
    qc[2 * i + 1] = (T)q[2 * o + 1];
  } else {
    qc[i] = (T)q[o];
  }
}

// Unroll of the outer stencil axis: complete up to order 12; orders 14 and
// 16 (up to 16^3 = 4,096 stencil points) keep it as a loop, so the unrolled
// inner P^2 block stays a size the instruction cache holds.
template <int P>
constexpr int kStencilUnroll = P <= 12 ? P : 1;

// Points of a brick are stored in rounds over the shared-memory banks of
// their stencil origins in the brick's tile (set-up, setup.cu): round r holds
// the r-th point of every bank that has more than r points, in bank order.
// Virtual warp vw of a brick with nb points takes the 32 consecutive points
// at positions 32 vw + lane (contiguous record loads).  Two lanes share a
// bank only where a warp's run of 32 spans rounds; but the bank counts of a
// brick are Poisson-like (uniform points over 512 stencil origins, 16 per
// bank), so a brick's fullest bank usually holds more points than the brick
// has warps, and no assignment of one point per lane avoids conflicts: at
// 1M points (244 per brick) a stencil step costs 2.08 shared wavefronts per
// warp on average, against 1.71 for the best possible assignment and 1 for
// none.
__device__ __forceinline__ int brick_point(int nb, int vw, int lane) {
  const int p = vw * 32 + lane;
  return p < nb ? p : -1;
}

// Spread of one brick by the whole CTA (src/RecSumQ.cpp:184-314): the
// brick's points accumulate their p^3 stencils into the shared tile of
// (kBrick + P - 1)^3 grid points, which is then added to the global grid.
template <typename T, int P, bool CPLX>
__device__ __forceinline__ void spread_brick_body(int brick, const int *__restrict__ brick_start,
                                                  const BrickPoint<T> *__restrict__ bp,
                                                  const double *__restrict__ q,
                                                  T *__restrict__ grid, int nb2, int nb3, long N1,
                                                  long N2, long N3, T *tile) {
  constexpr int TL = kBrick + P - 1;
  constexpr int TV = TL * TL * TL;
  constexpr int C = CPLX ? 2 : 1;
  const int b3 = brick % nb3, b2 = (brick / nb3) % nb2, b1 = brick / (nb3 * nb2);
  for (int t = threadIdx.x; t < TV * C; t += blockDim.x) tile[t] = T(0);
  __syncthreads();
  const int beg = brick_start[brick], nbp = brick_start[brick + 1] - beg;
  const int nvw = (nbp + 31) >> 5, lane = threadIdx.x & 31;
  for (int vw = threadIdx.x >> 5; vw < nvw; vw += blockDim.x >> 5) {
    const int pi = brick_point(nbp, vw, lane);
    if (pi < 0) continue;
    const BrickPoint<T> pt = bp[beg + pi];
    T w1[P], w2[P], w3[P], dummy[P];
    bspline_weights<T, P, false>(pt.u[0], w1, dummy);
    bspline_weights<T, P, false>(pt.u[1], w2, dummy);
    bspline_weights<T, P, false>(pt.u[2], w3, dummy);
    const int l1 = (int)(pt.g0 >> 20) - b1 * kBrick;
    const int l2 = (int)((pt.g0 >> 10) & 1023u) - b2 * kBrick;
    const int l3 = (int)(pt.g0 & 1023u) - b3 * kBrick;
    const T qr = (T)q[C * (long)pt.orig], qi = CPLX ? (T)q[2 * (long)pt.orig + 1] : T(0);
#pragma unroll(kStencilUnroll<P>)
    for (int t1 = 0; t1 < P; t1++) {
#pragma unroll
      for (int t2 = 0; t2 < P; t2++) {
        const T c12 = w1[t1] * w2[t2];
        T *row = tile + C * (((l1 + t1) * TL + (l2 + t2)) * TL + l3);
#pragma unroll
        for (int t3 = 0; t3 < P; t3++) {
          const T c = c12 * w3[t3];
          atomicAdd(row + C * t3, c * qr);
          if (CPLX) atomicAdd(row + C * t3 + 1, c * qi);
        }
      }
    }
  }
  __syncthreads();
  const long g1 = (long)b1 * kBrick, g2 = (long)b2 * kBrick, g3 = (long)b3 * kBrick;
  for (int t = threadIdx.x; t < TV; t += blockDim.x) {
    const int i3 = t % TL, i2 = (t / TL) % TL, i1 = t / (TL * TL);
    if (g1 + i1 >= N1) continue;
    if (g2 + i2 >= N2 || g3 + i3 >= N3) continue;  // beyond the box: always zero
    const long gi = ((g1 + i1) * N2 + (g2 + i2)) * N3 + (g3 + i3);
#pragma unroll
    for (int c = 0; c < C; c++) {
      const T v = tile[C * t + c];
      if (v != T(0)) atomicAdd(grid + C * gi + c, v);
    }
  }
}

// FP32 spreading with two native 32-bit integer shared atomics per
// contribution instead of one floating-point shared atomic (which the
// hardware does not have and executes as a compare-and-swap loop; a probe
// ran 3.5x faster with integer atomics).  Each contribution v = c q is
// scaled by S = 2^k so that |v S| <= 2^B, B = min(21, 30 - ceil(log2
// n_brick)): the high words round(v S) of all contributions to a tile point
// cannot exceed 2^30 in sum, and the low words round((v S - hi) 2^B) carry
// B more bits.  The integer sums are exact and independent of the order of
// the atomics; each tile value hi + lo 2^-L is rounded once, to float, when
// it is added to the grid.  Same points, weights and tile as
// spread_brick_body.
template <int P, bool CPLX>
__device__ __forceinline__ void spread_brick_fixed(int brick, const int *__restrict__ brick_start,
                                                   const BrickPoint<float> *__restrict__ bp,
                                                   const double *__restrict__ q,
                                                   float *__restrict__ grid, int nb2, int nb3,
                                                   long N1, long N2, long N3, int *tile) {
  constexpr int TL = kBrick + P - 1;
  constexpr int TV = TL * TL * TL;
  constexpr int C = CPLX ? 2 : 1;
  __shared__ float s_max[32];
  int *thi = tile, *tlo = tile + TV * C;
  const int b3 = brick % nb3, b2 = (brick / nb3) % nb2, b1 = brick / (nb3 * nb2);
  for (int t = threadIdx.x; t < 2 * TV * C; t += blockDim.x) tile[t] = 0;
  const int beg = brick_start[brick], nbp = brick_start[brick + 1] - beg;
  float m = 0.f;
  for (int i = threadIdx.x; i < nbp; i += blockDim.x) {
    const long o = bp[beg + i].orig;
    m = fmaxf(m, fabsf((float)q[C * o]));
    if (CPLX) m = fmaxf(m, fabsf((float)q[2 * o + 1]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
  m = s_max[0];
  for (int w = 1; w < nw; w++) m = fmaxf(m, s_max[w]);
  if (m == 0.f) return;  // nothing to spread (the whole CTA returns)
  const int lnb = 32 - __clz(max(nbp - 1, 1));  // ceil(log2(nbp)), nbp >= 2
  // bits per contribution: sums of nbp of them stay below 2^30, and single
  // words below 2^22 so that a float converts to int by the add-magic trick
  const int B = min(21, 30 - lnb);
  const int k = max(-120, min(120, B - (ilogbf(m) + 1)));
  const int L = B;
  const float S = ldexpf(1.f, k), SL = ldexpf(1.f, L);
  const int nvw = (nbp + 31) >> 5;
  for (int vw = threadIdx.x >> 5; vw < nvw; vw += nw) {
    const int pi = brick_point(nbp, vw, lane);
    if (pi < 0) continue;
    const BrickPoint<float> pt = bp[beg + pi];
    float w1[P], w2[P], w3[P], dummy[P];
    bspline_weights<float, P, false>(pt.u[0], w1, dummy);
    bspline_weights<float, P, false>(pt.u[1], w2, dummy);
    bspline_weights<float, P, false>(pt.u[2], w3, dummy);
    const int l1 = (int)(pt.g0 >> 20) - b1 * kBrick;
    const int l2 = (int)((pt.g0 >> 10) & 1023u) - b2 * kBrick;
    const int l3 = (int)(pt.g0 & 1023u) - b3 * kBrick;
    const float qr = (float)q[C * (long)pt.orig] * S;
    const float qi = CPLX ? (float)q[2 * (long)pt.orig + 1] * S : 0.f;
#pragma unroll(kStencilUnroll<P>)
    for (int t1 = 0; t1 < P; t1++) {
#pragma unroll
      for (int t2 = 0; t2 < P; t2++) {
        const float c12 = w1[t1] * w2[t2];
        const int row = C * (((l1 + t1) * TL + (l2 + t2)) * TL + l3);
#pragma unroll
        for (int t3 = 0; t3 < P; t3++) {
          const float c = c12 * w3[t3];
#pragma unroll
          for (int part = 0; part < C; part++) {
            // |v| <= 2^21: adding 1.5 * 2^23 rounds v to an integer held in
            // the low mantissa bits (no conversion instruction needed)
            constexpr float kMagic = 12582912.f;
            const float v = c * (part ? qi : qr);
            const float vm = v + kMagic;
            const float r = v - (vm - kMagic);  // exact remainder, |r| <= 1/2
            atomicAdd(thi + row + C * t3 + part, __float_as_int(vm) - 0x4B400000);
            atomicAdd(tlo + row + C * t3 + part,
                      __float_as_int(fmaf(r, SL, kMagic)) - 0x4B400000);
          }
        }
      }
    }
  }
  __syncthreads();
  const float invS = ldexpf(1.f, -k), invSL = ldexpf(1.f, -L);
  const long g1 = (long)b1 * kBrick, g2 = (long)b2 * kBrick, g3 = (long)b3 * kBrick;
  for (int t = threadIdx.x; t < TV; t += blockDim.x) {
    const int i3 = t % TL, i2 = (t / TL) % TL, i1 = t / (TL * TL);
    if (g1 + i1 >= N1) continue;
    if (g2 + i2 >= N2 || g3 + i3 >= N3) continue;  // beyond the box: always zero
    const long gi = ((g1 + i1) * N2 + (g2 + i2)) * N3 + (g3 + i3);
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int hv = thi[C * t + c], lv = tlo[C * t + c];
      if (hv != 0 || lv != 0) {
        const double v = ((double)hv + (double)lv * (double)invSL) * (double)invS;
        atomicAdd(grid + C * gi + c, (float)v);
      }
    }
  }
}

// Spreading without atomics, orders up to 8: the CTA's warp w takes the
// brick's points whose stencil starts at x = w of the tile, so that all of them
// touch the tile's planes w .. w + P - 1, and keeps those planes in registers:
// lane (z, y half) holds P x H sums, H = half of the tile's y range.  A point
// is one sweep of multiply-adds of its zero-padded weights over these registers
// (weights of a batch of points computed one point per lane, passed through
// shared memory).  Most of them multiply zeros (36 of 224 cells per plane are
// in the stencil at order 6), but they run on the FMA pipes of four schedulers,
// where the shared-memory atomics queue in one pipe, two per contribution with
// two wavefronts each (spread_brick_fixed).  At the end the warps add their
// planes to the shared tile in P steps, each on a plane of its own, and the
// tile goes to the global grid with atomics.  Sums are in T: two
// roundings per contribution (q w3, then times w2; the product with w1 is
// fused), one fewer than with the products of the fixed-point form.
template <typename T, int P, bool CPLX>
struct SpreadOwner {
  static constexpr bool kUse = P <= 8;
  static constexpr int TL = kBrick + P - 1, H = (TL + 1) / 2;
  static constexpr int C = CPLX ? 2 : 1;
  // complex FP64 sums do not fit the registers together: one pass per part
  static constexpr int CC = (CPLX && sizeof(T) == 4) ? 2 : 1;
  static constexpr int kBatch = sizeof(T) == 4 ? 32 : 16;  // points per batch
  static constexpr int kRow = 20, kX = 12;  // padded rows: z and y weights; x weights and q
  static constexpr size_t kRowBytes = sizeof(T) * kBatch * (2 * kRow + kX);  // a warp's rows
  static constexpr size_t kWarpBytes = kRowBytes + sizeof(int) * 64;
  static constexpr size_t kTileBytes = sizeof(T) * C * TL * TL * TL;
  static constexpr size_t kBytes = kBrick * kWarpBytes + kTileBytes;
  // spread_brick_shared: the window's points by plane and their counters; the
  // tile's second words
  static constexpr int kChunks = kSpreadWindow / 32;
  static constexpr size_t kSortBytes = 2 * kSpreadWindow + sizeof(int) * kBrick * kChunks;
  static constexpr size_t kSharedBytes =
      kBrick * kRowBytes + kSortBytes + (sizeof(T) == 4 ? 2 : 1) * kTileBytes;
};

// Points at(0) .. at(n - 1) (n <= kBatch) of a brick into the calling warp's sums, which
// are the tile's planes from the points' own on; rows: the warp's shared rows.
template <typename T, int P, bool CPLX, class At>
__device__ __forceinline__ void spread_batch(
    T (&acc)[SpreadOwner<T, P, CPLX>::CC][P][SpreadOwner<T, P, CPLX>::H], int n, const At &at,
    const BrickPoint<T> *__restrict__ bp, const double *__restrict__ q, int pass, int b2, int b3,
    T *rows, int lane) {
  using S = SpreadOwner<T, P, CPLX>;
  using V4 = typename Vec4<T>::type;
  constexpr int H = S::H, C = S::C, CC = S::CC;
  const int zl = lane & 15, half = lane >> 4;
  T *wz = rows, *wy = wz + S::kBatch * S::kRow, *wx = wy + S::kBatch * S::kRow;
  if (lane < n) {
    const BrickPoint<T> pt = bp[at(lane)];
    T a[P], dummy[P];
    T *rz = wz + lane * S::kRow, *ry = wy + lane * S::kRow, *rx = wx + lane * S::kX;
    V4 zero;
    zero.x = zero.y = zero.z = zero.w = T(0);
#pragma unroll
    for (int i = 0; i < 4; i++)
      reinterpret_cast<V4 *>(rz)[i] = zero, reinterpret_cast<V4 *>(ry)[i] = zero;
    const long o = pt.orig;
    T qz = T(1);
    if (CC == 2) {
      rx[8] = (T)q[2 * o], rx[9] = (T)q[2 * o + 1];
    } else {
      qz = (T)q[C * o + pass];
    }
    bspline_weights<T, P, false>(pt.u[2], a, dummy);
    const int l3 = (int)(pt.g0 & 1023u) - b3 * kBrick;
#pragma unroll
    for (int t = 0; t < P; t++) rz[l3 + t] = CC == 2 ? a[t] : qz * a[t];
    bspline_weights<T, P, false>(pt.u[1], a, dummy);
    const int l2 = (int)((pt.g0 >> 10) & 1023u) - b2 * kBrick;
#pragma unroll
    for (int t = 0; t < P; t++) {
      const int y = l2 + t;
      ry[y < H ? y : 8 + y - H] = a[t];
    }
    bspline_weights<T, P, false>(pt.u[0], a, dummy);
#pragma unroll
    for (int t = 0; t < P; t++) rx[t] = a[t];
  }
  __syncwarp();
#pragma unroll 1
  for (int p = 0; p < n; p++) {
    const T z = wz[p * S::kRow + zl];
    T y[8], x[8];
    const V4 *vy = reinterpret_cast<const V4 *>(wy + p * S::kRow + 8 * half);
    const V4 *vx = reinterpret_cast<const V4 *>(wx + p * S::kX);
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const V4 ay = vy[i], ax = vx[i];
      y[4 * i] = ay.x, y[4 * i + 1] = ay.y, y[4 * i + 2] = ay.z, y[4 * i + 3] = ay.w;
      x[4 * i] = ax.x, x[4 * i + 1] = ax.y, x[4 * i + 2] = ax.z, x[4 * i + 3] = ax.w;
    }
#pragma unroll
    for (int c = 0; c < CC; c++) {
      const T s = CC == 2 ? z * wx[p * S::kX + 8 + c] : z;
#pragma unroll
      for (int h = 0; h < H; h++) {
        const T v = s * y[h];
#pragma unroll
        for (int i = 0; i < P; i++) acc[c][i][h] = fma(x[i], v, acc[c][i][h]);
      }
    }
  }
  __syncwarp();
}

// The tile's rows to the grid, FP32 in pieces of 16 bytes: one vector atomic
// each (the atomic units count requests, and with 4 to 7 tile values per grid
// point they, not the sums, would be the bound).  A row starts at a multiple
// of 8 values; rows of the grid that are not 16-byte aligned, and pieces past
// the end of a row, go value by value.  TWO: the tile's second words are added.
template <typename T, int P, bool CPLX, bool TWO>
__device__ __forceinline__ void spread_tile_out(const T *tile, T *__restrict__ grid, int b1, int b2,
                                                int b3, long N1, long N2, long N3) {
  using S = SpreadOwner<T, P, CPLX>;
  constexpr int TL = S::TL, C = S::C;
  constexpr int kPiece = sizeof(T) == 4 ? 4 / C : 1;  // grid points per piece
  constexpr int kPieces = (TL + kPiece - 1) / kPiece;
  const T *low = tile + TL * TL * TL * C;
  const long g1 = (long)b1 * kBrick, g2 = (long)b2 * kBrick, g3 = (long)b3 * kBrick;
  const bool aligned = (N3 * C) % 4 == 0;
  for (int t = threadIdx.x; t < TL * TL * kPieces; t += blockDim.x) {
    const int row = t / kPieces, i3 = (t - row * kPieces) * kPiece;
    const int i1 = row / TL, i2 = row - i1 * TL;
    if (g1 + i1 >= N1 || g2 + i2 >= N2) continue;  // always zero there
    T *d = grid + C * (((g1 + i1) * N2 + (g2 + i2)) * N3 + (g3 + i3));
    T v[kPiece * C];
    bool any = false;
#pragma unroll
    for (int m = 0; m < kPiece * C; m++) {
      const int at = C * (row * TL + i3) + m;
      v[m] = i3 + m / C < TL ? tile[at] : T(0);
      if (TWO && i3 + m / C < TL) v[m] += low[at];
      any |= v[m] != T(0);
    }
    if (!any) continue;
    if constexpr (sizeof(T) == 4) {
      if (aligned && g3 + i3 + kPiece <= N3) {
        atomicAdd(reinterpret_cast<float4 *>(d), make_float4(v[0], v[1], v[2], v[3]));
        continue;
      }
    }
#pragma unroll
    for (int m = 0; m < kPiece * C; m++)
      if (v[m] != T(0) && g3 + i3 + m / C < N3) atomicAdd(d + m, v[m]);
  }
}

template <typename T, int P, bool CPLX>
__device__ __forceinline__ void spread_brick_owner(int brick, const int *__restrict__ brick_start,
                                                   const BrickPoint<T> *__restrict__ bp,
                                                   const double *__restrict__ q,
                                                   T *__restrict__ grid, int nb2, int nb3, long N1,
                                                   long N2, long N3, unsigned char *smem) {
  using S = SpreadOwner<T, P, CPLX>;
  constexpr int TL = S::TL, TV = TL * TL * TL, H = S::H, C = S::C, CC = S::CC, KB = S::kBatch;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, zl = lane & 15, half = lane >> 4;
  T *tile = reinterpret_cast<T *>(smem + kBrick * S::kWarpBytes);
  T *wz = reinterpret_cast<T *>(smem + w * S::kWarpBytes);
  int *list = reinterpret_cast<int *>(smem + w * S::kWarpBytes + S::kRowBytes);
  const int b3 = brick % nb3, b2 = (brick / nb3) % nb2, b1 = brick / (nb3 * nb2);
  const int beg = brick_start[brick], nbp = brick_start[brick + 1] - beg;
  for (int t = threadIdx.x; t < TV * C; t += blockDim.x) tile[t] = T(0);
  for (int pass = 0; pass < C / CC; pass++) {
    T acc[CC][P][H];
#pragma unroll
    for (int c = 0; c < CC; c++)
#pragma unroll
      for (int x = 0; x < P; x++)
#pragma unroll
        for (int h = 0; h < H; h++) acc[c][x][h] = T(0);
    auto batch = [&](int n) {  // points list[0 .. n) into the sums
      spread_batch<T, P, CPLX>(acc, n, [&](int i) { return list[i]; }, bp + beg, q, pass, b2, b3,
                               wz, lane);
    };
    // the warp's points, in batches
    int cnt = 0;
    uint32_t g0[4];  // four chunks of origins in flight (137 -> 131 us at 1M, FP32 order 6)
    for (int c0 = 0; c0 < nbp; c0 += 32) {
      if ((c0 & 127) == 0) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int i = c0 + 32 * u + lane;
          g0[u] = i < nbp ? bp[beg + i].g0 : 0xffffffffu;
        }
      }
      const int i = c0 + lane, u = c0 >> 5 & 3;
      const uint32_t g = u < 2 ? (u == 0 ? g0[0] : g0[1]) : (u == 2 ? g0[2] : g0[3]);
      const bool mine = i < nbp && (int)(g >> 20) - b1 * kBrick == w;
      const unsigned m = __ballot_sync(FULL, mine);
      if (mine) list[cnt + __popc(m & ((1u << lane) - 1u))] = i;
      cnt += __popc(m);
      __syncwarp();
      while (cnt >= KB) {
        batch(KB);
        const int rest = cnt - KB, next = lane < rest ? list[KB + lane] : 0;
        __syncwarp();
        if (lane < rest) list[lane] = next;
        __syncwarp();
        cnt = rest;
      }
    }
    if (cnt > 0) batch(cnt);
    // planes w + s of all warps are different ones in every step s
#pragma unroll
    for (int s = 0; s < P; s++) {
      __syncthreads();
#pragma unroll
      for (int h = 0; h < H; h++) {
        const int y = half * H + h;
        if (y < TL && zl < TL) {
          T *d = tile + C * (((w + s) * TL + y) * TL + zl) + pass;
#pragma unroll
          for (int c = 0; c < CC; c++) d[c] += acc[c][s][h];
        }
      }
    }
  }
  __syncthreads();
  spread_tile_out<T, P, CPLX, false>(tile, grid, b1, b2, b3, N1, N2, N3);
}

// The same for an odd brick (set-up, place_orders_kernel), one with many points in one
// plane x.  Above, a warp would be alone with them, and their number would set the
// error of FP32 sums: 200,000 points in a sheet normal to x (3,125 a brick), order 6,
// took 307 us, 93 here and 104 in fixed point; in one to eight bricks, order 8,
// they were off by 9e-5, 5e-7 here and 6e-7 in fixed point.
// Here the points are taken kSpreadWindow at a time, sorted by plane; a plane with
// more than a fifth of a window (and 32 points) is shared out over all warps, the
// others go to their own warp.  FP32 runs in registers have at most a third of a
// window's points, and the runs are collected in two floats per tile value.
template <typename T, int P, bool CPLX>
__device__ __forceinline__ void spread_brick_shared(int brick, const int *__restrict__ brick_start,
                                                    const BrickPoint<T> *__restrict__ bp,
                                                    const double *__restrict__ q,
                                                    T *__restrict__ grid, int nb2, int nb3,
                                                    long N1, long N2, long N3,
                                                    unsigned char *smem) {
  using S = SpreadOwner<T, P, CPLX>;
  constexpr int TL = S::TL, TV = TL * TL * TL, H = S::H, C = S::C, CC = S::CC, KB = S::kBatch;
  constexpr bool kTwo = sizeof(T) == 4;
  constexpr int kLoads = kSpreadWindow / 256;
  static_assert(kBrick == 8 && kLoads == 4, "8 warps, 8 counters a lane");
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, zl = lane & 15, half = lane >> 4;
  T *rows = reinterpret_cast<T *>(smem + w * S::kRowBytes);
  uint16_t *list = reinterpret_cast<uint16_t *>(smem + kBrick * S::kRowBytes);
  int *count = reinterpret_cast<int *>(list + kSpreadWindow);  // [plane][chunk of 32 points]
  T *tile = reinterpret_cast<T *>(smem + kBrick * S::kRowBytes + S::kSortBytes);
  const int b3 = brick % nb3, b2 = (brick / nb3) % nb2, b1 = brick / (nb3 * nb2);
  const int beg = brick_start[brick], nbp = brick_start[brick + 1] - beg;
  for (int t = threadIdx.x; t < (kTwo ? 2 : 1) * TV * C; t += blockDim.x) tile[t] = T(0);
  for (int pass = 0; pass < C / CC; pass++) {
    T acc[CC][P][H];
    auto clear = [&]() {
#pragma unroll
      for (int c = 0; c < CC; c++)
#pragma unroll
        for (int x = 0; x < P; x++)
#pragma unroll
          for (int h = 0; h < H; h++) acc[c][x][h] = T(0);
    };
    clear();
    int run = 0;  // points in the fullest warp's sums at most
    for (int w0 = 0; w0 < nbp; w0 += kSpreadWindow) {
      const int nw = min(kSpreadWindow, nbp - w0);
      // the window's points sorted by plane: chunk i is points 32 i .. of it
      int plane[kLoads], rank[kLoads];
#pragma unroll
      for (int u = 0; u < kLoads; u++) {
        const int i = 256 * u + threadIdx.x;
        plane[u] = i < nw ? (int)(bp[beg + w0 + i].g0 >> 20) - b1 * kBrick : -1;
      }
      __syncthreads();  // the last window's list is done with
#pragma unroll
      for (int u = 0; u < kLoads; u++) {
        int mine = 0;
        rank[u] = 0;
#pragma unroll
        for (int p = 0; p < kBrick; p++) {
          const unsigned m = __ballot_sync(FULL, plane[u] == p);
          if (plane[u] == p) rank[u] = __popc(m & ((1u << lane) - 1u));
          if (lane == p) mine = __popc(m);
        }
        if (lane < kBrick) count[lane * S::kChunks + 8 * u + w] = mine;
      }
      __syncthreads();
      // every warp: the places of the counters; lane 4 p + u has those of chunks 8 u ..
      const int4 n0 = reinterpret_cast<const int4 *>(count)[2 * lane];
      const int4 n1 = reinterpret_cast<const int4 *>(count)[2 * lane + 1];
      const int c[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
      int sum = 0, before = 0;  // before: this warp's counter
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (i < w) before += c[i];
        sum += c[i];
      }
      int first = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, first, o);
        if (lane >= o) first += v;
      }
      first -= sum;
#pragma unroll
      for (int u = 0; u < kLoads; u++) {
        const int p = __shfl_sync(FULL, first + before, 4 * max(plane[u], 0) + u);
        if (plane[u] >= 0) list[p + rank[u]] = (uint16_t)(256 * u + threadIdx.x);
      }
      // start and points of plane lane (lanes 0 .. 7), the planes to share out
      const int start = __shfl_sync(FULL, first, 4 * (lane & 7));
      const int next = __shfl_sync(FULL, first, (4 * (lane & 7) + 4) & 31);
      const int npl = ((lane & 7) < 7 ? next : nw) - start;
      const bool many = npl > max(32, nw / 5);
      unsigned over = __ballot_sync(FULL, many) & 0xffu;
      const int most = __reduce_max_sync(FULL, many ? 0 : npl);
      __syncthreads();
      // rounds: the warps' own planes, then the shared ones; the sums go to the tile
      // when the next points would not fit the run, before another plane's and at the
      // end
      const bool last = w0 + nw == nbp;
      bool own = true;
      do {
        int pl = w, from = __shfl_sync(FULL, start, w), n = __shfl_sync(FULL, npl, w);
        if (own) {
          if (over >> w & 1) n = 0;
          run += most;
        } else {  // this warp's share of a plane of many
          pl = __ffs(over) - 1;
          over &= over - 1;
          const int m = __shfl_sync(FULL, npl, pl), a = w * m >> 3, b = (w + 1) * m >> 3;
          from = __shfl_sync(FULL, start, pl) + a, n = b - a;
          run = 1;
        }
        for (; n > 0; from += KB, n -= KB)
          spread_batch<T, P, CPLX>(acc, min(n, KB), [&](int i) { return (int)list[from + i]; },
                                   bp + beg + w0, q, pass, b2, b3, rows, lane);
        const bool flush = own ? run > 0 && (over != 0 || last || run > kSpreadWindow / 8) : true;
        if (flush) {
          // in step s plane w + s of every warp's own P, or, of one plane's P, number
          // (w + s) mod 8
          for (int s = 0; s < (own ? P : kBrick); s++) {
            __syncthreads();
            const int k = own ? s : (w + s) & (kBrick - 1);
#pragma unroll
            for (int i = 0; i < P; i++) {
              if (i != k || zl >= TL) continue;
              T *d = tile + C * (((pl + i) * TL + half * H) * TL + zl) + pass;
              T v[CC][H];
#pragma unroll
              for (int c = 0; c < CC; c++)
#pragma unroll
                for (int h = 0; h < H; h++)
                  v[c][h] = half * H + h < TL ? d[C * TL * h + c] : T(0);
              if (kTwo) {  // what the additions round off (Knuth's two-sum)
                T e[CC][H];
#pragma unroll
                for (int c = 0; c < CC; c++)
#pragma unroll
                  for (int h = 0; h < H; h++) {
                    const T t = v[c][h], a = acc[c][i][h], x = t + a, b = x - t;
                    e[c][h] = half * H + h < TL ? (d + TV * C)[C * TL * h + c] : T(0);
                    e[c][h] += (t - (x - b)) + (a - b);
                  }
#pragma unroll
                for (int c = 0; c < CC; c++)
#pragma unroll
                  for (int h = 0; h < H; h++)
                    if (half * H + h < TL) (d + TV * C)[C * TL * h + c] = e[c][h];
              }
#pragma unroll
              for (int c = 0; c < CC; c++)
#pragma unroll
                for (int h = 0; h < H; h++)
                  if (half * H + h < TL) d[C * TL * h + c] = v[c][h] + acc[c][i][h];
            }
          }
          clear();
          run = 0;
        }
        own = false;
      } while (over != 0);
    }
  }
  __syncthreads();
  spread_tile_out<T, P, CPLX, kTwo>(tile, grid, b1, b2, b3, N1, N2, N3);
}

// FP32 order 4: its stencil of 64 points is too small for the sweep over zero-padded
// weights to pay in full bricks: odd ones, and for real kernels those of more than
// kFixedFrom4 points, take the fixed-point form (uniform points, 390 a brick: 23.5 us
// against 29.9; 78 a brick: 17.3 and 17.6; 8 a brick: 17.2 and 14.3).
constexpr int kFixedFrom4 = 96;

// Entries of the list of non-empty bricks: the brick, and whether it is odd.
__device__ __forceinline__ int list_brick(int e) { return e & 0x7fffffff; }

// resident CTAs of spread_brick_shared, by shared memory and registers for its sums
template <typename T, int P, bool CPLX>
constexpr int kSpreadOddCtas = sizeof(T) == 4 ? (P <= 6 && !CPLX ? 3 : P == 8 && CPLX ? 1 : 2)
                                              : (P <= 6 ? 2 : 1);

// true when odd bricks are left to a launch of their own (spread_brick_shared)
template <typename T, int P>
constexpr bool kSpreadApart = P <= 8 && !(P == 4 && sizeof(T) == 4);

// The spread body of an order and precision for the brick of a list entry (apart: odd
// ones are left out), and its shared memory.
template <typename T, int P, bool CPLX>
__device__ __forceinline__ void spread_brick(int entry, const int *__restrict__ brick_start,
                                             const BrickPoint<T> *__restrict__ bp,
                                             const double *__restrict__ q, T *__restrict__ grid,
                                             int nb2, int nb3, long N1, long N2, long N3,
                                             unsigned char *smem, bool apart) {
  const int brick = list_brick(entry);
  if constexpr (SpreadOwner<T, P, CPLX>::kUse) {
    if constexpr (kSpreadApart<T, P>) {
      if (apart && entry < 0) return;
    } else {
      const int n = brick_start[brick + 1] - brick_start[brick];
      if (entry < 0 || (!CPLX && n > kFixedFrom4)) {
        spread_brick_fixed<P, CPLX>(brick, brick_start, bp, q, grid, nb2, nb3, N1, N2, N3,
                                    reinterpret_cast<int *>(smem));
        return;
      }
    }
    spread_brick_owner<T, P, CPLX>(brick, brick_start, bp, q, grid, nb2, nb3, N1, N2, N3, smem);
  } else if constexpr (std::is_same<T, float>::value)
    spread_brick_fixed<P, CPLX>(brick, brick_start, bp, q, grid, nb2, nb3, N1, N2, N3,
                                reinterpret_cast<int *>(smem));
  else
    spread_brick_body<T, P, CPLX>(brick, brick_start, bp, q, grid, nb2, nb3, N1, N2, N3,
                                  reinterpret_cast<T *>(smem));
}

template <typename T, int P, bool CPLX>
constexpr size_t spread_smem() {
  constexpr int TL = kBrick + P - 1;
  // fixed point: two int words per tile value; FP64: one double
  return SpreadOwner<T, P, CPLX>::kUse
             ? SpreadOwner<T, P, CPLX>::kBytes
             : (sizeof(T) == 4 ? 8 : sizeof(T)) * TL * TL * TL * (CPLX ? 2 : 1);
}

// X(k) *= G(|k1|, |k2|, k3) on the R2C half spectrum (src/RecSumV.cpp:639-707),
// one spectrum row (k1, k2) = (r / N2, r % N2) per warp: one division per
// row, and the lanes stride the row's contiguous k3 run (coalesced X and G
// rows; the compact G octant stays in L2).
template <typename T>
__device__ __forceinline__ void multiply_real_row(typename Vec2<T>::type *__restrict__ X,
                                                  const T *__restrict__ G, int r, int N1, int N2,
                                                  int N3h, int M2, int M3, int lane) {
  const int k1 = r / N2, k2 = r - k1 * N2;
  const int f1 = k1 <= N1 / 2 ? k1 : N1 - k1;
  const int f2 = k2 <= N2 / 2 ? k2 : N2 - k2;
  const T *__restrict__ g = G + ((long)f1 * M2 + f2) * M3;
  typename Vec2<T>::type *__restrict__ x = X + (long)r * N3h;
  for (int k3 = lane; k3 < N3h; k3 += 32) {
    const T gv = __ldg(g + k3);
    typename Vec2<T>::type v = x[k3];
    v.x *= gv;
    v.y *= gv;
    x[k3] = v;
  }
}

// X(k) *= G(|k1|, |k2|, |k3|) on the full complex spectrum, one row per warp.
template <typename T>
__device__ __forceinline__ void multiply_cplx_row(typename Vec2<T>::type *__restrict__ X,
                                                  const typename Vec2<T>::type *__restrict__ G,
                                                  int r, int N1, int N2, int N3, int M2, int M3,
                                                  int lane) {
  const int k1 = r / N2, k2 = r - k1 * N2;
  const int f1 = k1 <= N1 / 2 ? k1 : N1 - k1;
  const int f2 = k2 <= N2 / 2 ? k2 : N2 - k2;
  const typename Vec2<T>::type *__restrict__ g = G + ((long)f1 * M2 + f2) * M3;
  typename Vec2<T>::type *__restrict__ x = X + (long)r * N3;
  for (int k3 = lane; k3 < N3; k3 += 32) {
    const int f3 = k3 <= N3 / 2 ? k3 : N3 - k3;
    const typename Vec2<T>::type gv = g[f3];
    const typename Vec2<T>::type v = x[k3];
    typename Vec2<T>::type o;
    o.x = v.x * gv.x - v.y * gv.y;
    o.y = v.x * gv.y + v.y * gv.x;
    x[k3] = o;
  }
}

// One element of the windowed eight-image sum that samples f_LR on the
// compact octant for the kernel transform (src/RecSumGrid.cpp:45-282): per
// axis the two image coordinates x1, x2 and window values T1, T2 are stored
// as ax[0..M) = x1, ax[M..2M) = x2, ax[2M..3M) = T1, ax[3M..4M) = T2.  LR is
// a functor double2 operator()(double r2) returning f_LR (re, im).
template <class LR>
__device__ __forceinline__ double2 fhat_sample_body(const LR &lr, long idx, int M1, int M2,
                                                    int M3, const double *__restrict__ ax,
                                                    const double *__restrict__ ay,
                                                    const double *__restrict__ az) {
  const int i3 = idx % M3, i2 = (idx / M3) % M2, i1 = idx / ((long)M2 * M3);
  double sr = 0, si = 0;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int s1 = c >> 2, s2 = (c >> 1) & 1, s3 = c & 1;
    const double x = ax[s1 * M1 + i1], y = ay[s2 * M2 + i2], z = az[s3 * M3 + i3];
    const double t = ax[(2 + s1) * M1 + i1] * ay[(2 + s2) * M2 + i2] * az[(2 + s3) * M3 + i3];
    if (t == 0.0) continue;
    const double2 f = lr(x * x + y * y + z * z);
    sr += t * f.x;
    si += t * f.y;
  }
  return make_double2(sr, si);
}

// Interpolation of one brick by the whole CTA (src/RecSumV.cpp:201-306):
// the brick's theta tile of (kBrick + P - 1)^3 grid points is read into
// shared memory once, then every point gathers its p^3 stencil from the
// tile: V += sum theta B1 B2 B3, grad += (N/L) sum theta dB ..., added into
// the caller-order output; c1, c2, c3 are N/L times the scale of weights to
// that of their derivatives (bspline_weights).  With vsrc (CalcV after a pair-once direct sum)
// the point's source-side direct-sum slot (same brick-order position) is
// added in the same read-modify-write of V (potential scaled by vs,
// gradient by gs) and cleared for the next call.
template <typename T, int P, bool CPLX>
__device__ __forceinline__ void interp_brick_body(int brick, const int *__restrict__ brick_start,
                                                  const BrickPoint<T> *__restrict__ bp,
                                                  const T *__restrict__ theta,
                                                  double *__restrict__ V, int nb2, int nb3,
                                                  long N1, long N2, long N3, T c1, T c2, T c3,
                                                  T *tile, void *vsrc = nullptr, double vs = 1.0,
                                                  double gs = 1.0) {
  constexpr int TL = kBrick + P - 1;
  constexpr int TV = TL * TL * TL;
  constexpr int C = CPLX ? 2 : 1;
  const int b3 = brick % nb3, b2 = (brick / nb3) % nb2, b1 = brick / (nb3 * nb2);
  const long g1 = (long)b1 * kBrick, g2 = (long)b2 * kBrick, g3 = (long)b3 * kBrick;
  for (int t = threadIdx.x; t < TV; t += blockDim.x) {
    const int i3 = t % TL, i2 = (t / TL) % TL, i1 = t / (TL * TL);
    T vr = T(0), vi = T(0);
    if (g1 + i1 < N1 && g2 + i2 < N2 && g3 + i3 < N3) {
      const long gi = ((g1 + i1) * N2 + (g2 + i2)) * N3 + (g3 + i3);
      vr = theta[C * gi];
      if (CPLX) vi = theta[C * gi + 1];
    }
    tile[C * t] = vr;
    if (CPLX) tile[C * t + 1] = vi;
  }
  __syncthreads();
  const int beg = brick_start[brick], nbp = brick_start[brick + 1] - beg;
  const int nvw = (nbp + 31) >> 5, lane = threadIdx.x & 31;
  for (int vw = threadIdx.x >> 5; vw < nvw; vw += blockDim.x >> 5) {
    const int pi = brick_point(nbp, vw, lane);
    if (pi < 0) continue;
    const BrickPoint<T> pt = bp[beg + pi];
    T w1[P], w2[P], w3[P], d1[P], d2[P], d3[P];
    bspline_weights<T, P, true>(pt.u[0], w1, d1);
    bspline_weights<T, P, true>(pt.u[1], w2, d2);
    bspline_weights<T, P, true>(pt.u[2], w3, d3);
    const int l1 = (int)(pt.g0 >> 20) - b1 * kBrick;
    const int l2 = (int)((pt.g0 >> 10) & 1023u) - b2 * kBrick;
    const int l3 = (int)(pt.g0 & 1023u) - b3 * kBrick;
    T v[4] = {0, 0, 0, 0}, vi[4] = {0, 0, 0, 0};
#pragma unroll(kStencilUnroll<P>)
    for (int t1 = 0; t1 < P; t1++) {
#pragma unroll
      for (int t2 = 0; t2 < P; t2++) {
        const T *row = tile + C * (((l1 + t1) * TL + (l2 + t2)) * TL + l3);
        T tb = 0, td = 0, tbi = 0, tdi = 0;
#pragma unroll
        for (int t3 = 0; t3 < P; t3++) {
          const T th = row[C * t3];
          tb = fma(th, w3[t3], tb);
          td = fma(th, d3[t3], td);
          if (CPLX) {
            const T thi = row[C * t3 + 1];
            tbi = fma(thi, w3[t3], tbi);
            tdi = fma(thi, d3[t3], tdi);
          }
        }
        const T A1 = w1[t1] * w2[t2], A2 = d1[t1] * w2[t2], A3 = w1[t1] * d2[t2];
        v[0] = fma(A1, tb, v[0]);
        v[1] = fma(A2, tb, v[1]);
        v[2] = fma(A3, tb, v[2]);
        v[3] = fma(A1, td, v[3]);
        if (CPLX) {
          vi[0] = fma(A1, tbi, vi[0]);
          vi[1] = fma(A2, tbi, vi[1]);
          vi[2] = fma(A3, tbi, vi[2]);
          vi[3] = fma(A1, tdi, vi[3]);
        }
      }
    }
    const T sc[4] = {T(1), c1, c2, c3};
    const long o = pt.orig, slot = beg + pi;
    if (CPLX) {
      // source-side slot: (V re, V im, x re, x im), (y .., z ..)
      double d[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (vsrc) {
        using V4 = typename Vec4<T>::type;
        V4 *vp = reinterpret_cast<V4 *>(vsrc) + 2 * slot;
        const V4 a = vp[0], b = vp[1];
        V4 z;
        z.x = z.y = z.z = z.w = T(0);
        vp[0] = vp[1] = z;
        d[0] = a.x, d[1] = a.y, d[2] = a.z, d[3] = a.w;
        d[4] = b.x, d[5] = b.y, d[6] = b.z, d[7] = b.w;
      }
      double2 *Vo = reinterpret_cast<double2 *>(V) + 4 * o;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        double2 a = Vo[m];
        a.x += (double)(v[m] * sc[m]) + d[2 * m];
        a.y += (double)(vi[m] * sc[m]) + d[2 * m + 1];
        Vo[m] = a;
      }
    } else {
      double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
      if (vsrc) {
        if (sizeof(T) == 4) {  // FP32: float4 per slot, scaled frame
          float4 *vp = reinterpret_cast<float4 *>(vsrc) + slot;
          const float4 a = *vp;
          *vp = make_float4(0.f, 0.f, 0.f, 0.f);
          s0 = vs * (double)a.x, s1 = gs * (double)a.y, s2 = gs * (double)a.z,
          s3 = gs * (double)a.w;
        } else {  // FP64: [4] doubles per slot
          double4 *vp = reinterpret_cast<double4 *>(vsrc) + slot;
          const double4 a = *vp;
          *vp = make_double4(0, 0, 0, 0);
          s0 = vs * a.x, s1 = gs * a.y, s2 = gs * a.z, s3 = gs * a.w;
        }
      }
      double4 *Vo = reinterpret_cast<double4 *>(V) + o;
      double4 a = *Vo;
      a.x += (double)v[0] + s0;
      a.y += (double)(v[1] * c1) + s1;
      a.z += (double)(v[2] * c2) + s2;
      a.w += (double)(v[3] * c3) + s3;
      *Vo = a;
    }
  }
}

// kPackedBlock consecutive source-pair steps of the packed direct sum: the
// differences and distances of all steps first, then the refinement of close
// pairs (rare, a divergent branch), then the pair kernel of all steps without
// branches, so that the scheduler can interleave the independent polynomial
// chains of the block.  Pairs outside the cutoff (and the target itself) get
// r^2 = Rdir^2 and charge 0.  The whole pair phase is skipped when no lane
// of the warp has a hit in the block.
#ifndef NPME_PACKED_BLOCK
#define NPME_PACKED_BLOCK 2
#endif
constexpr int kPackedBlock = NPME_PACKED_BLOCK;

// Real DM pair kernel in the scaled frame (coordinates in units of Rdir,
// s = r^2 <= 1) for two squared distances at once: f0 = scaled f_SR = s^a - P
// and t = (scaled f1) / alpha, a = alpha / 2, from the Taylor form of the
// derivative match in u = 1 - s (PairCoef; src/KernelFunctionLaplace.cpp:394-436,
// src/KernelFunctionRalpha.cpp:342-384).
// ND > 0: the derivative-match order as a compile-time constant and alpha < 0:
// P by Horner, t = (f0 + K u^ND) / s, which needs no second polynomial (1/r,
// order 6: 6 multiply-adds for t against 7; order 8: 6 against 9) and has no
// cancellation, both terms being positive.  ND = 0: any order up to
// kMaxDeriv and any alpha (for alpha >= 0 the two terms of that t cancel at
// small s), both polynomials evaluated at degree kMaxDeriv with zero
// coefficients above the order, so that every coefficient sits at a fixed
// offset of the parameter bank (a loop over a run-time degree indexes it
// dynamically and is ~2x slower still).
// At s = 1 the result is exactly zero in f0 and t: a miss is a pair with its
// s clamped to 1.
// FUNC 2: the original Ewald split, f0 = erfc(b sqrt(s))/sqrt(s) with b = beta
// Rdir (src/PotentialLaplace.cpp:614-719), about 20 operations like the DM
// kernel; erfcf and expf take about twice that.
template <int ND>
constexpr int dm_degree() {
  return ND > 0 ? ND : kMaxDeriv;
}

// 1/x and 2^x by the special-function unit (1 and 2 ulp)
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool FTZ>
__device__ __forceinline__ float2 rsqrt2(float2 s) {
  if (!FTZ) return make_float2(rsqrtf(s.x), rsqrtf(s.y));
  float2 r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(s.x));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(s.y));
  return r;
}

// u^N, N > 0 known at compile time
template <int N>
__device__ __forceinline__ float2 pow2_n(float2 u) {
  if constexpr (N == 1) {
    return u;
  } else {
    const float2 h = pow2_n<N / 2>(u), h2 = __fmul2_rn(h, h);
    if constexpr (N % 2) return __fmul2_rn(h2, u);
    else return h2;
  }
}

// FTZ: s is a normal number (no pair of a sweep is close), so the
// special-function unit's rsqrt is taken as it is; rsqrtf adds four
// instructions per value for subnormal arguments.
template <int FUNC, int ND, bool FTZ = false>
__device__ __forceinline__ void dm_eval2(const PairCoef<float> &k, float2 s, float2 &f0,
                                         float2 &t) {
  constexpr int nd = dm_degree<ND>();
  const float2 one = make_float2(1.f, 1.f), mone = make_float2(-1.f, -1.f);
  if constexpr (FUNC == 2) {  // original Ewald split: not zero at s = 1
    // erfc(x) = exp(-x^2) erfcx(x), x = beta r; erfcx a polynomial in v = x / (x
    // + 2) (kErfcxFit), so that the exponential serves f0 and t
    const float2 ri = rsqrt2<FTZ>(s);
    const float2 x = __fmul2_rn(__fmul2_rn(s, k.nq2[0]), ri);
    const float2 d = __fadd2_rn(x, make_float2(2.f, 2.f));
    const float2 v = __fmul2_rn(x, make_float2(rcp_approx(d.x), rcp_approx(d.y)));
    float2 h = k.nc2[9];
#pragma unroll
    for (int n = 8; n >= 0; n--) h = __ffma2_rn(h, v, k.nc2[n]);
    const float2 a = __fmul2_rn(s, k.nq2[1]);
    const float2 e = make_float2(ex2_approx(a.x), ex2_approx(a.y));
    f0 = __fmul2_rn(__fmul2_rn(__ffma2_rn(h, v, one), e), ri);
    t = __fmul2_rn(__ffma2_rn(e, k.kn2, f0), __fmul2_rn(ri, ri));
    return;
  }
  const float2 u = __ffma2_rn(s, mone, one);
  float2 h = k.nc2[nd];
#pragma unroll
  for (int n = nd - 1; n >= 1; n--) h = __ffma2_rn(h, u, k.nc2[n]);
  const float2 ri = rsqrt2<FTZ>(s);
  // 1/r: s^a = rsqrt(s); r^alpha: 2^(a log2 s) on the special-function unit
  float2 e0 = ri;
  if (FUNC == 1)
    e0 = FTZ ? make_float2(ex2_approx(k.half_alpha * __log2f(s.x)),
                           ex2_approx(k.half_alpha * __log2f(s.y)))
             : make_float2(exp2f(k.half_alpha * __log2f(s.x)),
                           exp2f(k.half_alpha * __log2f(s.y)));
  f0 = __ffma2_rn(h, u, __fadd2_rn(e0, mone));
  const float2 ri2 = __fmul2_rn(ri, ri);
  if constexpr (ND > 0) {
    t = __fmul2_rn(__ffma2_rn(pow2_n<ND>(u), k.kn2, f0), ri2);
  } else {
    float2 d = k.nq2[nd - 1];
#pragma unroll
    for (int n = nd - 2; n >= 0; n--) d = __ffma2_rn(d, u, k.nq2[n]);
    t = __ffma2_rn(e0, ri2, d);
  }
}

// The same pair kernel for one squared distance.
template <int FUNC, int ND>
__device__ __forceinline__ void dm_eval1(const PairCoef<float> &k, float s, float &f0, float &t) {
  float2 f, g;
  dm_eval2<FUNC, ND>(k, make_float2(s, s), f, g);
  f0 = f.x;
  t = g.x;
}

template <int FUNC, int ND, bool REFINE>
__device__ __forceinline__ void packed_block(
    const PairCoef<float> &k, const float4 *sp, const float4 *slo, int s0, float2 tx2,
    float2 ty2, float2 tz2, float2 tl2x, float2 tl2y, float2 tl2z, float R2, float refine2,
    float2 &P0, float2 &N1, float2 &N2, float2 &N3) {
  constexpr int U = kPackedBlock;
  // rr: r^2 of the pairs inside the cutoff, R2 for the others (and for the
  // target itself); qm: their charges, 0 for the others.  A pair is inside
  // iff 0 < r^2 <= R2, i.e. iff bits(r^2) - 1 < bits(R2) as unsigned
  // integers (r^2 >= 0).
  float2 x[U], y[U], z[U], rr[U], qm[U];
  float rmin = 3.0e38f;
  bool any = false;
  const unsigned rb = __float_as_uint(R2);
#pragma unroll
  for (int u = 0; u < U; u++) {
    const float4 A = sp[s0 + u], B = sp[16 + s0 + u];
    x[u] = __fadd2_rn(tx2, make_float2(A.x, A.y));
    y[u] = __fadd2_rn(ty2, make_float2(A.z, A.w));
    z[u] = __fadd2_rn(tz2, make_float2(B.x, B.y));
    const float2 r2 = __ffma2_rn(x[u], x[u], __ffma2_rn(y[u], y[u], __fmul2_rn(z[u], z[u])));
    const bool h0 = __float_as_uint(r2.x) - 1u < rb, h1 = __float_as_uint(r2.y) - 1u < rb;
    rr[u] = make_float2(h0 ? r2.x : R2, h1 ? r2.y : R2);
    qm[u] = make_float2(h0 ? B.z : 0.f, h1 ? B.w : 0.f);
    if (REFINE) rmin = fminf(rmin, fminf(rr[u].x, rr[u].y));
    any |= h0 | h1;
  }
  if (!__any_sync(0xffffffffu, any)) return;
  if (REFINE && rmin < refine2) {  // close pair: exact difference from head + residual
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (fminf(rr[u].x, rr[u].y) < refine2) {
        const float4 LA = slo[s0 + u], LB = slo[16 + s0 + u];
        x[u] = __fadd2_rn(x[u], __fadd2_rn(tl2x, make_float2(LA.x, LA.y)));
        y[u] = __fadd2_rn(y[u], __fadd2_rn(tl2y, make_float2(LA.z, LA.w)));
        z[u] = __fadd2_rn(z[u], __fadd2_rn(tl2z, make_float2(LB.x, LB.y)));
        const float2 rn = __ffma2_rn(x[u], x[u], __ffma2_rn(y[u], y[u], __fmul2_rn(z[u], z[u])));
        // the hit decision stays that of the unrefined distance
        rr[u].x = rr[u].x < R2 ? rn.x : rr[u].x;
        rr[u].y = rr[u].y < R2 ? rn.y : rr[u].y;
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    float2 f0, t;  // t = -f1
    dm_eval2<FUNC, ND>(k, rr[u], f0, t);
    const float2 gq = __fmul2_rn(t, qm[u]);
    P0 = __ffma2_rn(f0, qm[u], P0);
    N1 = __ffma2_rn(gq, x[u], N1);
    N2 = __ffma2_rn(gq, y[u], N2);
    N3 = __ffma2_rn(gq, z[u], N3);
  }
}

// Position of a lane in the virtual concatenation of a group's source
// segments (segment index and offset in it), so that a staged chunk of 32
// sources runs across segment boundaries.
struct SrcCursor {
  int seg, off;
  __device__ __forceinline__ void normalize(const int2 *__restrict__ segs, int end) {
    while (seg < end) {
      const int c = segs[seg].y;
      if (off < c) break;
      off -= c;
      seg++;
    }
  }
};

// A lane's K positions (lane, lane + 32, ...) in the chunks of 32 K sources of a
// group's half-shell segments, zone by zone (both halves of the targets, lower,
// upper half: setup.cu); a chunk belongs to one zone.  Of nsplit warps that
// share the group, warp `part` takes every nsplit-th chunk of a zone.  ZONED =
// false: the zones are one (the set-up makes them so for these kernels).
template <int K, bool ZONED = true>
struct ZoneWalk {
  const int2 *__restrict__ segs;
  int ends[3];  // of the zones' segments
  int zone, lane, first, stride;
  SrcCursor cur[K];
  bool v[K];

  __device__ __forceinline__ ZoneWalk(const int2 *__restrict__ segs_, const int4 G,
                                      const int2 zones, int lane_, int part, int nsplit)
      : segs(segs_), ends{zones.x, zones.y, G.w}, zone(0), lane(lane_),
        first(lane_ + 32 * K * part), stride(32 * K * nsplit) {
    start(G.z);
    skip();
  }
  __device__ __forceinline__ int end() const {
    return !ZONED ? ends[2] : zone == 0 ? ends[0] : zone == 1 ? ends[1] : ends[2];
  }
  __device__ __forceinline__ void start(int seg) {
    cur[0] = SrcCursor{seg, first};
    cur[0].normalize(segs, end());
    v[0] = cur[0].seg < end();
#pragma unroll
    for (int i = 1; i < K; i++) {
      cur[i] = SrcCursor{cur[i - 1].seg, cur[i - 1].off + 32};
      cur[i].normalize(segs, end());
      v[i] = cur[i].seg < end();
    }
  }
  // on to the zone that has a chunk left (the valid lanes are a prefix)
  __device__ __forceinline__ void skip() {
    if (!ZONED) return;
    while (zone < 2 && !__any_sync(0xffffffffu, v[0])) {
      const int seg = end();
      zone++;
      start(seg);
    }
  }
  __device__ __forceinline__ bool any() const { return __any_sync(0xffffffffu, v[0]); }
  __device__ __forceinline__ void next() {
#pragma unroll
    for (int i = 0; i < K; i++) {
      cur[i].off += stride;
      cur[i].normalize(segs, end());
      v[i] = cur[i].seg < end();
    }
    skip();
  }
  __device__ __forceinline__ long index(int i) const {
    return (long)segs[cur[i].seg].x + cur[i].off;
  }
};

// Real derivative-match kernels (1/r, r^alpha) of the FP32 direct sum with
// packed arithmetic: every lane evaluates its target against two sources per
// step with sm_100's two-wide FP32 instructions (__fadd2_rn / __fmul2_rn /
// __ffma2_rn), which halves the issued arithmetic of the distance test and
// of the polynomial.  The staged chunk is laid out in source pairs:
//   sp[p]      = (-x_2p, -x_2p+1, -y_2p, -y_2p+1)
//   sp[16 + p] = (-z_2p, -z_2p+1,  q_2p,  q_2p+1)
// (coordinates negated so that t + (-s) gives t - s exactly), slo the same
// for the low parts of the rounded differences.  Slots past the chunk hold a
// far source with charge 0.  Same arithmetic per pair as the scalar body
// (difference, r^2, hit test, refinement below refine2, polynomial in
// s = r^2/Rdir^2), except that a refined step refines both of its pairs.
template <int FUNC, int ND>
__device__ __forceinline__ void direct_group_packed(
    const PairCoef<float> &k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller, const int4 G,
    const double4 c, const int2 *__restrict__ segs, const uint32_t *__restrict__ perm,
    float refine2, double fself_r, double *__restrict__ V, float4 *sp, float4 *slo, int lane) {
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  // idle lanes sit far outside the cutoff
  float tx = 1e18f, ty = 1e18f, tz = 1e18f, tlx = 0.f, tly = 0.f, tlz = 0.f;
  const double ir = k.invR;  // coordinates in units of Rdir
  if (active) {
    const double4 p = gpos[ti];
    const double dx = (p.x - c.x) * ir, dy = (p.y - c.y) * ir, dz = (p.z - c.z) * ir;
    tx = (float)dx, ty = (float)dy, tz = (float)dz;
    tlx = (float)(dx - (double)tx), tly = (float)(dy - (double)ty), tlz = (float)(dz - (double)tz);
  }
  const float2 tx2 = make_float2(tx, tx), ty2 = make_float2(ty, ty), tz2 = make_float2(tz, tz);
  const float2 tl2x = make_float2(tlx, tlx), tl2y = make_float2(tly, tly),
               tl2z = make_float2(tlz, tlz);
  const float R2 = 1.f;
  refine2 = (float)((double)refine2 * ir * ir);
  double acc[4] = {0, 0, 0, 0};
  float *sa = reinterpret_cast<float *>(sp), *la = reinterpret_cast<float *>(slo);
  const int slot = (lane >> 1) * 4 + (lane & 1);

  // A pair closer than sqrt(refine2) needs its source within the group's
  // half-diagonal (c.w) plus sqrt(refine2) of the centre; chunks with no
  // such source skip the refinement bookkeeping.
  const double rfs = sqrt((double)refine2) + c.w * ir;
  const double near2 = rfs * rfs;
  bool near = false;
  // register prefetch of the next chunk: lane l holds source l of the chunk
  SrcCursor cur{G.z, lane};
  cur.normalize(segs, G.w);
  bool pv = cur.seg < G.w;
  double px = 0, py = 0, pz = 0;
  float pq = 0.f;
  if (pv) {
    const long j = (long)segs[cur.seg].x + cur.off;
    const double4 p = spos[j];
    px = p.x, py = p.y, pz = p.z, pq = qs[j];
  }
  while (__any_sync(0xffffffffu, pv)) {
    const int pcnt = __popc(__ballot_sync(0xffffffffu, pv));  // valid lanes form a prefix
    __syncwarp();
    {
      float hx = 1e18f, hy = 1e18f, hz = 1e18f, q = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
      near = false;
      if (pv) {
        const double dx = (px - c.x) * ir, dy = (py - c.y) * ir, dz = (pz - c.z) * ir;
        hx = (float)dx, hy = (float)dy, hz = (float)dz;
        lx = (float)(dx - (double)hx), ly = (float)(dy - (double)hy), lz = (float)(dz - (double)hz);
        q = pq;
        near = dx * dx + dy * dy + dz * dz < near2;
      }
      sa[slot] = -hx;
      sa[slot + 2] = -hy;
      sa[64 + slot] = -hz;
      sa[64 + slot + 2] = q;
      la[slot] = -lx;
      la[slot + 2] = -ly;
      la[64 + slot] = -lz;
    }
    __syncwarp();
    cur.off += 32;
    cur.normalize(segs, G.w);
    pv = cur.seg < G.w;
    if (pv) {
      const long j = (long)segs[cur.seg].x + cur.off;
      const double4 p = spos[j];
      px = p.x, py = p.y, pz = p.z, pq = qs[j];
    }
    const int npair = (pcnt + 1) >> 1;
    float2 P0 = make_float2(0.f, 0.f), N1 = P0, N2 = P0, N3 = P0;  // N*: minus the gradient
    // blocks of kPackedBlock steps; slots past the chunk hold far sources, so
    // the step count is rounded up to whole blocks
    if (__any_sync(0xffffffffu, near)) {
      for (int s0 = 0; s0 < npair; s0 += kPackedBlock)
        packed_block<FUNC, ND, true>(k, sp, slo, s0, tx2, ty2, tz2, tl2x, tl2y, tl2z, R2, refine2,
                                     P0, N1, N2, N3);
    } else {
      for (int s0 = 0; s0 < npair; s0 += kPackedBlock)
        packed_block<FUNC, ND, false>(k, sp, slo, s0, tx2, ty2, tz2, tl2x, tl2y, tl2z, R2,
                                      refine2, P0, N1, N2, N3);
    }
    acc[0] += (double)P0.x + (double)P0.y;
    acc[1] -= (double)N1.x + (double)N1.y;
    acc[2] -= (double)N2.x + (double)N2.y;
    acc[3] -= (double)N3.x + (double)N3.y;
  }
  if (active) {
    const long o = perm[ti];
    const double vs = k.vscale, gs = k.gscale;
    // V -= f_LR(0) q (src/Interface.cpp:2061-2062)
    reinterpret_cast<double4 *>(V)[o] =
        make_double4(vs * acc[0] - fself_r * qcaller[o], gs * acc[1], gs * acc[2], gs * acc[3]);
  }
}

// The two sources of a lane in the pair-once sweep: coordinates relative to
// the group centre, negated (so that t + (-s) gives t - s exactly), each as the
// pair (v, v) that meets two targets at once.
struct SymSource {
  float2 x, y, z, q;
};
// Sources per lane.  One (80 registers, 24 resident warps per SM instead of 16)
// was slower, 3,293-3,377 us against 3,094 for 1/r at 1M: twice the shuffles and
// shared loads per pair, and latency is not what bounds the sweep.
constexpr int kSymSources = 2;

// What a warp of the pair-once sweep keeps in shared memory: the group's targets
// in pairs (t[j] = x0 x1 y0 y1, t[16 + j] = z0 z1 q0 q1), the residuals of
// their coordinates and, for the chunks that need them, of the sources' (negated,
// as the coordinates), the target sums across chunks, and the group's centre
// with near2 (below).  The last three would take 20 registers that are used once
// per chunk.
struct SymWarp {
  float4 t[32], lo[32];
  float res[kSymSources][3][32];
  double acc[4][32];
  double4 c;
};

// One step of the Newton's-third-law sweep (below): the lane's two sources
// against one pair of targets (A = x0 x1 y0 y1, B = z0 z1 q0 q1; LA, LB the
// residuals), four pairs, every one evaluated once for both of its points:
// target sums aV.. (packed over the two targets) and source sums S[i].
// CHECKED = false: no pair of the chunk is closer than the refinement radius
// and all charges are finite, so a miss needs nothing but s clamped to 1,
// where the pair kernel is exactly zero.  CHECKED = true: close pairs are
// recomputed from heads and residuals, coincident points are no pair, and
// misses also get charge 0 (a non-finite charge stays out of their sums).
template <int FUNC, int ND, bool CHECKED>
__device__ __forceinline__ void sym_step(const PairCoef<float> &k, const SymWarp &W, int j,
                                         int lane, const SymSource (&src)[kSymSources],
                                         float refine2, float2 &aV, float2 &aX, float2 &aY,
                                         float2 &aZ, float2 (&S)[kSymSources][4]) {
  const float4 A = W.t[j], B = W.t[16 + j];
  float2 x[kSymSources], y[kSymSources], z[kSymSources], s[kSymSources], qs[kSymSources],
      qt[kSymSources];
#pragma unroll
  for (int i = 0; i < kSymSources; i++) {
    x[i] = __fadd2_rn(make_float2(A.x, A.y), src[i].x);
    y[i] = __fadd2_rn(make_float2(A.z, A.w), src[i].y);
    z[i] = __fadd2_rn(make_float2(B.x, B.y), src[i].z);
    float2 r2 = __ffma2_rn(x[i], x[i], __ffma2_rn(y[i], y[i], __fmul2_rn(z[i], z[i])));
    qs[i] = src[i].q;
    qt[i] = make_float2(B.z, B.w);
    if (CHECKED) {
      if (fminf(r2.x, r2.y) < refine2) {  // exact differences from head + residual
        const float4 LA = W.lo[j], LB = W.lo[16 + j];
        const float lx = W.res[i][0][lane], ly = W.res[i][1][lane], lz = W.res[i][2][lane];
        x[i] = __fadd2_rn(x[i], __fadd2_rn(make_float2(LA.x, LA.y), make_float2(lx, lx)));
        y[i] = __fadd2_rn(y[i], __fadd2_rn(make_float2(LA.z, LA.w), make_float2(ly, ly)));
        z[i] = __fadd2_rn(z[i], __fadd2_rn(make_float2(LB.x, LB.y), make_float2(lz, lz)));
        r2 = __ffma2_rn(x[i], x[i], __ffma2_rn(y[i], y[i], __fmul2_rn(z[i], z[i])));
      }
      // a pair is inside iff 0 < r^2 <= 1, i.e. bits(r^2) - 1 < bits(1) as
      // unsigned integers (r^2 >= 0)
      const unsigned one = __float_as_uint(1.f);
      const bool h0 = __float_as_uint(r2.x) - 1u < one, h1 = __float_as_uint(r2.y) - 1u < one;
      s[i] = make_float2(h0 ? r2.x : 1.f, h1 ? r2.y : 1.f);
      qs[i] = make_float2(h0 ? qs[i].x : 0.f, h1 ? qs[i].y : 0.f);
      qt[i] = make_float2(h0 ? qt[i].x : 0.f, h1 ? qt[i].y : 0.f);
    } else {
      s[i] = make_float2(fminf(r2.x, 1.f), fminf(r2.y, 1.f));
      if (FUNC == 2) {  // the Ewald kernel is not zero at Rdir: misses get charge 0
        const bool h0 = r2.x <= 1.f, h1 = r2.y <= 1.f;
        qs[i] = make_float2(h0 ? qs[i].x : 0.f, h1 ? qs[i].y : 0.f);
        qt[i] = make_float2(h0 ? qt[i].x : 0.f, h1 ? qt[i].y : 0.f);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kSymSources; i++) {
    float2 f0, t;  // t = -f1
    dm_eval2<FUNC, ND, !CHECKED>(k, s[i], f0, t);
    const float2 gs = __fmul2_rn(t, qs[i]), gt = __fmul2_rn(t, qt[i]);
    aV = __ffma2_rn(f0, qs[i], aV);
    aX = __ffma2_rn(gs, x[i], aX);
    aY = __ffma2_rn(gs, y[i], aY);
    aZ = __ffma2_rn(gs, z[i], aZ);
    S[i][0] = __ffma2_rn(f0, qt[i], S[i][0]);
    S[i][1] = __ffma2_rn(gt, x[i], S[i][1]);
    S[i][2] = __ffma2_rn(gt, y[i], S[i][2]);
    S[i][3] = __ffma2_rn(gt, z[i], S[i][3]);
  }
}

// v of lane (lane + 1) mod 32, both halves
__device__ __forceinline__ float2 rotate2(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// The steps of one chunk, 16 over all target pairs or 8 over one half of them
// (zone 1: pairs 0-7, zone 2: pairs 8-15); target sums rotate after each.
template <int FUNC, int ND, bool CHECKED>
__device__ __forceinline__ void sym_sweep(const PairCoef<float> &k, const SymWarp &W,
                                          const SymSource (&src)[kSymSources], float refine2,
                                          int lane, int zone, float2 &aV,
                                          float2 &aX, float2 &aY, float2 &aZ,
                                          float2 (&S)[kSymSources][4]) {
  constexpr int kUnroll = CHECKED ? 1 : 8;
  const int next = (lane + 1) & 31;
  const int mask = zone == 0 ? 15 : 7, from = zone == 2 ? 8 : 0;
#pragma unroll 1
  for (int k0 = 0; k0 <= mask; k0 += 8) {
#pragma unroll kUnroll
    for (int kk = 0; kk < 8; kk++) {
      const int j = from + ((lane + k0 + kk) & mask);
      sym_step<FUNC, ND, CHECKED>(k, W, j, lane, src, refine2, aV, aX, aY, aZ, S);
      aV = rotate2(aV, next), aX = rotate2(aX, next);
      aY = rotate2(aY, next), aZ = rotate2(aZ, next);
    }
  }
}

// Real derivative-match kernels (1/r, r^alpha) and the original Ewald split of
// the FP32 direct sum with every unordered pair evaluated once (Newton's third law, as the
// reference's own cell-pair loops do: src/PotentialLaplace.cpp:145-197,
// :3447-3610).  The group walks its half-shell source segments: sources
// whose point lies in a later coarse column, or later in the group's own
// column, than the group's targets (set-up, setup.cu); the pairs inside the
// group are the first phase, from both sides with target-side sums only.
// The group's targets sit in shared memory as 16 pairs; a lane holds two
// sources of a 64-source chunk in registers and meets target pair (lane + k)
// mod 16 at step k, four pairs of points per step in packed FP32.  The
// target sums of a pair travel with it, one lane down per step; after 16
// steps lanes l and l + 16 hold the two halves of the sums of pair l mod 16,
// and lane l keeps target 2 (l mod 16) + l / 16.  Packing over targets (the
// former sweep packed the lane's two sources) leaves no scalar arithmetic in
// the target sums, makes the operands of every packed instruction register
// pairs as loaded, and reads two lanes' targets with one shared wavefront.
// Target-side sums accumulate per chunk in FP32 and across chunks in FP64,
// as in the one-sided body; the source-side sums of a chunk are added to
// vsrc (FP32, scaled frame; slot = the source's brick-order position, from
// spos[j].w) with one vector atomic per source, and folded into V by the
// interpolation (CalcV) or by merge_source_kernel.
// r^alpha: sources that only one half of the targets (16 in z order) can reach
// are met by that half alone, in half the steps.
// The group's work is shared by nsplit warps of the CTA, warp `part` taking
// chunks part, part + nsplit, ... (and every nsplit-th source of the pairs
// inside the group); the caller adds their sums (sym_store).
template <int FUNC, int ND>
__device__ __forceinline__ void direct_group_sym(
    const PairCoef<float> &k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller, const int4 G,
    const double4 c, const int2 *__restrict__ segs, const int2 zones,
    const uint32_t *__restrict__ perm, float refine2, float4 *__restrict__ vsrc, SymWarp &W,
    int lane, int part, int nsplit) {
  const unsigned FULL = 0xffffffffu;
  const int tid = 2 * (lane & 15) + (lane >> 4);  // the lane's target in the group
  // absent targets sit far outside the cutoff with charge 0
  float tx = 1e18f, ty = 1e18f, tz = 1e18f, tlx = 0.f, tly = 0.f, tlz = 0.f, tq = 0.f;
  const double ir = k.invR;  // coordinates in units of Rdir
  if (tid < G.y) {
    const double4 p = gpos[G.x + tid];
    const double dx = (p.x - c.x) * ir, dy = (p.y - c.y) * ir, dz = (p.z - c.z) * ir;
    tx = (float)dx, ty = (float)dy, tz = (float)dz;
    tlx = (float)(dx - (double)tx), tly = (float)(dy - (double)ty), tlz = (float)(dz - (double)tz);
    tq = (float)qcaller[perm[G.x + tid]];
  }
  refine2 = (float)((double)refine2 * ir * ir);
  {
    float *ts = reinterpret_cast<float *>(W.t), *tl = reinterpret_cast<float *>(W.lo);
    const int at = 4 * (lane & 15) + (lane >> 4);
    ts[at] = tx, ts[at + 2] = ty, ts[at + 64] = tz, ts[at + 66] = tq;
    tl[at] = tlx, tl[at + 2] = tly, tl[at + 64] = tlz, tl[at + 66] = 0.f;
  }
  if (lane == 0) {
    // a chunk with a source nearer to the centre than this takes the checked steps
    const double rfs = sqrt((double)refine2) + c.w * ir;
    W.c = make_double4(c.x, c.y, c.z, rfs * rfs);
  }
  __syncwarp();
  // a non-finite charge in the group: every chunk takes the checked steps
  const bool odd_group = __any_sync(FULL, !(fabsf(tq) <= 3.402823466e38f));

  // pairs inside the group, from both sides; the differences are always
  // refined (head difference + residual difference)
  {
    const float *ts = reinterpret_cast<const float *>(W.t),
                *tl = reinterpret_cast<const float *>(W.lo);
    const unsigned rb = __float_as_uint(1.f);
    float aV = 0.f, aX = 0.f, aY = 0.f, aZ = 0.f;
    for (int s = part; s < G.y; s += nsplit) {
      const int at = 4 * (s >> 1) + (s & 1);
      const float x = (tx - ts[at]) + (tlx - tl[at]), y = (ty - ts[at + 2]) + (tly - tl[at + 2]),
                  z = (tz - ts[at + 64]) + (tlz - tl[at + 64]);
      const float r2 = fmaf(x, x, fmaf(y, y, z * z));
      const bool hit = __float_as_uint(r2) - 1u < rb;  // 0 < r^2 <= 1, not the target itself
      float f0, t;
      dm_eval1<FUNC, ND>(k, hit ? r2 : 1.f, f0, t);
      const float q = hit ? ts[at + 66] : 0.f, g = t * q;
      aV = fmaf(f0, q, aV);
      aX = fmaf(g, x, aX);
      aY = fmaf(g, y, aY);
      aZ = fmaf(g, z, aZ);
    }
    W.acc[0][lane] = (double)aV;
    W.acc[1][lane] = -(double)aX;
    W.acc[2][lane] = -(double)aY;
    W.acc[3][lane] = -(double)aZ;
  }

  // half-shell segments in chunks of 64 sources: lane l holds positions l
  // and l + 32 of the chunk (register prefetch of the next chunk)
  constexpr bool kZoned = FUNC == 1;  // measured: set-up (describe)
  ZoneWalk<kSymSources, kZoned> walk(segs, G, zones, lane, part, nsplit);
  double4 p[kSymSources];
  float q[kSymSources];
#pragma unroll
  for (int i = 0; i < kSymSources; i++) {
    p[i] = make_double4(0, 0, 0, 0);
    q[i] = 0.f;
    if (walk.v[i]) {
      const long j = walk.index(i);
      p[i] = spos[j], q[i] = qs[j];
    }
  }
  while (walk.any()) {
    // this chunk's sources, relative to the group centre; empty slots far
    // away (on the other side from absent targets) with charge 0
    SymSource src[kSymSources];
    int slot[kSymSources];  // source-side slots: the sources' brick-order positions
    bool checked = odd_group;
    const int zone = kZoned ? walk.zone : 0;
    {
      const double4 o = W.c;
      double d[kSymSources][3];
#pragma unroll
      for (int i = 0; i < kSymSources; i++) {
        float hx = -1e18f, hy = -1e18f, hz = -1e18f, qv = 0.f;
        slot[i] = -1;
        d[i][0] = d[i][1] = d[i][2] = -1e18;
        if (walk.v[i]) {
          d[i][0] = (p[i].x - o.x) * ir, d[i][1] = (p[i].y - o.y) * ir;
          d[i][2] = (p[i].z - o.z) * ir;
          hx = (float)d[i][0], hy = (float)d[i][1], hz = (float)d[i][2];
          qv = q[i];
          slot[i] = (int)p[i].w;
          checked = checked ||
                    d[i][0] * d[i][0] + d[i][1] * d[i][1] + d[i][2] * d[i][2] < o.w ||
                    !(fabsf(qv) <= 3.402823466e38f);
        }
        src[i].x = make_float2(-hx, -hx), src[i].y = make_float2(-hy, -hy);
        src[i].z = make_float2(-hz, -hz), src[i].q = make_float2(qv, qv);
      }
      checked = __any_sync(FULL, checked);
      if (checked) {
#pragma unroll
        for (int i = 0; i < kSymSources; i++) {
          W.res[i][0][lane] = -(float)(d[i][0] + (double)src[i].x.x);
          W.res[i][1][lane] = -(float)(d[i][1] + (double)src[i].y.x);
          W.res[i][2][lane] = -(float)(d[i][2] + (double)src[i].z.x);
        }
      }
    }
    // prefetch the next chunk
    walk.next();
#pragma unroll
    for (int i = 0; i < kSymSources; i++)
      if (walk.v[i]) {
        const long j = walk.index(i);
        p[i] = spos[j], q[i] = qs[j];
      }
    float2 aV = make_float2(0.f, 0.f), aX = aV, aY = aV, aZ = aV;
    float2 S[kSymSources][4];
#pragma unroll
    for (int i = 0; i < kSymSources; i++)
      S[i][0] = S[i][1] = S[i][2] = S[i][3] = make_float2(0.f, 0.f);
    if (checked)
      sym_sweep<FUNC, ND, true>(k, W, src, refine2, lane, zone, aV, aX, aY, aZ, S);
    else
      sym_sweep<FUNC, ND, false>(k, W, src, refine2, lane, zone, aV, aX, aY, aZ, S);
    // lanes l and l + 16 hold half of the sums of target pair l mod 16 each;
    // after a sweep over one half of the pairs lanes l, l + 8, l + 16 and l + 24
    // hold a quarter each of pair l mod 8 of that half
    const bool hi = lane >= 16, other_half = zone != 0 && (lane >> 3 & 1) != zone - 1;
    auto total = [&](float2 a) {
      if (zone != 0) {
        a.x += __shfl_xor_sync(FULL, a.x, 8);
        a.y += __shfl_xor_sync(FULL, a.y, 8);
      }
      const float give = hi ? a.x : a.y, keep = hi ? a.y : a.x;
      const float sum = keep + __shfl_xor_sync(FULL, give, 16);
      return other_half ? 0.f : sum;
    };
    W.acc[0][lane] += (double)total(aV);
    W.acc[1][lane] -= (double)total(aX);
    W.acc[2][lane] -= (double)total(aY);
    W.acc[3][lane] -= (double)total(aZ);
#pragma unroll
    for (int i = 0; i < kSymSources; i++)
      if (slot[i] >= 0)
        atomicAdd(vsrc + slot[i], make_float4(S[i][0].x + S[i][0].y, S[i][1].x + S[i][1].y,
                                              S[i][2].x + S[i][2].y, S[i][3].x + S[i][3].y));
  }
}

// Sum over the nsplit warps of a CTA that share one group: acc of every part
// into that of part 0 (same lane, same target).  red: [nsplit][32][4].
__device__ __forceinline__ void reduce_parts(double (&acc)[4], double (*red)[32][4], int part,
                                             int nsplit, int lane) {
  if (part > 0)
#pragma unroll
    for (int m = 0; m < 4; m++) red[part][lane][m] = acc[m];
  __syncthreads();
  if (part == 0)
    for (int w = 1; w < nsplit; w++)
#pragma unroll
      for (int m = 0; m < 4; m++) acc[m] += red[w][lane][m];
}

// The target sums of direct_group_sym (of nsplit warps) to V, less the self term
// f_LR(0) q (src/Interface.cpp:2061-2062).
__device__ __forceinline__ void sym_store(const PairCoef<float> &k, const int4 G,
                                          const uint32_t *__restrict__ perm,
                                          const double *__restrict__ qcaller, double fself_r,
                                          double *__restrict__ V, int lane, const SymWarp *W,
                                          int nsplit) {
  const int tid = 2 * (lane & 15) + (lane >> 4);
  if (tid >= G.y) return;
  double acc[4];
#pragma unroll
  for (int m = 0; m < 4; m++) acc[m] = W[0].acc[m][lane];
  for (int w = 1; w < nsplit; w++)
#pragma unroll
    for (int m = 0; m < 4; m++) acc[m] += W[w].acc[m][lane];
  const long o = perm[G.x + tid];
  const double vs = k.vscale, gs = k.gscale;
  reinterpret_cast<double4 *>(V)[o] =
      make_double4(vs * acc[0] - fself_r * qcaller[o], gs * acc[1], gs * acc[2], gs * acc[3]);
}

// sin and cos of x on the special-function unit after a Cody-Waite
// reduction to [-pi, pi] (2 pi split as 6.28125 + 1.9353071795864769e-3, the
// first part exact in 8 bits so n * 6.28125 is exact for |n| < 2^16).
__device__ __forceinline__ float2 sincos_sfu(float x) {
  const float n = rintf(x * 0.15915494309189535f);
  float y = fmaf(-n, 6.28125f, x);
  y = fmaf(-n, 1.9353071795864769e-3f, y);
  return make_float2(__cosf(y), __sinf(y));
}

// Helmholtz DM pair kernel at squared distance rr (FP32, complex as float2):
// F0 = exp(i k0 r)/r - f_LR (the DM polynomial in s = rr / Rdir^2, held
// negated in nac2) and F1 = (1/r) dF0/dr, with sin / cos on the
// special-function unit (src/KernelFunctionHelmholtz.cpp:506-563).
template <int ND>
__device__ __forceinline__ void helm_eval(const PairCoef<float> &k, float rr, float2 &F0,
                                          float2 &F1) {
  const float2 ik = make_float2(-k.k0i, k.k0r);  // i k0
  const float ri = rsqrtf(rr), r = rr * ri;
  const float2 cs = sincos_sfu(k.k0r * r);
  const float damp = k.k0i != 0.f ? __expf(-k.k0i * r) * ri : ri;
  const float2 E = __fmul2_rn(cs, make_float2(damp, damp));  // exp(i k0 r) / r
  // E1 = (i k0 E - E / r) / r, the radial derivative over r
  const float2 IK = __ffma2_rn(make_float2(ik.x, ik.x), E,
                               __fmul2_rn(make_float2(-ik.y, ik.y), make_float2(E.y, E.x)));
  const float ri2 = ri * ri;
  const float2 E1 = __ffma2_rn(E, make_float2(-ri2, -ri2), __fmul2_rn(IK, make_float2(ri, ri)));
  const float sv = rr * k.invR2;
  const float2 s2 = make_float2(sv, sv);
  constexpr int nd = dm_degree<ND>();  // ND = 0: zero-padded to kMaxDeriv
  float2 P = k.nac2[nd];
#pragma unroll
  for (int n = nd - 1; n >= 0; n--) P = __ffma2_rn(P, s2, k.nac2[n]);
  float2 D = k.nbc2[nd - 1];
#pragma unroll
  for (int n = nd - 2; n >= 0; n--) D = __ffma2_rn(D, s2, k.nbc2[n]);
  F0 = __fadd2_rn(E, P);
  F1 = __fadd2_rn(E1, D);
}

// Helmholtz DM kernel exp(i k0 r)/r of the FP32 direct sum with packed
// complex arithmetic: one source per lane per step, the (re, im) parts of
// exp(i k0 r)/r, of the DM polynomials and of the charge products in
// FP32x2 instructions, sin / cos on the special-function unit.  Same staged
// chunk as the scalar body (sp: x, y, z, Re q; slo: low parts, Im q); pairs
// outside the cutoff get r^2 = Rdir^2 and charge 0, the rare close pairs
// are refined as in the scalar body.
template <int ND>
__device__ __forceinline__ void helmholtz_steps(const PairCoef<float> &k, const float4 *sp,
                                                const float4 *slo, int cnt, float tx, float ty,
                                                float tz, float tlx, float tly, float tlz,
                                                float refine2, float2 &Pv, float2 &Gx,
                                                float2 &Gy, float2 &Gz) {
  const float R2 = k.R2;
  const unsigned rb = __float_as_uint(R2);
#pragma unroll 4
  for (int s = 0; s < cnt; s++) {
    const float4 src = sp[s];
    float x = tx - src.x, y = ty - src.y, z = tz - src.z;
    float r2 = fmaf(x, x, fmaf(y, y, z * z));
    const bool hit = __float_as_uint(r2) - 1u < rb;  // 0 < r2 <= R2
    if (hit && r2 < refine2) {  // close pair: exact difference from head + residual
      const float4 lo = slo[s];
      x += tlx - lo.x;
      y += tly - lo.y;
      z += tlz - lo.z;
      r2 = fmaf(x, x, fmaf(y, y, z * z));
    }
    const float rr = hit ? r2 : R2;
    const float4 lo = slo[s];
    const float2 q = hit ? make_float2(src.w, lo.w) : make_float2(0.f, 0.f);
    float2 F0, F1;
    helm_eval<ND>(k, rr, F0, F1);
    const float2 qs = make_float2(q.y, q.x);
    // V += F0 q, G = F1 q (complex products)
    Pv = __ffma2_rn(make_float2(F0.x, F0.x), q, Pv);
    Pv = __ffma2_rn(make_float2(-F0.y, F0.y), qs, Pv);
    const float2 G = __ffma2_rn(make_float2(-F1.y, F1.y), qs,
                                __fmul2_rn(make_float2(F1.x, F1.x), q));
    Gx = __ffma2_rn(G, make_float2(x, x), Gx);
    Gy = __ffma2_rn(G, make_float2(y, y), Gy);
    Gz = __ffma2_rn(G, make_float2(z, z), Gz);
  }
}

// complex a * b + c and a * b on float2 (re, im)
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  c = __ffma2_rn(make_float2(a.x, a.x), b, c);
  return __ffma2_rn(make_float2(-a.y, a.y), make_float2(b.y, b.x), c);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return __ffma2_rn(make_float2(-a.y, a.y), make_float2(b.y, b.x),
                    __fmul2_rn(make_float2(a.x, a.x), b));
}

// Helmholtz DM kernel of the FP32 direct sum with every unordered pair
// evaluated once (the complex counterpart of direct_group_sym): the group's
// targets sit in shared memory (th = heads and Re q, tl = residuals and Im
// q), each lane holds two sources of a 64-source chunk of the half-shell
// segments, target (l + k) mod 32 meets lane l at step k and its complex sums
// (V, dV/dx, dV/dy, dV/dz) rotate one lane down per step; the source-side
// sums of a chunk go to vsrc as two float4 per source (V re, V im, x re,
// x im; y re, y im, z re, z im) with vector atomics.  Coordinates are
// unscaled offsets from the group centre, close pairs refined as in the
// one-sided body; pairs inside the group are a first, one-sided pass.
template <int ND>
__device__ __forceinline__ void direct_group_sym_helm(
    const PairCoef<float> &k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller, const int4 G,
    const double4 c, const int2 *__restrict__ segs, const int2 zones,
    const uint32_t *__restrict__ perm, float refine2, float4 *__restrict__ vsrc, float4 *th,
    float4 *tl, int lane, int part, int nsplit, double (&acc)[4], double (&acci)[4]) {
  const unsigned FULL = 0xffffffffu;
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  float tx = 1e18f, ty = 1e18f, tz = 1e18f, tlx = 0.f, tly = 0.f, tlz = 0.f;
  float2 tq = make_float2(0.f, 0.f);
  if (active) {
    const double4 p = gpos[ti];
    const long o = perm[ti];
    const double dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
    tx = (float)dx, ty = (float)dy, tz = (float)dz;
    tlx = (float)(dx - (double)tx), tly = (float)(dy - (double)ty), tlz = (float)(dz - (double)tz);
    tq = make_float2((float)qcaller[2 * o], (float)qcaller[2 * o + 1]);
  }
  th[lane] = make_float4(tx, ty, tz, tq.x);
  tl[lane] = make_float4(tlx, tly, tlz, tq.y);
  __syncwarp();
  const float R2 = k.R2;
  const unsigned rb = __float_as_uint(R2);

  // pairs inside the group, target side only, differences always refined
  {
    float2 Pv = make_float2(0.f, 0.f), Gx = Pv, Gy = Pv, Gz = Pv;
    for (int s = part; s < G.y; s += nsplit) {
      const float4 S = th[s], L = tl[s];
      const float x = (tx - S.x) + (tlx - L.x), y = (ty - S.y) + (tly - L.y),
                  z = (tz - S.z) + (tlz - L.z);
      const float r2 = fmaf(x, x, fmaf(y, y, z * z));
      if (__float_as_uint(r2) - 1u < rb) {  // 0 < r^2 <= R2
        float2 F0, F1;
        helm_eval<ND>(k, r2, F0, F1);
        const float2 q = make_float2(S.w, L.w), g = cmul(F1, q);
        Pv = cfma(F0, q, Pv);
        Gx = __ffma2_rn(g, make_float2(x, x), Gx);
        Gy = __ffma2_rn(g, make_float2(y, y), Gy);
        Gz = __ffma2_rn(g, make_float2(z, z), Gz);
      }
    }
    acc[0] += Pv.x, acci[0] += Pv.y, acc[1] += Gx.x, acci[1] += Gx.y;
    acc[2] += Gy.x, acci[2] += Gy.y, acc[3] += Gz.x, acci[3] += Gz.y;
  }

  ZoneWalk<2> walk(segs, G, zones, lane, part, nsplit);
  double4 p[2];
  float2 q[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    p[i] = make_double4(0, 0, 0, 0);
    q[i] = make_float2(0.f, 0.f);
    if (walk.v[i]) {
      const long j = walk.index(i);
      p[i] = spos[j], q[i] = make_float2(qs[2 * j], qs[2 * j + 1]);
    }
  }
  while (walk.any()) {
    const int zone = walk.zone;
    // this chunk's two sources of the lane; empty slots far away on the
    // other side from idle targets, with charge 0
    float sx[2] = {-1e18f, -1e18f}, sy[2] = {-1e18f, -1e18f}, sz[2] = {-1e18f, -1e18f};
    float lx[2] = {0.f, 0.f}, ly[2] = {0.f, 0.f}, lz[2] = {0.f, 0.f};
    float2 sq[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    int kidx[2];  // brick positions
#pragma unroll
    for (int i = 0; i < 2; i++) {
      kidx[i] = -1;
      if (walk.v[i]) {
        const double dx = p[i].x - c.x, dy = p[i].y - c.y, dz = p[i].z - c.z;
        sx[i] = (float)dx, sy[i] = (float)dy, sz[i] = (float)dz;
        lx[i] = (float)(dx - (double)sx[i]), ly[i] = (float)(dy - (double)sy[i]);
        lz[i] = (float)(dz - (double)sz[i]);
        sq[i] = q[i];
        kidx[i] = (int)p[i].w;
      }
    }
    walk.next();
#pragma unroll
    for (int i = 0; i < 2; i++)
      if (walk.v[i]) {
        const long j = walk.index(i);
        p[i] = spos[j], q[i] = make_float2(qs[2 * j], qs[2 * j + 1]);
      }

    float2 Pv = make_float2(0.f, 0.f), Gx = Pv, Gy = Pv, Gz = Pv;  // target side, rotating
    float2 SV[2], SX[2], SY[2], SZ[2];                              // source side
#pragma unroll
    for (int u = 0; u < 2; u++) SV[u] = SX[u] = SY[u] = SZ[u] = make_float2(0.f, 0.f);
    const int src = (lane + 1) & 31;
    const int mask = zone == 0 ? 31 : 15, from = zone == 2 ? 16 : 0;
    for (int kk = 0; kk <= mask; kk++) {
      const int tt = from + ((lane + kk) & mask);
      const float4 T = th[tt], L = tl[tt];
      float x[2], y[2], z[2], rr[2];
      bool hit[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        x[u] = T.x - sx[u], y[u] = T.y - sy[u], z[u] = T.z - sz[u];
        float r2 = fmaf(x[u], x[u], fmaf(y[u], y[u], z[u] * z[u]));
        hit[u] = __float_as_uint(r2) - 1u < rb;
        if (hit[u] && r2 < refine2) {  // close pair: exact difference from head + residual
          x[u] += L.x - lx[u];
          y[u] += L.y - ly[u];
          z[u] += L.z - lz[u];
          r2 = fmaf(x[u], x[u], fmaf(y[u], y[u], z[u] * z[u]));
        }
        rr[u] = hit[u] ? r2 : R2;
      }
      if (__any_sync(FULL, hit[0] | hit[1])) {
        const float2 qt = make_float2(T.w, L.w);
#pragma unroll
        for (int u = 0; u < 2; u++) {
          float2 F0, F1;
          helm_eval<ND>(k, rr[u], F0, F1);
          const float2 qm = hit[u] ? sq[u] : make_float2(0.f, 0.f);
          const float2 qn = hit[u] ? qt : make_float2(0.f, 0.f);
          const float2 g = cmul(F1, qm), gs = cmul(F1, qn);
          Pv = cfma(F0, qm, Pv);
          Gx = __ffma2_rn(g, make_float2(x[u], x[u]), Gx);
          Gy = __ffma2_rn(g, make_float2(y[u], y[u]), Gy);
          Gz = __ffma2_rn(g, make_float2(z[u], z[u]), Gz);
          SV[u] = cfma(F0, qn, SV[u]);
          SX[u] = __ffma2_rn(gs, make_float2(-x[u], -x[u]), SX[u]);
          SY[u] = __ffma2_rn(gs, make_float2(-y[u], -y[u]), SY[u]);
          SZ[u] = __ffma2_rn(gs, make_float2(-z[u], -z[u]), SZ[u]);
        }
      }
      Pv.x = __shfl_sync(FULL, Pv.x, src), Pv.y = __shfl_sync(FULL, Pv.y, src);
      Gx.x = __shfl_sync(FULL, Gx.x, src), Gx.y = __shfl_sync(FULL, Gx.y, src);
      Gy.x = __shfl_sync(FULL, Gy.x, src), Gy.y = __shfl_sync(FULL, Gy.y, src);
      Gz.x = __shfl_sync(FULL, Gz.x, src), Gz.y = __shfl_sync(FULL, Gz.y, src);
    }
    if (zone != 0) {  // lanes l and l + 16 hold half of the sums of one target
      float2 *const sums[4] = {&Pv, &Gx, &Gy, &Gz};
#pragma unroll
      for (int m = 0; m < 4; m++) {
        sums[m]->x += __shfl_xor_sync(FULL, sums[m]->x, 16);
        sums[m]->y += __shfl_xor_sync(FULL, sums[m]->y, 16);
      }
    }
    if (zone == 0 || lane >> 4 == zone - 1) {
      acc[0] += Pv.x, acci[0] += Pv.y, acc[1] += Gx.x, acci[1] += Gx.y;
      acc[2] += Gy.x, acci[2] += Gy.y, acc[3] += Gz.x, acci[3] += Gz.y;
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (kidx[u] >= 0) {
        atomicAdd(vsrc + 2L * kidx[u], make_float4(SV[u].x, SV[u].y, SX[u].x, SX[u].y));
        atomicAdd(vsrc + 2L * kidx[u] + 1, make_float4(SY[u].x, SY[u].y, SZ[u].x, SZ[u].y));
      }
    }
  }
}

// Target sums of a complex walk to V (potential times vs, gradient times gs),
// less the self term (src/Interface.cpp:2909-2910).
__device__ __forceinline__ void store_targets_cplx(const int4 G, const uint32_t *__restrict__ perm,
                                                   const double *__restrict__ qcaller,
                                                   double fself_r, double fself_i, double vs,
                                                   double gs, double *__restrict__ V, int lane,
                                                   const double (&acc)[4],
                                                   const double (&acci)[4]) {
  if (lane >= G.y) return;
  const long o = perm[G.x + lane];
  const double qr = qcaller[2 * o], qi = qcaller[2 * o + 1];
  double2 *Vo = reinterpret_cast<double2 *>(V) + 4 * o;
  Vo[0] = make_double2(vs * acc[0] - (fself_r * qr - fself_i * qi),
                       vs * acci[0] - (fself_r * qi + fself_i * qr));
#pragma unroll
  for (int m = 1; m < 4; m++) Vo[m] = make_double2(gs * acc[m], gs * acci[m]);
}

// FP32 direct sum of one warp group (see direct.cu for the scheme): targets
// gpos[G.x, G.x + G.y) in group order, sources spos / qs (charges gathered
// into source order) over the segments [G.z, G.w); qcaller holds the
// caller-order charges for the self term.  sp and slo are this warp's
// 32-entry shared staging arrays.
template <bool CPLX, int FUNC, int SPLIT, int ND, class PK = BuiltinPair>
__device__ __forceinline__ void direct_group_body(
    const PairCoef<float> &k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller, const int4 G,
    const double4 c, const int2 *__restrict__ segs, const uint32_t *__restrict__ perm,
    float refine2, double fself_r, double fself_i, double *__restrict__ V, float4 *sp,
    float4 *slo, int lane) {
#if !defined(NPME_SCALAR_DIRECT)
  if constexpr (!CPLX && SPLIT == 0 && std::is_same<PK, BuiltinPair>::value) {
    direct_group_packed<FUNC, ND>(k, gpos, spos, qs, qcaller, G, c, segs, perm, refine2, fself_r,
                                  V, sp, slo, lane);
    return;
  }
#endif
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  // idle lanes sit far outside the cutoff
  float tx = 1e18f, ty = 1e18f, tz = 1e18f, tlx = 0.f, tly = 0.f, tlz = 0.f;
  if (active) {
    const double4 p = gpos[ti];
    const double dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
    tx = (float)dx, ty = (float)dy, tz = (float)dz;
    tlx = (float)(dx - (double)tx), tly = (float)(dy - (double)ty), tlz = (float)(dz - (double)tz);
  }
  const float R2 = k.R2;
  double acc[4] = {0, 0, 0, 0}, acci[4] = {0, 0, 0, 0};

  // register prefetch of the next chunk: lane l holds source l of the chunk
  SrcCursor cur{G.z, lane};
  cur.normalize(segs, G.w);
  bool pv = cur.seg < G.w;
  double px = 0, py = 0, pz = 0;
  float pq = 0.f, pqi = 0.f;
#define NPME_PREFETCH                                          \
  if (pv) {                                                    \
    const long j_ = (long)segs[cur.seg].x + cur.off;           \
    const double4 p_ = spos[j_];                               \
    px = p_.x, py = p_.y, pz = p_.z;                           \
    if (CPLX) {                                                \
      pq = qs[2 * j_];                                         \
      pqi = qs[2 * j_ + 1];                                    \
    } else {                                                   \
      pq = qs[j_];                                             \
    }                                                          \
  }
  NPME_PREFETCH
  while (__any_sync(0xffffffffu, pv)) {
    const int cnt = __popc(__ballot_sync(0xffffffffu, pv));  // valid lanes form a prefix
    __syncwarp();
    if (pv) {
      const double dx = px - c.x, dy = py - c.y, dz = pz - c.z;
      const float hx = (float)dx, hy = (float)dy, hz = (float)dz;
      sp[lane] = make_float4(hx, hy, hz, pq);
      slo[lane] = make_float4((float)(dx - (double)hx), (float)(dy - (double)hy),
                              (float)(dz - (double)hz), pqi);
    }
    __syncwarp();
    cur.off += 32;
    cur.normalize(segs, G.w);
    pv = cur.seg < G.w;
    NPME_PREFETCH
    float p0 = 0, p1 = 0, p2 = 0, p3 = 0, p0i = 0, p1i = 0, p2i = 0, p3i = 0;
#if !defined(NPME_SCALAR_DIRECT)
    if constexpr (CPLX && SPLIT == 0 && std::is_same<PK, BuiltinPair>::value) {
      float2 Pv = make_float2(0.f, 0.f), Gx = Pv, Gy = Pv, Gz = Pv;
      helmholtz_steps<ND>(k, sp, slo, cnt, tx, ty, tz, tlx, tly, tlz, refine2, Pv, Gx, Gy, Gz);
      p0 = Pv.x, p0i = Pv.y, p1 = Gx.x, p1i = Gx.y, p2 = Gy.x, p2i = Gy.y, p3 = Gz.x, p3i = Gz.y;
    } else
#endif
#pragma unroll kDirectUnroll
    for (int s = 0; s < cnt; s++) {
      const float4 src = sp[s];
      float x = tx - src.x, y = ty - src.y, z = tz - src.z;
      float r2 = fmaf(x, x, fmaf(y, y, z * z));
      if (r2 <= R2 && r2 > 0.f) {
        if (r2 < refine2) {  // close pair: exact difference from head + residual
          const float4 lo = slo[s];
          x += tlx - lo.x;
          y += tly - lo.y;
          z += tlz - lo.z;
          r2 = fmaf(x, x, fmaf(y, y, z * z));
        }
        if (!CPLX) {
          float f1;
          const float f0 = pair_sr<float, FUNC, SPLIT, ND, PK>(k, r2, f1);
          const float gq = f1 * src.w;
          p0 = fmaf(f0, src.w, p0);
          p1 = fmaf(gq, x, p1);
          p2 = fmaf(gq, y, p2);
          p3 = fmaf(gq, z, p3);
        } else {
          float f0r, f0i, f1r, f1i;
          pair_sr_cplx<float, ND, PK>(k, r2, f0r, f0i, f1r, f1i);
          const float qr = src.w, qi = slo[s].w;
          p0 = fmaf(f0r, qr, fmaf(-f0i, qi, p0));
          p0i = fmaf(f0r, qi, fmaf(f0i, qr, p0i));
          const float gr = f1r * qr - f1i * qi, gi = f1r * qi + f1i * qr;
          p1 = fmaf(gr, x, p1);
          p2 = fmaf(gr, y, p2);
          p3 = fmaf(gr, z, p3);
          p1i = fmaf(gi, x, p1i);
          p2i = fmaf(gi, y, p2i);
          p3i = fmaf(gi, z, p3i);
        }
      }
    }
    acc[0] += p0, acc[1] += p1, acc[2] += p2, acc[3] += p3;
    if (CPLX) acci[0] += p0i, acci[1] += p1i, acci[2] += p2i, acci[3] += p3i;
  }
#undef NPME_PREFETCH
  if (active) {
    const long o = perm[ti];
    if (CPLX) {
      const double qr = qcaller[2 * o], qi = qcaller[2 * o + 1];
      acc[0] -= fself_r * qr - fself_i * qi;  // src/Interface.cpp:2909-2910
      acci[0] -= fself_r * qi + fself_i * qr;
      double2 *Vo = reinterpret_cast<double2 *>(V) + 4 * o;
#pragma unroll
      for (int m = 0; m < 4; m++) Vo[m] = make_double2(acc[m], acci[m]);
    } else {
      acc[0] -= fself_r * qcaller[o];  // src/Interface.cpp:2061-2062
      reinterpret_cast<double4 *>(V)[o] = make_double4(acc[0], acc[1], acc[2], acc[3]);
    }
  }
}

// FP64 direct sum of one warp group (the plain precision): the same groups
// and source segments as the FP32 body, every difference and pair kernel in
// double, no head/residual split needed.  sp holds 32 (x, y, z, Re q)
// entries relative to the group centre, sqi the imaginary parts.
template <bool CPLX, int FUNC, int SPLIT, int ND, class PK = BuiltinPair>
__device__ __forceinline__ void direct_group_fp64(
    const PairCoef<double> &k, const double4 *__restrict__ gpos,
    const double4 *__restrict__ spos, const double *__restrict__ qs,
    const double *__restrict__ qcaller, const int4 G, const double4 c,
    const int2 *__restrict__ segs, const uint32_t *__restrict__ perm, double fself_r,
    double fself_i, double *__restrict__ V, double4 *sp, double *sqi, int lane) {
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  double tx = 1e150, ty = 1e150, tz = 1e150;  // idle lanes sit far outside the cutoff
  if (active) {
    const double4 p = gpos[ti];
    tx = p.x - c.x, ty = p.y - c.y, tz = p.z - c.z;
  }
  const double R2 = k.R2;
  double acc[4] = {0, 0, 0, 0}, acci[4] = {0, 0, 0, 0};
  SrcCursor cur{G.z, lane};
  cur.normalize(segs, G.w);
  bool pv = cur.seg < G.w;
  double4 pp = make_double4(0, 0, 0, 0);
  double pqi = 0;
#define NPME_PREFETCH64                                     \
  if (pv) {                                                 \
    const long j_ = (long)segs[cur.seg].x + cur.off;        \
    const double4 p_ = spos[j_];                            \
    pp = make_double4(p_.x - c.x, p_.y - c.y, p_.z - c.z,   \
                      CPLX ? qs[2 * j_] : qs[j_]);          \
    if (CPLX) pqi = qs[2 * j_ + 1];                         \
  }
  NPME_PREFETCH64
  while (__any_sync(0xffffffffu, pv)) {
    const int cnt = __popc(__ballot_sync(0xffffffffu, pv));  // valid lanes form a prefix
    __syncwarp();
    if (pv) {
      sp[lane] = pp;
      if (CPLX) sqi[lane] = pqi;
    }
    __syncwarp();
    cur.off += 32;
    cur.normalize(segs, G.w);
    pv = cur.seg < G.w;
    NPME_PREFETCH64
#pragma unroll 4
    for (int s = 0; s < cnt; s++) {
      const double4 src = sp[s];
      const double x = tx - src.x, y = ty - src.y, z = tz - src.z;
      const double r2 = fma(x, x, fma(y, y, z * z));
      if (r2 <= R2 && r2 > 0.0) {
        if (!CPLX) {
          double f1;
          const double f0 = pair_sr<double, FUNC, SPLIT, ND, PK>(k, r2, f1);
          const double gq = f1 * src.w;
          acc[0] = fma(f0, src.w, acc[0]);
          acc[1] = fma(gq, x, acc[1]);
          acc[2] = fma(gq, y, acc[2]);
          acc[3] = fma(gq, z, acc[3]);
        } else {
          double f0r, f0i, f1r, f1i;
          pair_sr_cplx<double, ND, PK>(k, r2, f0r, f0i, f1r, f1i);
          const double qr = src.w, qi = sqi[s];
          acc[0] = fma(f0r, qr, fma(-f0i, qi, acc[0]));
          acci[0] = fma(f0r, qi, fma(f0i, qr, acci[0]));
          const double gr = f1r * qr - f1i * qi, gi = f1r * qi + f1i * qr;
          acc[1] = fma(gr, x, acc[1]);
          acc[2] = fma(gr, y, acc[2]);
          acc[3] = fma(gr, z, acc[3]);
          acci[1] = fma(gi, x, acci[1]);
          acci[2] = fma(gi, y, acci[2]);
          acci[3] = fma(gi, z, acci[3]);
        }
      }
    }
  }
#undef NPME_PREFETCH64
  if (active) {
    const long o = perm[ti];
    if (CPLX) {
      const double qr = qcaller[2 * o], qi = qcaller[2 * o + 1];
      acc[0] -= fself_r * qr - fself_i * qi;  // src/Interface.cpp:2909-2910
      acci[0] -= fself_r * qi + fself_i * qr;
      double2 *Vo = reinterpret_cast<double2 *>(V) + 4 * o;
#pragma unroll
      for (int m = 0; m < 4; m++) Vo[m] = make_double2(acc[m], acci[m]);
    } else {
      acc[0] -= fself_r * qcaller[o];  // src/Interface.cpp:2061-2062
      reinterpret_cast<double4 *>(V)[o] = make_double4(acc[0], acc[1], acc[2], acc[3]);
    }
  }
}

// FP32 direct sum of one warp group with every unordered pair evaluated once,
// for real caller-defined kernels: the pair-once walk of direct_group_sym with the
// scalar pair kernel (pair_sr) of the one-sided body.  Coordinates are
// unscaled FP32 offsets from the group centre (heads in th with the target
// charge, residuals in tl), close pairs refined from the residuals; the
// source-side sums go to vsrc as the gradient itself (merge scale 1).
template <int FUNC, int SPLIT, int ND, class PK = BuiltinPair>
__device__ __forceinline__ void direct_group_sym_scalar(
    const PairCoef<float> &k, const double4 *__restrict__ gpos, const double4 *__restrict__ spos,
    const float *__restrict__ qs, const double *__restrict__ qcaller, const int4 G,
    const double4 c, const int2 *__restrict__ segs, const uint32_t *__restrict__ perm,
    float refine2, double fself_r, double *__restrict__ V, float4 *__restrict__ vsrc,
    float4 *th, float4 *tl, int lane) {
  const unsigned FULL = 0xffffffffu;
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  float tx = 1e18f, ty = 1e18f, tz = 1e18f, tlx = 0.f, tly = 0.f, tlz = 0.f, tq = 0.f;
  long o = 0;
  if (active) {
    const double4 p = gpos[ti];
    o = perm[ti];
    const double dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
    tx = (float)dx, ty = (float)dy, tz = (float)dz;
    tlx = (float)(dx - (double)tx), tly = (float)(dy - (double)ty), tlz = (float)(dz - (double)tz);
    tq = (float)qcaller[o];
  }
  th[lane] = make_float4(tx, ty, tz, tq);
  tl[lane] = make_float4(tlx, tly, tlz, 0.f);
  __syncwarp();
  const float R2 = k.R2;
  double acc[4] = {0, 0, 0, 0};
  {  // pairs inside the group, target side only, differences always refined
    float aV = 0.f, aX = 0.f, aY = 0.f, aZ = 0.f;
    for (int s = 0; s < G.y; s++) {
      const float4 S = th[s], L = tl[s];
      const float x = (tx - S.x) + (tlx - L.x), y = (ty - S.y) + (tly - L.y),
                  z = (tz - S.z) + (tlz - L.z);
      const float r2 = fmaf(x, x, fmaf(y, y, z * z));
      if (r2 <= R2 && r2 > 0.f) {
        float f1;
        const float f0 = pair_sr<float, FUNC, SPLIT, ND, PK>(k, r2, f1);
        const float g = f1 * S.w;
        aV = fmaf(f0, S.w, aV);
        aX = fmaf(g, x, aX);
        aY = fmaf(g, y, aY);
        aZ = fmaf(g, z, aZ);
      }
    }
    acc[0] += aV, acc[1] += aX, acc[2] += aY, acc[3] += aZ;
  }
  SrcCursor ca{G.z, lane};
  ca.normalize(segs, G.w);
  SrcCursor cb{ca.seg, ca.off + 32};
  cb.normalize(segs, G.w);
  bool va = ca.seg < G.w, vb = cb.seg < G.w;
  long ja = -1, jb = -1;
  double4 pa = make_double4(0, 0, 0, 0), pb = pa;
  float qa = 0.f, qb = 0.f;
  if (va) ja = (long)segs[ca.seg].x + ca.off, pa = spos[ja], qa = qs[ja];
  if (vb) jb = (long)segs[cb.seg].x + cb.off, pb = spos[jb], qb = qs[jb];
  while (__any_sync(FULL, va)) {
    // the lane's two sources; empty slots far away on the other side from
    // idle targets, with charge 0
    float sx[2] = {-1e18f, -1e18f}, sy[2] = {-1e18f, -1e18f}, sz[2] = {-1e18f, -1e18f};
    float lx[2] = {0.f, 0.f}, ly[2] = {0.f, 0.f}, lz[2] = {0.f, 0.f}, sq[2] = {0.f, 0.f};
    const long kidx[2] = {va ? (long)pa.w : -1, vb ? (long)pb.w : -1};  // brick positions
    if (va) {
      const double dx = pa.x - c.x, dy = pa.y - c.y, dz = pa.z - c.z;
      sx[0] = (float)dx, sy[0] = (float)dy, sz[0] = (float)dz;
      lx[0] = (float)(dx - (double)sx[0]), ly[0] = (float)(dy - (double)sy[0]);
      lz[0] = (float)(dz - (double)sz[0]);
      sq[0] = qa;
    }
    if (vb) {
      const double dx = pb.x - c.x, dy = pb.y - c.y, dz = pb.z - c.z;
      sx[1] = (float)dx, sy[1] = (float)dy, sz[1] = (float)dz;
      lx[1] = (float)(dx - (double)sx[1]), ly[1] = (float)(dy - (double)sy[1]);
      lz[1] = (float)(dz - (double)sz[1]);
      sq[1] = qb;
    }
    ca.off += 64;
    ca.normalize(segs, G.w);
    cb.off += 64;
    cb.normalize(segs, G.w);
    va = ca.seg < G.w, vb = cb.seg < G.w;
    if (va) ja = (long)segs[ca.seg].x + ca.off, pa = spos[ja], qa = qs[ja];
    if (vb) jb = (long)segs[cb.seg].x + cb.off, pb = spos[jb], qb = qs[jb];

    float aV = 0.f, aX = 0.f, aY = 0.f, aZ = 0.f;  // target side, rotating
    float S[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};  // source side
    const int src = (lane + 1) & 31;
    for (int kk = 0; kk < 32; kk++) {
      const int tt = (lane + kk) & 31;
      const float4 T = th[tt];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        float x = T.x - sx[u], y = T.y - sy[u], z = T.z - sz[u];
        float r2 = fmaf(x, x, fmaf(y, y, z * z));
        if (r2 <= R2 && r2 > 0.f) {
          if (r2 < refine2) {  // close pair: exact difference from head + residual
            const float4 L = tl[tt];
            x += L.x - lx[u];
            y += L.y - ly[u];
            z += L.z - lz[u];
            r2 = fmaf(x, x, fmaf(y, y, z * z));
          }
          float f1;
          const float f0 = pair_sr<float, FUNC, SPLIT, ND, PK>(k, r2, f1);
          const float g = f1 * sq[u], gs = f1 * T.w;
          aV = fmaf(f0, sq[u], aV);
          aX = fmaf(g, x, aX);
          aY = fmaf(g, y, aY);
          aZ = fmaf(g, z, aZ);
          S[u][0] = fmaf(f0, T.w, S[u][0]);
          S[u][1] = fmaf(-gs, x, S[u][1]);
          S[u][2] = fmaf(-gs, y, S[u][2]);
          S[u][3] = fmaf(-gs, z, S[u][3]);
        }
      }
      aV = __shfl_sync(FULL, aV, src);
      aX = __shfl_sync(FULL, aX, src);
      aY = __shfl_sync(FULL, aY, src);
      aZ = __shfl_sync(FULL, aZ, src);
    }
    acc[0] += aV, acc[1] += aX, acc[2] += aY, acc[3] += aZ;
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (kidx[u] >= 0) atomicAdd(vsrc + kidx[u], make_float4(S[u][0], S[u][1], S[u][2], S[u][3]));
  }
  if (active) {
    acc[0] -= fself_r * qcaller[o];  // src/Interface.cpp:2061-2062
    reinterpret_cast<double4 *>(V)[o] = make_double4(acc[0], acc[1], acc[2], acc[3]);
  }
}

// 1/sqrt(s) for normal finite s > 0: the hardware's approximation (20 bits or
// more) and one step of Householder's cubically convergent iteration, y + y e
// (1/2 + 3/8 e) with e = 1 - s y^2, whose error is 5/16 e^3 < 2^-57.  Five
// FP64 operations and no branch.
__device__ __forceinline__ double rsqrt_iter(double s) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  const double e = fma(-(s * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

template <int N>
__device__ __forceinline__ double pow_n(double u) {
  if constexpr (N == 1) {
    return u;
  } else {
    const double h = pow_n<N / 2>(u), h2 = h * h;
    return N % 2 ? h2 * u : h2;
  }
}

// The real DM pair kernel of dm_eval2 in FP64 (s = (r / Rdir)^2 in (0, 1]; ND > 0
// for alpha < 0, ND = 0 any order and alpha).
template <int FUNC, int ND>
__device__ __forceinline__ void dm_eval64(const PairCoef<double> &k, double s, double &f0,
                                          double &t) {
  constexpr int nd = dm_degree<ND>();
  const double u = 1.0 - s;
  double h = k.nc2[nd].x;
#pragma unroll
  for (int n = nd - 1; n >= 1; n--) h = fma(h, u, k.nc2[n].x);
  const double ri = rsqrt_iter(s), ri2 = ri * ri;
  const double e0 = FUNC == 1 ? rpow_t(s, k.half_alpha) : ri;
  f0 = fma(h, u, e0 - 1.0);
  if constexpr (ND > 0) {
    t = fma(pow_n<ND>(u), k.kn2.x, f0) * ri2;
  } else {
    double d = k.nq2[nd - 1].x;
#pragma unroll
    for (int n = nd - 2; n >= 0; n--) d = fma(d, u, k.nq2[n].x);
    t = fma(e0, ri2, d);
  }
}

// FP64 real DM kernels with every unordered pair evaluated once: the walk of
// direct_group_sym64 (below) without branches.  A pair is a hit when s = (r /
// Rdir)^2 is a normal number below 1 (compared on its high word, an integer
// operation: the FP64 pipe, at half the FP32 rate, is what bounds the kernel); a
// miss gets s = 1 and charge 0 on both sides.  36 FP64 operations per pair at order
// 6, 41 and a hit branch before.  (Scaling the coordinates instead of r^2 takes one
// operation less, 1,186 against 1,200 us at 200,000 points, but rounds the
// differences of near points; scaling by a power of two and expanding about (Rdir /
// unit)^2 gave 1,274: its constants take registers.)  The group's work is shared by
// nsplit warps as in direct_group_sym.
template <int FUNC, int ND>
__device__ __forceinline__ void direct_group_sym64_dm(
    const PairCoef<double> &k, const double4 *__restrict__ gpos,
    const double4 *__restrict__ spos, const double *__restrict__ qs,
    const double *__restrict__ qcaller, const int4 G, const double4 c,
    const int2 *__restrict__ segs, const int2 zones, const uint32_t *__restrict__ perm,
    double *__restrict__ vsrc, double4 *tsm, int lane, int part, int nsplit,
    double (&acc)[4]) {
  const unsigned FULL = 0xffffffffu;
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  const double vs = k.vscale, gsc = k.gscale;
  double tx = 1e150, ty = 1e150, tz = 1e150, tq = 0.0;  // idle lanes: far away, no charge
  if (active) {
    const double4 p = gpos[ti];
    tx = p.x - c.x, ty = p.y - c.y, tz = p.z - c.z;
    tq = qcaller[perm[ti]];
  }
  tsm[lane] = make_double4(tx, ty, tz, tq);
  __syncwarp();
  // s in [2^-1022, 1): the high word in [0x00100000, 0x3ff00000)
  auto inside = [](double s) {
    return (unsigned)__double2hiint(s) - 0x00100000u < 0x3fe00000u;
  };
  // pairs inside the group, target side only (each is met from both ends)
  for (int s = part; s < G.y; s += nsplit) {
    const double4 S = tsm[s];
    const double x = tx - S.x, y = ty - S.y, z = tz - S.z;
    const double d2 = fma(x, x, fma(y, y, z * z)) * k.invR2;
    const bool hit = inside(d2);
    double f0, t;
    dm_eval64<FUNC, ND>(k, hit ? d2 : 1.0, f0, t);
    const double q = hit ? S.w : 0.0, gq = t * q;
    acc[0] = fma(f0, q, acc[0]);
    acc[1] = fma(-gq, x, acc[1]);
    acc[2] = fma(-gq, y, acc[2]);
    acc[3] = fma(-gq, z, acc[3]);
  }
  // half-shell segments in chunks of 64 sources (register prefetch)
  ZoneWalk<2> walk(segs, G, zones, lane, part, nsplit);
  double4 p[2];
  int slot[2] = {-1, -1};  // source-side slots (brick positions)
#pragma unroll
  for (int i = 0; i < 2; i++) {
    p[i] = make_double4(0, 0, 0, 0);
    if (walk.v[i]) {
      const long j = walk.index(i);
      p[i] = spos[j], slot[i] = (int)p[i].w, p[i].w = qs[j];
    }
  }
  while (walk.any()) {
    const int zone = walk.zone;
    // empty slots far away on the other side from idle targets, no charge
    double4 src[2];
    int to[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      src[i] = make_double4(-1e150, -1e150, -1e150, 0.0);
      to[i] = walk.v[i] ? slot[i] : -1;
      if (walk.v[i])
        src[i] = make_double4(p[i].x - c.x, p[i].y - c.y, p[i].z - c.z, p[i].w);
    }
    walk.next();
#pragma unroll
    for (int i = 0; i < 2; i++)
      if (walk.v[i]) {
        const long j = walk.index(i);
        p[i] = spos[j], slot[i] = (int)p[i].w, p[i].w = qs[j];
      }
    double aV = 0, aX = 0, aY = 0, aZ = 0;                   // target side, rotating
    double S[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};           // source side
    const int next = (lane + 1) & 31;
    // all targets, or the half that the zone reaches
    const int mask = zone == 0 ? 31 : 15, from = zone == 2 ? 16 : 0;
#pragma unroll 2
    for (int kk = 0; kk <= mask; kk++) {
      const double4 T = tsm[from + ((lane + kk) & mask)];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const double x = T.x - src[i].x, y = T.y - src[i].y, z = T.z - src[i].z;
        const double d2 = fma(x, x, fma(y, y, z * z)) * k.invR2;
        const bool hit = inside(d2);
        double f0, t;
        dm_eval64<FUNC, ND>(k, hit ? d2 : 1.0, f0, t);
        const double qm = hit ? src[i].w : 0.0, qt = hit ? T.w : 0.0;
        const double gm = t * qm, gt = t * qt;
        aV = fma(f0, qm, aV);
        aX = fma(-gm, x, aX);
        aY = fma(-gm, y, aY);
        aZ = fma(-gm, z, aZ);
        S[i][0] = fma(f0, qt, S[i][0]);
        S[i][1] = fma(gt, x, S[i][1]);
        S[i][2] = fma(gt, y, S[i][2]);
        S[i][3] = fma(gt, z, S[i][3]);
      }
      aV = __shfl_sync(FULL, aV, next);
      aX = __shfl_sync(FULL, aX, next);
      aY = __shfl_sync(FULL, aY, next);
      aZ = __shfl_sync(FULL, aZ, next);
    }
    if (zone != 0) {  // lanes l and l + 16 hold half of the sums of one target
      aV += __shfl_xor_sync(FULL, aV, 16), aX += __shfl_xor_sync(FULL, aX, 16);
      aY += __shfl_xor_sync(FULL, aY, 16), aZ += __shfl_xor_sync(FULL, aZ, 16);
    }
    if (zone == 0 || lane >> 4 == zone - 1) {
      acc[0] += aV;
      acc[1] += aX;
      acc[2] += aY;
      acc[3] += aZ;
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
      if (to[i] >= 0) {
        double *d = vsrc + 4L * to[i];
        atomicAdd(d, vs * S[i][0]);
#pragma unroll
        for (int m = 1; m < 4; m++) atomicAdd(d + m, gsc * S[i][m]);
      }
  }
}

// sin and cos of x in FP64, |x| < kMaxHelmArg, without a branch: Cody-Waite
// reduction to [-pi/4, pi/4] with pi/2 as the sum of two doubles, Taylor
// polynomials of degree 15 and 16 (truncation below 5e-17), quadrant by
// selects.  About half the FP64 operations of the general sincos.
constexpr double kMaxHelmArg = 1e5;
__device__ __forceinline__ void sincos_taylor(double x, double &sn, double &cs) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
  const double m = fma(x, 0.63661977236758134308, kMagic), n = m - kMagic;
  double r = fma(-n, 1.57079632679489661923, x);
  r = fma(-n, 6.12323399573676603587e-17, r);
  const double z = r * r;
  double a = -1.0 / 1307674368000.0;  // -1/15!
  a = fma(a, z, 1.0 / 6227020800.0);
  a = fma(a, z, -1.0 / 39916800.0);
  a = fma(a, z, 1.0 / 362880.0);
  a = fma(a, z, -1.0 / 5040.0);
  a = fma(a, z, 1.0 / 120.0);
  a = fma(a, z, -1.0 / 6.0);
  const double s = fma(a * z, r, r);
  double b = 1.0 / 20922789888000.0;  // 1/16!
  b = fma(b, z, -1.0 / 87178291200.0);
  b = fma(b, z, 1.0 / 479001600.0);
  b = fma(b, z, -1.0 / 3628800.0);
  b = fma(b, z, 1.0 / 40320.0);
  b = fma(b, z, -1.0 / 720.0);
  b = fma(b, z, 1.0 / 24.0);
  b = fma(b, z, -0.5);
  const double c = fma(b, z, 1.0);
  const int q = __double2loint(m);  // n mod 2^32
  sn = q & 1 ? c : s;
  cs = q & 1 ? s : c;
  if (q & 2) sn = -sn;
  if ((q + 1) & 2) cs = -cs;
}

// Helmholtz DM pair kernel in FP64 (coordinates times k.invR, s = r^2 in (0, cut2]):
// F0 = exp(i kap r)/r - P and F1 = (1/r) dF0/dr, P the matched polynomial in u =
// cut2 - s (PairCoef; src/KernelFunctionHelmholtz.cpp:506-563).  ND = 0: the order
// at run time, in a loop.  (Zero-padded to kMaxDeriv as in FP32, the 62 coefficients
// spilled 560 bytes a thread: 62,501 points 1,840 us at every order, in the loop
// 1,206 at order 5, 1,423 at 10 and 1,616 at 15.)
template <int ND>
__device__ __forceinline__ void helm_eval64(const PairCoef<double> &k, double s, double2 &F0,
                                            double2 &F1) {
  const double ri = rsqrt_iter(s), r = s * ri, u = k.cut2 - s;
  double sn, cs;
  sincos_taylor(k.kapr * r, sn, cs);
  const double damp = k.kapi != 0.0 ? exp(-k.kapi * r) * ri : ri;
  const double er = cs * damp, ei = sn * damp;  // exp(i kap r) / r
  // its radial derivative over r: E (i kap / r - 1 / r^2)
  const double A = fma(-k.kapi, ri, -ri * ri), B = k.kapr * ri;
  double pr, pi, dr, di;
  if constexpr (ND == 0) {
    const int N = k.nder;  // 2 at least
    pr = fma(k.hc[N].x, u, k.hc[N - 1].x), pi = fma(k.hc[N].y, u, k.hc[N - 1].y);
    dr = k.hd[N - 1].x, di = k.hd[N - 1].y;
#pragma unroll 2
    for (int n = N - 2; n >= 0; n--) {
      pr = fma(pr, u, k.hc[n].x), pi = fma(pi, u, k.hc[n].y);
      dr = fma(dr, u, k.hd[n].x), di = fma(di, u, k.hd[n].y);
    }
  } else {
    pr = k.hc[ND].x, pi = k.hc[ND].y, dr = k.hd[ND - 1].x, di = k.hd[ND - 1].y;
#pragma unroll
    for (int n = ND - 1; n >= 0; n--) pr = fma(pr, u, k.hc[n].x), pi = fma(pi, u, k.hc[n].y);
#pragma unroll
    for (int n = ND - 2; n >= 0; n--) dr = fma(dr, u, k.hd[n].x), di = fma(di, u, k.hd[n].y);
  }
  F0 = make_double2(er + pr, ei + pi);
  F1 = make_double2(fma(A, er, fma(-B, ei, dr)), fma(A, ei, fma(B, er, di)));
}

// complex a * b + c on (re, im) doubles
__device__ __forceinline__ void cfma64(double2 a, double2 b, double &cr, double &ci) {
  cr = fma(a.x, b.x, fma(-a.y, b.y, cr));
  ci = fma(a.x, b.y, fma(a.y, b.x, ci));
}

// 0 < r^2 < cut2 (r^2 a normal number) by its bits, in integer operations
__device__ __forceinline__ bool inside64(const PairCoef<double> &k, double r2) {
  return (unsigned long long)__double_as_longlong(r2) - kMinNormal64 < k.cut_bits;
}

// FP64 Helmholtz with every unordered pair evaluated once, the complex
// counterpart of direct_group_sym64_dm: coordinates scaled by a power of two,
// misses at s = cut2 with charge 0, no branch.  One source per lane and chunks of
// 32 (two would take 170-200 registers and halve the resident warps); the eight
// target sums rotate one lane down per step, the source sums go to vsrc ([n][8]
// doubles: V, x, y, z as re, im).  About 105 FP64 operations per pair at order 8; the
// one-sided walk spends about 130 on each of the pair's two directions.
// tsm: the targets' x, y, z, Re q, Im q.
template <int ND>
__device__ __forceinline__ void direct_group_sym64_helm(
    const PairCoef<double> &k, const double4 *__restrict__ gpos,
    const double4 *__restrict__ spos, const double *__restrict__ qs,
    const double *__restrict__ qcaller, const int4 G, const double4 c,
    const int2 *__restrict__ segs, const int2 zones, const uint32_t *__restrict__ perm,
    double *__restrict__ vsrc, double (*tsm)[32], int lane, int part, int nsplit,
    double (&acc)[4], double (&acci)[4]) {
  const unsigned FULL = 0xffffffffu;
  const int ti = G.x + lane;
  const double ir = k.invR, gsc = ir * ir;  // F0 / unit, F1 x / unit^2
  double tx = 1e150, ty = 1e150, tz = 1e150;  // idle lanes: far away, no charge
  double2 tq = make_double2(0.0, 0.0);
  if (lane < G.y) {
    const double4 p = gpos[ti];
    tx = (p.x - c.x) * ir, ty = (p.y - c.y) * ir, tz = (p.z - c.z) * ir;
    const long o = perm[ti];
    tq = make_double2(qcaller[2 * o], qcaller[2 * o + 1]);
  }
  tsm[0][lane] = tx, tsm[1][lane] = ty, tsm[2][lane] = tz;
  tsm[3][lane] = tq.x, tsm[4][lane] = tq.y;
  __syncwarp();
  // pairs inside the group, target side only (each is met from both ends)
  for (int s = part; s < G.y; s += nsplit) {
    const double x = tx - tsm[0][s], y = ty - tsm[1][s], z = tz - tsm[2][s];
    const double r2 = fma(x, x, fma(y, y, z * z));
    const bool hit = inside64(k, r2);
    double2 F0, F1;
    helm_eval64<ND>(k, hit ? r2 : k.cut2, F0, F1);
    const double2 q = make_double2(hit ? tsm[3][s] : 0.0, hit ? tsm[4][s] : 0.0);
    double gr = 0, gi = 0;
    cfma64(F0, q, acc[0], acci[0]);
    cfma64(F1, q, gr, gi);
    acc[1] = fma(gr, x, acc[1]), acci[1] = fma(gi, x, acci[1]);
    acc[2] = fma(gr, y, acc[2]), acci[2] = fma(gi, y, acci[2]);
    acc[3] = fma(gr, z, acc[3]), acci[3] = fma(gi, z, acci[3]);
  }
  ZoneWalk<1> walk(segs, G, zones, lane, part, nsplit);
  double4 p = make_double4(0, 0, 0, 0);
  double2 q = make_double2(0, 0);
  if (walk.v[0]) {
    const long j = walk.index(0);
    p = spos[j], q = reinterpret_cast<const double2 *>(qs)[j];
  }
  while (walk.any()) {
    const int zone = walk.zone;
    // empty slots far away on the other side from idle targets, no charge
    double sx = -1e150, sy = -1e150, sz = -1e150;
    double2 sq = make_double2(0.0, 0.0);
    int slot = -1;
    if (walk.v[0]) {
      sx = (p.x - c.x) * ir, sy = (p.y - c.y) * ir, sz = (p.z - c.z) * ir;
      sq = q;
      slot = (int)p.w;
    }
    walk.next();
    if (walk.v[0]) {
      const long j = walk.index(0);
      p = spos[j], q = reinterpret_cast<const double2 *>(qs)[j];
    }
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // target side, rotating
    double S[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // source side
    const int next = (lane + 1) & 31;
    const int mask = zone == 0 ? 31 : 15, from = zone == 2 ? 16 : 0;
#pragma unroll 1
    for (int kk = 0; kk <= mask; kk++) {
      const int t = from + ((lane + kk) & mask);
      const double x = tsm[0][t] - sx, y = tsm[1][t] - sy, z = tsm[2][t] - sz;
      const double r2 = fma(x, x, fma(y, y, z * z));
      const bool hit = inside64(k, r2);
      double2 F0, F1;
      helm_eval64<ND>(k, hit ? r2 : k.cut2, F0, F1);
      const double2 qm = make_double2(hit ? sq.x : 0.0, hit ? sq.y : 0.0);
      const double2 qt = make_double2(hit ? tsm[3][t] : 0.0, hit ? tsm[4][t] : 0.0);
      const double gr = fma(F1.x, qm.x, -F1.y * qm.y), gi = fma(F1.x, qm.y, F1.y * qm.x);
      cfma64(F0, qm, a[0], a[1]);
      a[2] = fma(gr, x, a[2]), a[3] = fma(gi, x, a[3]);
      a[4] = fma(gr, y, a[4]), a[5] = fma(gi, y, a[5]);
      a[6] = fma(gr, z, a[6]), a[7] = fma(gi, z, a[7]);
      const double hr = fma(F1.x, qt.x, -F1.y * qt.y), hi = fma(F1.x, qt.y, F1.y * qt.x);
      cfma64(F0, qt, S[0], S[1]);
      S[2] = fma(-hr, x, S[2]), S[3] = fma(-hi, x, S[3]);
      S[4] = fma(-hr, y, S[4]), S[5] = fma(-hi, y, S[5]);
      S[6] = fma(-hr, z, S[6]), S[7] = fma(-hi, z, S[7]);
#pragma unroll
      for (int m = 0; m < 8; m++) a[m] = __shfl_sync(FULL, a[m], next);
    }
    if (zone != 0)  // lanes l and l + 16 hold half of the sums of one target
#pragma unroll
      for (int m = 0; m < 8; m++) a[m] += __shfl_xor_sync(FULL, a[m], 16);
    if (zone == 0 || lane >> 4 == zone - 1)
#pragma unroll
      for (int m = 0; m < 4; m++) acc[m] += a[2 * m], acci[m] += a[2 * m + 1];
    if (slot >= 0) {
      double *d = vsrc + 8L * slot;
#pragma unroll
      for (int m = 0; m < 8; m++) atomicAdd(d + m, (m < 2 ? ir : gsc) * S[m]);
    }
  }
}

// Target sums of the FP64 pair-once walk to V (sums scaled by vs, gs), less
// the self term f_LR(0) q (src/Interface.cpp:2061-2062).
__device__ __forceinline__ void store_targets64(const int4 G, const uint32_t *__restrict__ perm,
                                                const double *__restrict__ qcaller,
                                                double fself_r, double vs, double gs,
                                                double *__restrict__ V, int lane,
                                                const double (&acc)[4]) {
  if (lane >= G.y) return;
  const long o = perm[G.x + lane];
  reinterpret_cast<double4 *>(V)[o] =
      make_double4(vs * acc[0] - fself_r * qcaller[o], gs * acc[1], gs * acc[2], gs * acc[3]);
}

// FP64 direct sum of one warp group with every unordered pair evaluated once
// (the FP64 counterpart of direct_group_sym, for the real kernels): the
// group's targets (x, y, z, q) sit in shared memory, each lane holds two
// sources of a 64-source chunk of the half-shell segments, target (l + k)
// mod 32 meets lane l at step k and its sums rotate one lane down per step;
// the source-side sums of a chunk go to vsrc ([n][4] doubles, slot = the
// source's brick-order position) with one FP64 atomic per component.  Pairs
// inside the group are a first, one-sided pass.  Same pair arithmetic as direct_group_fp64.
template <int FUNC, int SPLIT, int ND, class PK = BuiltinPair>
__device__ __forceinline__ void direct_group_sym64(
    const PairCoef<double> &k, const double4 *__restrict__ gpos,
    const double4 *__restrict__ spos, const double *__restrict__ qs,
    const double *__restrict__ qcaller, const int4 G, const double4 c,
    const int2 *__restrict__ segs, const uint32_t *__restrict__ perm, double fself_r,
    double *__restrict__ V, double *__restrict__ vsrc, double4 *tsm, int lane) {
  const unsigned FULL = 0xffffffffu;
  const int ti = G.x + lane;
  const bool active = lane < G.y;
  double tx = 1e150, ty = 1e150, tz = 1e150, tq = 0.0;  // idle lanes: far away, no charge
  long o = 0;
  if (active) {
    const double4 p = gpos[ti];
    o = perm[ti];
    tx = p.x - c.x, ty = p.y - c.y, tz = p.z - c.z;
    tq = qcaller[o];
  }
  tsm[lane] = make_double4(tx, ty, tz, tq);
  __syncwarp();
  const double R2 = k.R2;
  double acc[4] = {0, 0, 0, 0};
  // pairs inside the group, target side only (each is met from both ends)
  for (int s = 0; s < G.y; s++) {
    const double4 S = tsm[s];
    const double x = tx - S.x, y = ty - S.y, z = tz - S.z;
    const double r2 = fma(x, x, fma(y, y, z * z));
    if (r2 <= R2 && r2 > 0.0) {
      double f1;
      const double f0 = pair_sr<double, FUNC, SPLIT, ND, PK>(k, r2, f1);
      const double gq = f1 * S.w;
      acc[0] = fma(f0, S.w, acc[0]);
      acc[1] = fma(gq, x, acc[1]);
      acc[2] = fma(gq, y, acc[2]);
      acc[3] = fma(gq, z, acc[3]);
    }
  }
  // half-shell segments in chunks of 64 sources (register prefetch)
  SrcCursor ca{G.z, lane};
  ca.normalize(segs, G.w);
  SrcCursor cb{ca.seg, ca.off + 32};
  cb.normalize(segs, G.w);
  bool va = ca.seg < G.w, vb = cb.seg < G.w;
  long ja = -1, jb = -1, sla = -1, slb = -1;  // sla, slb: source-side slots (brick positions)
  double4 pa = make_double4(0, 0, 0, 0), pb = pa;
  if (va) ja = (long)segs[ca.seg].x + ca.off, pa = spos[ja], sla = (long)pa.w, pa.w = qs[ja];
  if (vb) jb = (long)segs[cb.seg].x + cb.off, pb = spos[jb], slb = (long)pb.w, pb.w = qs[jb];
  while (__any_sync(FULL, va)) {
    // empty slots far away on the other side from idle targets, no charge
    double4 A = make_double4(-1e150, -1e150, -1e150, 0.0), B = A;
    if (va) A = make_double4(pa.x - c.x, pa.y - c.y, pa.z - c.z, pa.w);
    if (vb) B = make_double4(pb.x - c.x, pb.y - c.y, pb.z - c.z, pb.w);
    const long ka = va ? sla : -1, kb = vb ? slb : -1;
    ca.off += 64;
    ca.normalize(segs, G.w);
    cb.off += 64;
    cb.normalize(segs, G.w);
    va = ca.seg < G.w, vb = cb.seg < G.w;
    if (va) ja = (long)segs[ca.seg].x + ca.off, pa = spos[ja], sla = (long)pa.w, pa.w = qs[ja];
    if (vb) jb = (long)segs[cb.seg].x + cb.off, pb = spos[jb], slb = (long)pb.w, pb.w = qs[jb];

    double aV = 0, aX = 0, aY = 0, aZ = 0;           // target side, rotating
    double sa[4] = {0, 0, 0, 0}, sb[4] = {0, 0, 0, 0};  // source side
    const int src = (lane + 1) & 31;
#pragma unroll 2
    for (int kk = 0; kk < 32; kk++) {
      const double4 T = tsm[(lane + kk) & 31];
      {
        const double x = T.x - A.x, y = T.y - A.y, z = T.z - A.z;
        const double r2 = fma(x, x, fma(y, y, z * z));
        if (r2 <= R2 && r2 > 0.0) {
          double f1;
          const double f0 = pair_sr<double, FUNC, SPLIT, ND, PK>(k, r2, f1);
          const double gq = f1 * A.w, gs = f1 * T.w;
          aV = fma(f0, A.w, aV);
          aX = fma(gq, x, aX);
          aY = fma(gq, y, aY);
          aZ = fma(gq, z, aZ);
          sa[0] = fma(f0, T.w, sa[0]);
          sa[1] = fma(-gs, x, sa[1]);
          sa[2] = fma(-gs, y, sa[2]);
          sa[3] = fma(-gs, z, sa[3]);
        }
      }
      {
        const double x = T.x - B.x, y = T.y - B.y, z = T.z - B.z;
        const double r2 = fma(x, x, fma(y, y, z * z));
        if (r2 <= R2 && r2 > 0.0) {
          double f1;
          const double f0 = pair_sr<double, FUNC, SPLIT, ND, PK>(k, r2, f1);
          const double gq = f1 * B.w, gs = f1 * T.w;
          aV = fma(f0, B.w, aV);
          aX = fma(gq, x, aX);
          aY = fma(gq, y, aY);
          aZ = fma(gq, z, aZ);
          sb[0] = fma(f0, T.w, sb[0]);
          sb[1] = fma(-gs, x, sb[1]);
          sb[2] = fma(-gs, y, sb[2]);
          sb[3] = fma(-gs, z, sb[3]);
        }
      }
      aV = __shfl_sync(FULL, aV, src);
      aX = __shfl_sync(FULL, aX, src);
      aY = __shfl_sync(FULL, aY, src);
      aZ = __shfl_sync(FULL, aZ, src);
    }
    acc[0] += aV;
    acc[1] += aX;
    acc[2] += aY;
    acc[3] += aZ;
    if (ka >= 0)
#pragma unroll
      for (int m = 0; m < 4; m++) atomicAdd(vsrc + 4 * ka + m, sa[m]);
    if (kb >= 0)
#pragma unroll
      for (int m = 0; m < 4; m++) atomicAdd(vsrc + 4 * kb + m, sb[m]);
  }
  if (active) {
    acc[0] -= fself_r * qcaller[o];  // src/Interface.cpp:2061-2062
    reinterpret_cast<double4 *>(V)[o] = make_double4(acc[0], acc[1], acc[2], acc[3]);
  }
}

}  // namespace npme
