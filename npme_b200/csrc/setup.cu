// Per-geometry set-up on the device: everything CalcV needs that depends on
// the point positions, built from the caller's coordinates in HBM.
//
//  * bounding box and coordinate check (one reduction, read back by the host,
//    which derives the PME box, src/RecSumSupportFunctions.cpp:182-201,
//    276-296);
//  * brick order of the spreading and interpolation (src/RecSumQ.cpp:527-895,
//    NPME_RecSumQ_CreateBlock): each point's stencil origin and fractional
//    offset (src/RecSumSupportFunctions.h:123-151), points sorted by brick
//    and, inside a brick, by the shared-memory bank of their stencil origin;
//  * the direct sum's warp groups (the reference's cells and cluster pairs,
//    src/PartitionEmbeddedBox.cpp:47-205, src/PartitionBox.cpp:789-923):
//    targets sorted by (xy column, quantised z, index) and cut into runs of
//    32, sources sorted by (fine xy column, quantised z, index); for every group the z
//    ranges of the fine columns that can hold a point within Rdir of the
//    group's bounding box, and the half-shell part of them for the
//    every-pair-once walk; groups ordered by their work, heaviest first.
//
// Any number of systems are set up in one pass (a batch: the serving queue
// sets up the requests it admits together; npme_gpu_setup is a batch of
// one), so the kernel launches of a set-up are shared by all its systems.
// Sorting is done with stable radix sorts (values = point indices in
// increasing order) on keys that start with the system's index, so every
// order is (system, key, index) lexicographic and the result does not
// depend on timing or on the other systems of the batch.  Work per point or
// per group is a thread or a warp.  Buffers are sized from upper bounds and
// the host reads the counts once, when the set-up has completed.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

#include "internal.h"

namespace npme {
namespace {

constexpr int kSourceSplit = 2;  // fine source columns per coarse column edge
constexpr long kHostBoxPoints = 1L << 15;  // below: bounding box on the host

// Order-preserving 64-bit key of a double (total order of the finite values).
__device__ __forceinline__ unsigned long long dkey(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
inline double dkey_inv(unsigned long long k) {
  const unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  double x;
  std::memcpy(&x, &u, sizeof(x));
  return x;
}

// The bounding box of one system's coordinates, read back by the host.
struct SetupStats {
  unsigned long long mn[3], mx[3];  // dkey of the per-axis minimum / maximum
  unsigned int nonfinite;
};

__global__ void init_stats_kernel(SetupStats *st) {
  for (int d = 0; d < 3; d++) st->mn[d] = ~0ull, st->mx[d] = 0ull;
  st->nonfinite = 0;
}

__global__ void bbox_kernel(const double *__restrict__ coord, long n, SetupStats *st) {
  unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0ull, 0ull, 0ull};
  unsigned bad = 0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double x = coord[3 * i + d];
      if (!isfinite(x)) {
        bad = 1;
        continue;
      }
      const unsigned long long k = dkey(x);
      lo[d] = min(lo[d], k);
      hi[d] = max(hi[d], k);
    }
  }
  const unsigned FULL = 0xffffffffu;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = min(lo[d], __shfl_xor_sync(FULL, lo[d], o));
      hi[d] = max(hi[d], __shfl_xor_sync(FULL, hi[d], o));
    }
    bad |= __shfl_xor_sync(FULL, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    for (int d = 0; d < 3; d++) {
      atomicMin(&st->mn[d], lo[d]);
      atomicMax(&st->mx[d], hi[d]);
    }
    if (bad) atomicOr(&st->nonfinite, 1u);
  }
}

// Geometry the binning kernel needs (host-computed from the box).
struct BinGeom {
  double N[3], L[3], R[3];
  long Nl[3], H[3], nb[3];
  int P, TL, nkeys;
  // direct-sum columns
  double mn[2], edge[2], sedge[2];
  int nc[2], ns[2];
  // quantised z: floor((z - zmin) * zscale) in [0, 2^zbits)
  double zmin, zscale;
  int zbits;
};

// z quantised to zbits bits (a quantum of at most 1/1024 of the column edge),
// non-decreasing in z.  The direct sum's two point orders sort by (column,
// quantised z, index); the source segments are searched with the same
// quantisation, widened to whole quanta, so a segment is a superset of the
// sources within reach (the pair test rejects the few extra) and no pair is
// lost.
__device__ __forceinline__ unsigned zquant(double z, double zmin, double zscale, int zbits) {
  const double t = __dmul_rn(__dsub_rn(z, zmin), zscale);
  if (!(t > 0.0)) return 0u;
  const double mx = (double)((1u << zbits) - 1u);
  return (unsigned)floor(fmin(t, mx));
}

// start index of the B-spline stencil (src/RecSumSupportFunctions.h:123-127)
__device__ __forceinline__ long stencil_start(double w) {
  return w < 0 ? (long)(-w) + 1 : (long)(-w);
}

struct GroupGeom {
  double R, R2;
  double mn[2], sedge[2];
  int ns[2], nc1;
  double zmin, zscale;  // the z quantisation of the sort keys
  int zbits;
};

// One system of a set-up batch: its geometry and sizes, where its elements
// start in the batch's concatenated scratch arrays, and its handle's output
// buffers.  Index spaces of the batch: points (p_off), brick slots (b_off,
// nbt + 1 per system: the bricks and an empty end slot), coarse and fine
// column slots (c_off, s_off: columns and an end slot), group slots (g_off,
// ngb per system: an upper bound of its groups).  Every sort key of the
// batch starts with the system's index, so a system's elements stay
// contiguous and in their own order through every sort.
struct SysDesc {
  BinGeom g;
  GroupGeom gg;
  long n, nbt, ncol, nscol, ngb;
  long wmax;         // segments of a group at most: the stride of its list
  bool full;         // the one-sided walk's lists are wanted too
  bool zones;        // the half shell's segments are cut into zones
  long p_off, b_off, c_off, s_off, g_off;
  const double *coord;
  void *bpts;        // BrickPoint<T>[n]
  int *brick_start;  // [nbt + 1]
  int *brick_list;   // [min(n, nbt)]
  int *odd_list;     // [min(n, nbt)]
  uint32_t *cperm, *sperm, *bperm;
  double4 *gpos, *spos;
  int2 *segs, *hsegs;
  int4 *groups, *hgroups;
  int2 *hzones;
  double4 *gcen, *hcen;
};

// Per system, accumulated on the device.
constexpr int kWorkBins = 1024;
struct SysStats {
  long long bad;                   // lowest index whose stencil leaves the octant
  unsigned long long cand, hcand;  // staged (target, source) candidates, both walks
  int nodd, must;                  // odd bricks, whether some have to go by themselves
  // groups per work bin and the places handed out in each, full and half lists
  int bins[2][kWorkBins], taken[2][kWorkBins];
};

// The counts the host reads once the set-up has completed.
struct SetupCounts {
  long long bad;
  unsigned long long cand, hcand;
  int ngroups, nnonempty, nodd, must;
};

constexpr int kMaxZBits = 20;  // bits of the quantised z at most

// The system owning element x of an index space with starts off[0..R).
__device__ __forceinline__ int owner(const long *__restrict__ off, int R, long x) {
  int lo = 0, hi = R - 1;
  while (lo < hi) {
    const int m = (lo + hi + 1) >> 1;
    if (off[m] <= x) lo = m;
    else hi = m - 1;
  }
  return lo;
}

// one CTA per system
__global__ void init_sys_stats_kernel(const SysDesc *__restrict__ d, SysStats *st) {
  SysStats &S = st[blockIdx.x];
  if (threadIdx.x == 0) {
    S.bad = d[blockIdx.x].n;
    S.cand = S.hcand = 0;
    S.nodd = S.must = 0;
  }
  for (int i = threadIdx.x; i < 2 * kWorkBins; i += blockDim.x)
    S.bins[i / kWorkBins][i % kWorkBins] = S.taken[i / kWorkBins][i % kWorkBins] = 0;
}

// Per point: the spread/interpolation record, its brick-and-bank sort key,
// its (coarse column, quantised z) and (fine column, quantised z) sort keys (z
// in the low zf bits).  Arithmetic as the host restatement
// of the reference (explicit round-to-nearest operations, no contraction),
// so that every point lands in the same brick, bank and column on any
// machine.
template <typename T>
__global__ void bin_kernel(const SysDesc *__restrict__ d, const long *__restrict__ poff, int R,
                           long P, int bbits, int cbits, int sbits, int zf,
                           BrickPoint<T> *__restrict__ pts, unsigned long long *__restrict__ bkey,
                           unsigned long long *__restrict__ ckey,
                           unsigned long long *__restrict__ skey, unsigned *__restrict__ iota,
                           SysStats *st) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  const int r = owner(poff, R, p);
  const SysDesc &D = d[r];
  const BinGeom &g = D.g;
  const long i = p - D.p_off;
  const double x[3] = {D.coord[3 * i], D.coord[3 * i + 1], D.coord[3 * i + 2]};
  long o[3];
  T u[3];
  bool out = false;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double w = __dmul_rn(__ddiv_rn(g.N[a], g.L[a]), __dsub_rn(x[a], g.R[a]));
    const long ms = stencil_start(w);
    o[a] = ms + g.Nl[a] / 4;
    if (o[a] < 0 || o[a] + g.P - 1 > g.H[a] - 1) out = true;
    u[a] = (T)__dadd_rn(w, (double)ms);
  }
  if (out) {
    atomicMin(&st[r].bad, (long long)i);
    o[0] = o[1] = o[2] = 0;  // any in-range brick: the set-up fails anyway
  }
  const long b1 = o[0] / kBrick, b2 = o[1] / kBrick, b3 = o[2] / kBrick;
  const long bid = (b1 * g.nb[1] + b2) * g.nb[2] + b3;
  const long l1 = o[0] - b1 * kBrick, l2 = o[1] - b2 * kBrick, l3 = o[2] - b3 * kBrick;
  const unsigned key = (unsigned)(((l1 * g.TL + l2) * g.TL + l3) % g.nkeys);
  BrickPoint<T> bp;
  bp.u[0] = u[0], bp.u[1] = u[1], bp.u[2] = u[2];
  bp.g0 = ((uint32_t)o[0] << 20) | ((uint32_t)o[1] << 10) | (uint32_t)o[2];
  bp.orig = (uint32_t)i;
  pts[p] = bp;
  bkey[p] = ((unsigned long long)r << (bbits + 5)) | ((unsigned long long)bid << 5) | key;
  int cs[2], ss[2];
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const double v = __dsub_rn(x[a], g.mn[a]);
    cs[a] = min(g.nc[a] - 1, max(0, (int)__ddiv_rn(v, g.edge[a])));
    const double rr = __dsub_rn(v, __dmul_rn((double)cs[a], g.edge[a]));
    ss[a] = cs[a] * kSourceSplit + min(kSourceSplit - 1, max(0, (int)__ddiv_rn(rr, g.sedge[a])));
  }
  const unsigned long long cc = (unsigned long long)(cs[0] * g.nc[1] + cs[1]);
  const unsigned long long sc = (unsigned long long)(ss[0] * g.ns[1] + ss[1]);
  const unsigned long long zq = zquant(x[2], g.zmin, g.zscale, g.zbits);
  ckey[p] = ((unsigned long long)r << (cbits + zf)) | (cc << zf) | zq;
  skey[p] = ((unsigned long long)r << (sbits + zf)) | (sc << zf) | zq;
  iota[p] = (unsigned)p;
}

// Where every brick, coarse column and fine column of the batch begins in its
// sorted keys (one thread per slot, binary search), and P past the last: the
// counts are differences of neighbours.  The slot after a system's last brick
// or column is where the next system begins.  (Counting with atomics in the
// binning took three quarters of it: a few hundred columns share all points.)
__global__ void starts_kernel(const SysDesc *__restrict__ d, int R,
                              const long *__restrict__ boff, const long *__restrict__ coff,
                              const long *__restrict__ soff, long P, long B, long C, long S,
                              int bbits, int cbits, int sbits, int zf,
                              const unsigned long long *__restrict__ bkey,
                              const unsigned long long *__restrict__ ckey,
                              const unsigned long long *__restrict__ skey,
                              int *__restrict__ bstart, int *__restrict__ cstart,
                              int *__restrict__ sstart) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long *key = bkey;
  int *out = bstart;
  long last = B;
  const long *off = boff;
  int idbits = bbits, low = 5;
  if (t > B) {
    t -= B + 1, key = ckey, out = cstart, last = C, off = coff, idbits = cbits, low = zf;
    if (t > C) t -= C + 1, key = skey, out = sstart, last = S, off = soff, idbits = sbits;
  }
  if (t > last) return;
  if (t == last) {
    out[t] = (int)P;
    return;
  }
  const int r = owner(off, R, t);
  const unsigned long long want = (((unsigned long long)r << idbits) + (t - off[r])) << low;
  long lo = 0, hi = P;
  while (lo < hi) {
    const long m = (lo + hi) >> 1;
    if (key[m] < want) lo = m + 1;
    else hi = m;
  }
  out[t] = (int)lo;
}

// What the two scans of a set-up add up: non-empty bricks (CTA 0) and groups
// per coarse column (CTA 1).
struct NonEmpty {
  const int *start;
  __host__ __device__ int operator()(int i) const { return start[i + 1] > start[i]; }
};
struct GroupsOf {
  const int *start;
  __host__ __device__ int operator()(int i) const { return (start[i + 1] - start[i] + 31) / 32; }
};

// Both exclusive sums in one launch, a CTA each, for up to kOneScan elements.
constexpr long kOneScan = 1L << 16;
__global__ void __launch_bounds__(1024) scans_kernel(const int *__restrict__ bstart, int B,
                                                     int *__restrict__ pos,
                                                     const int *__restrict__ cstart, int C,
                                                     int *__restrict__ goff) {
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool first = blockIdx.x == 0;
  const int n = first ? B : C;
  int *out = first ? pos : goff;
  // consecutive elements per thread: one pass of loads, one CTA-wide scan
  const int per = (n + 1023) / 1024, i0 = threadIdx.x * per, i1 = min(n, i0 + per);
  int sum = 0;
  for (int i = i0; i < i1; i++) sum += first ? NonEmpty{bstart}(i) : GroupsOf{cstart}(i);
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) warp_sum[w] = inc;
  __syncthreads();
  if (w == 0) {
    int v = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    warp_sum[lane] = v;
  }
  __syncthreads();
  int run = inc - sum + (w > 0 ? warp_sum[w - 1] : 0);
  for (int i = i0; i < i1; i++) {
    out[i] = run;
    run += first ? NonEmpty{bstart}(i) : GroupsOf{cstart}(i);
  }
}

template <class F>
__global__ void values_kernel(F f, long n, int *__restrict__ out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = f((int)i);
}

// Brick order inside each brick in rounds over the banks: round r holds the
// r-th point (in index order) of every bank with more than r points, banks
// ascending, i.e. the order of a stable sort by (system, brick, rank inside
// the bank, bank).  Input: the point indices sorted by (system, brick, bank)
// and those keys; one warp per brick slot, lane b owns bank b (keys carry the
// bank in their low 5 bits), whose run is found where the bank changes.
constexpr int kPlaceWarps = 8;
__global__ void __launch_bounds__(32 * kPlaceWarps)
    round_place_kernel(const unsigned long long *__restrict__ key,
                       const unsigned *__restrict__ in, const int *__restrict__ bstart, long B,
                       unsigned *__restrict__ out) {
  __shared__ int run[kPlaceWarps][33];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long b = (long)blockIdx.x * kPlaceWarps + w;
  if (b >= B) return;  // warp-uniform
  const int s = bstart[b], c = bstart[b + 1] - s;
  if (c == 0) return;
  // run[v]: first position whose bank is >= v
  for (int i = lane; i <= c; i += 32) {
    const int prev = i > 0 ? (int)(key[s + i - 1] & 31ull) : -1;
    const int cur = i < c ? (int)(key[s + i] & 31ull) : 32;
    for (int v = prev + 1; v <= cur; v++) run[w][v] = s + i;
  }
  __syncwarp();
  const int lo = run[w][lane], cnt = run[w][lane + 1] - lo;
  int rounds = cnt;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rounds = max(rounds, __shfl_xor_sync(0xffffffffu, rounds, o));
  const unsigned below = (1u << lane) - 1u;
  int base = s;
#pragma unroll 4
  for (int r = 0; r < rounds; r++) {
    const unsigned m = __ballot_sync(0xffffffffu, cnt > r);
    if (cnt > r) out[base + __popc(m & below)] = in[lo + r];
    base += __popc(m);
  }
}

// Final brick order of every system: its records, the brick-order
// permutation, and each point's brick-order position (the slot of its
// source-side direct-sum sums); and every system's brick starts (local
// positions) and non-empty brick list.
template <typename T>
__global__ void place_bricks_kernel(const SysDesc *__restrict__ d, const long *__restrict__ poff,
                                    const long *__restrict__ boff, int R, long P, long B,
                                    const unsigned *__restrict__ order,
                                    const BrickPoint<T> *__restrict__ pts,
                                    const int *__restrict__ start, const int *__restrict__ pos,
                                    unsigned *__restrict__ bpos) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < P) {
    const int r = owner(poff, R, k);
    const SysDesc &D = d[r];
    const long p = order[k], kl = k - D.p_off;
    reinterpret_cast<BrickPoint<T> *>(D.bpts)[kl] = pts[p];
    D.bperm[kl] = (uint32_t)(p - D.p_off);
    bpos[p] = (unsigned)kl;
  }
  if (k < B) {
    const int r = owner(boff, R, k);
    const SysDesc &D = d[r];
    const long b = k - D.b_off;  // 0 .. nbt (end slot)
    D.brick_start[b] = start[k] - start[D.b_off];
    if (b < D.nbt && start[k + 1] > start[k]) D.brick_list[pos[k] - pos[D.b_off]] = (int)b;
  }
}

// The direct sum's two orders of every system: local permutations, FP64
// positions (a source's w holds its brick-order position) and each point's
// position in the target (group) order.  CTAs from nblocks on: the odd bricks, a warp
// per brick slot, by the points of their fullest plane (one stencil start along x, of
// eight): more than 256, where the error of FP32 sums by one warp shows (must), or
// more than 96 and a third of the brick's, where the time of one warp does.  (Here
// beside the orders they cost set-up nothing; in round_place_kernel, whose latency
// they lengthen, 8 us.)
template <typename T>
__global__ void __launch_bounds__(256)
    place_orders_kernel(const SysDesc *__restrict__ d, const long *__restrict__ poff, int R, long P,
                        const unsigned *__restrict__ corder, const unsigned *__restrict__ sorder,
                        const unsigned *__restrict__ bpos, unsigned *__restrict__ cpos,
                        unsigned nblocks, const long *__restrict__ boff, long B,
                        const int *__restrict__ start, const int *__restrict__ pos, SysStats *st) {
  if (blockIdx.x >= nblocks) {
    const long b = (long)(blockIdx.x - nblocks) * 8 + (threadIdx.x >> 5);
    if (b >= B) return;  // warp-uniform
    const int c = start[b + 1] - start[b], lane = threadIdx.x & 31;
    if (c <= 96) return;
    const int r = owner(boff, R, b);
    const SysDesc &D = d[r];
    const BrickPoint<T> *pts =
        static_cast<const BrickPoint<T> *>(D.bpts) + (start[b] - start[D.b_off]);
    int mine = 0;  // lane p < 8: points of plane p
    for (int i = lane; i - lane < c; i += 32) {
      const int p = i < c ? (int)(pts[i].g0 >> 20) & (kBrick - 1) : -1;
#pragma unroll
      for (int v = 0; v < kBrick; v++) {
        const unsigned m = __ballot_sync(0xffffffffu, p == v);
        if (lane == v) mine += __popc(m);
      }
    }
    const int most = __reduce_max_sync(0xffffffffu, mine);
    if (lane == 0 && most > min(256, max(96, c / 3))) {
      D.brick_list[pos[b] - pos[D.b_off]] = (int)(b - D.b_off) | (int)0x80000000;
      D.odd_list[atomicAdd(&st[r].nodd, 1)] = (int)(b - D.b_off);
      if (most > 256) st[r].must = 1;
    }
    return;
  }
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P) return;
  const int r = owner(poff, R, k);
  const SysDesc &D = d[r];
  const long kl = k - D.p_off;
  const long pc = corder[k], ic = pc - D.p_off;
  D.cperm[kl] = (uint32_t)ic;
  cpos[pc] = (unsigned)k;
  const double *x = D.coord + 3 * ic;
  D.gpos[kl] = make_double4(x[0], x[1], x[2], 0.0);
  const long ps = sorder[k], is = ps - D.p_off;
  D.sperm[kl] = (uint32_t)is;
  const double *y = D.coord + 3 * is;
  D.spos[kl] = make_double4(y[0], y[1], y[2], (double)bpos[ps]);
}

// the number of groups of system D (on the device)
__device__ __forceinline__ long sys_groups(const SysDesc &D, const int *__restrict__ goff) {
  return goff[D.c_off + D.ncol] - goff[D.c_off];
}

// first index in [a, b) with f(index) >= x
template <class F>
__device__ __forceinline__ int lower_idx(const F &f, int a, int b, unsigned x) {
  while (a < b) {
    const int m = (a + b) >> 1;
    if (f(m) < x) a = m + 1;
    else b = m;
  }
  return a;
}

// Bin of a group's work (staged sources): 32 bins per power of two, the
// heaviest first.
__device__ __forceinline__ int work_bin(unsigned long long work) {
  const unsigned u = __float_as_uint((float)min(work, 0x7fffffffull)) >> 18;  // 5 mantissa bits
  const unsigned one = 0x3f800000u >> 18;                                     // bin of 1
  return kWorkBins - 1 - (int)min(u > one ? u - one : 0u, (unsigned)kWorkBins - 1);
}

// One warp per group slot: the group's points (a run of 32 of one coarse
// column of the batch's target order), its bounding box and frame origin, and
// its source segments (lanes over the fine columns of the group's window in
// (s0, s1) order, so that a group's segments come in the same order as a
// sequential sweep).  A fine column contributes the z range of its sources
// within Rdir of the group's box: |dz| <= sqrt(Rdir^2 - d_xy^2), d_xy the xy
// distance from the box to the column; the half shell keeps the fine columns of
// later coarse columns and, in the group's own coarse column, the sources after
// the group in the group order.  The half shell's ranges are cut into three
// zones: within reach of both halves of the group (its targets are in z order),
// of the lower or of the upper half only; the walks spend half the steps on the
// last two.  Positions are the batch's (cstart, sstart); the written segments
// and group records are the system's own (local).  A group's segments start at
// its number times a bound of their count, so that no pass over all groups has
// to count them first.
__global__ void __launch_bounds__(256)
    groups_kernel(const SysDesc *__restrict__ d, const long *__restrict__ goffs, int R, long G,
                  const int *__restrict__ goff, const int *__restrict__ cstart,
                  const int *__restrict__ sstart, const unsigned long long *__restrict__ skey,
                  int zf, const unsigned *__restrict__ sorder,
                  const unsigned *__restrict__ cpos, int4 *__restrict__ ug,
                  int4 *__restrict__ uh, int2 *__restrict__ uz,
                  double4 *__restrict__ cen, int *__restrict__ bin,
                  int *__restrict__ hbin, SysStats *st) {
  const long slot = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (slot >= G) return;  // warp-uniform
  const int r = owner(goffs, R, slot);
  const SysDesc &D = d[r];
  const int gi = (int)(slot - D.g_off);
  if (gi >= sys_groups(D, goff)) return;  // a spare slot of the bound
  const GroupGeom &gg = D.gg;
  const unsigned FULL = 0xffffffffu;
  const unsigned zmask = (unsigned)((1ull << zf) - 1ull);
  // the coarse column: the last with at most gi groups before it
  int c, p0, p1;
  {
    const int *go = goff + D.c_off;
    const int want = go[0] + gi;
    int a = 0, b = (int)D.ncol;  // first column in (a, b] with more than gi groups before it
    while (a < b) {
      const int m = (a + b + 1) >> 1;
      if (go[m] <= want) a = m;
      else b = m - 1;
    }
    c = a;
    p0 = cstart[D.c_off + c] + 32 * (want - go[c]);
    p1 = min(p0 + 32, cstart[D.c_off + c + 1]);
  }
  const int pl = (int)D.p_off;  // batch position -> system position
  double l[3] = {1e300, 1e300, 1e300}, h[3] = {-1e300, -1e300, -1e300};
  if (p0 + lane < p1) {
    const double4 p = D.gpos[p0 + lane - pl];
    l[0] = h[0] = p.x, l[1] = h[1] = p.y, l[2] = h[2] = p.z;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < 3; a++) {
      l[a] = fmin(l[a], __shfl_xor_sync(FULL, l[a], o));
      h[a] = fmax(h[a], __shfl_xor_sync(FULL, h[a], o));
    }
  if (lane == 0) {
    const double dx = __dsub_rn(h[0], l[0]), dy = __dsub_rn(h[1], l[1]),
                 dz = __dsub_rn(h[2], l[2]);
    cen[slot] = make_double4(
        __dmul_rn(0.5, __dadd_rn(l[0], h[0])), __dmul_rn(0.5, __dadd_rn(l[1], h[1])),
        __dmul_rn(0.5, __dadd_rn(l[2], h[2])),
        __dmul_rn(0.5, __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                                            __dmul_rn(dz, dz)))));
  }
  int lo[2], hi[2];
#pragma unroll
  for (int a = 0; a < 2; a++) {
    // one column of margin on each side: the distance test below decides
    lo[a] = max(0, (int)floor((l[a] - gg.R - gg.mn[a]) / gg.sedge[a]) - 1);
    hi[a] = min(gg.ns[a] - 1, (int)floor((h[a] + gg.R - gg.mn[a]) / gg.sedge[a]) + 1);
  }
  const int w1 = hi[1] - lo[1] + 1;
  const int nwin = (hi[0] - lo[0] + 1) * w1;
  // z extents of the group's halves (targets 0-15 and 16-31)
  double zl = l[2], zh = h[2], hl[2], hh[2];
  {
    double a = 1e300, b = -1e300;
    if (p0 + lane < p1) a = b = D.gpos[p0 + lane - pl].z;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      a = fmin(a, __shfl_xor_sync(FULL, a, o));
      b = fmax(b, __shfl_xor_sync(FULL, b, o));
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
      hl[i] = __shfl_sync(FULL, a, 16 * i), hh[i] = __shfl_sync(FULL, b, 16 * i);
  }
  const int cl = min(16, p1 - p0), cu = p1 - p0 - cl;  // targets of the halves
  const long stride = D.zones ? 3 * D.wmax : D.wmax;
  const int base = (int)(gi * stride);
  auto zq = [&](int i) { return (unsigned)skey[i] & zmask; };
  auto zquantum = [&](double z) { return zquant(z, gg.zmin, gg.zscale, gg.zbits); };
  // Window column t: [a, b) the sources within reach of the group (one-sided
  // walk); of those in the half shell, [u[0], v[0]) within reach of both
  // halves, [u[1], v[1]) of the lower and [u[2], v[2]) of the upper one only
  // (whole quanta: every source within reach is inside).
  auto column = [&](int t, int &a, int &b, int (&u)[3], int (&v)[3]) {
    a = b = 0;
#pragma unroll
    for (int i = 0; i < 3; i++) u[i] = v[i] = 0;
    if (t >= nwin) return;
    const int s0 = lo[0] + t / w1, s1 = lo[1] + t % w1;
    const long sc = D.s_off + (long)s0 * gg.ns[1] + s1;
    const int zb = sstart[sc], ze = sstart[sc + 1];
    if (ze <= zb) return;
    const double l0 = __dadd_rn(gg.mn[0], __dmul_rn((double)s0, gg.sedge[0]));
    const double h0 = __dadd_rn(l0, gg.sedge[0]);
    const double l1 = __dadd_rn(gg.mn[1], __dmul_rn((double)s1, gg.sedge[1]));
    const double h1 = __dadd_rn(l1, gg.sedge[1]);
    const double dx = fmax(0.0, fmax(__dsub_rn(l0, h[0]), __dsub_rn(l[0], h0)));
    const double dy = fmax(0.0, fmax(__dsub_rn(l1, h[1]), __dsub_rn(l[1], h1)));
    const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    if (d2 > gg.R2) return;
    const double hz = __dsqrt_rn(__dsub_rn(gg.R2, d2));
    a = lower_idx(zq, zb, ze, zquantum(__dsub_rn(zl, hz)));
    b = lower_idx(zq, a, ze, zquantum(__dadd_rn(zh, hz)) + 1u);
    const long cc = (long)(s0 / kSourceSplit) * gg.nc1 + s1 / kSourceSplit;
    if (b <= a || cc < c) return;
    const int a2 =
        cc == c ? lower_idx([&](int i) { return cpos[sorder[i]]; }, a, b, (unsigned)p1) : a;
    if (a2 >= b) return;
    if (!D.zones) {
      u[0] = a2, v[0] = b;
      return;
    }
    if (cu == 0) {
      u[1] = a2, v[1] = b;
      return;
    }
    // the halves are in z order: the lower reaches [a2, e), the upper [f, b)
    const int e = lower_idx(zq, a2, b, zquantum(__dadd_rn(hh[0], hz)) + 1u);
    const int f = lower_idx(zq, a2, b, zquantum(__dsub_rn(hl[1], hz)));
    u[0] = f, v[0] = max(e, f);
    u[1] = a2, v[1] = min(e, f);
    u[2] = max(e, f), v[2] = b;
  };
  // segments of every zone, then their places: both halves, lower, upper
  int n[3] = {0, 0, 0}, nf = 0;
  unsigned long long src[4] = {0, 0, 0, 0};  // sources per zone; one-sided walk
  for (int t0 = 0; t0 < nwin; t0 += 32) {
    int a, b, u[3], v[3];
    column(t0 + lane, a, b, u, v);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      n[i] += __popc(__ballot_sync(FULL, v[i] > u[i]));
      src[i] += (unsigned)max(0, v[i] - u[i]);
    }
    src[3] += (unsigned)(b - a);
  }
  int at[3] = {base, base + n[0], base + n[0] + n[1]};
  for (int t0 = 0; t0 < nwin; t0 += 32) {
    int a, b, u[3], v[3];
    column(t0 + lane, a, b, u, v);
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const unsigned m = __ballot_sync(FULL, v[i] > u[i]);
      if (v[i] > u[i]) D.hsegs[at[i] + __popc(m & below)] = make_int2(u[i] - pl, v[i] - u[i]);
      at[i] += __popc(m);
    }
    if (D.full) {
      const unsigned m = __ballot_sync(FULL, b > a);
      if (b > a) D.segs[gi * D.wmax + nf + __popc(m & below)] = make_int2(a - pl, b - a);
      nf += __popc(m);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < 4; i++) src[i] += __shfl_xor_sync(FULL, src[i], o);
  if (lane == 0) {
    uh[slot] = make_int4(p0 - pl, p1 - p0, base, base + n[0] + n[1] + n[2]);
    uz[slot] = make_int2(base + n[0], base + n[0] + n[1]);
    const int hb = work_bin(2 * src[0] + src[1] + src[2]);
    hbin[slot] = hb;
    atomicAdd(&st[r].bins[1][hb], 1);
    if (D.full) {
      ug[slot] = make_int4(p0 - pl, p1 - p0, (int)(gi * D.wmax), (int)(gi * D.wmax) + nf);
      const int fb = work_bin(src[3]);
      bin[slot] = fb;
      atomicAdd(&st[r].bins[0][fb], 1);
    }
    atomicAdd(&st[r].cand, src[3] * (unsigned long long)(p1 - p0));
    atomicAdd(&st[r].hcand, src[0] * (unsigned long long)(p1 - p0) +
                                src[1] * (unsigned long long)cl + src[2] * (unsigned long long)cu);
  }
}

// A system's final group records and frame origins, heaviest bin first (the
// order inside a bin is that of the atomics: it decides only which warp walks
// a group, no result), so that the last wave of a direct-sum launch holds the
// light ones.  Grid: (CTAs of 256 slots of the longest system, systems, lists).
__global__ void __launch_bounds__(256)
    order_groups_kernel(const SysDesc *__restrict__ d, const int *__restrict__ goff,
                        const int4 *__restrict__ ug, const int4 *__restrict__ uh,
                        const int2 *__restrict__ uz, const double4 *__restrict__ cen,
                        const int *__restrict__ bin,
                        const int *__restrict__ hbin, SysStats *st) {
  __shared__ int first[kWorkBins];
  __shared__ int warp_sum[8];
  const SysDesc &D = d[blockIdx.y];
  SysStats &S = st[blockIdx.y];
  const bool half = blockIdx.z == 0;
  if (!half && !D.full) return;
  const long n = sys_groups(D, goff), g0 = (long)blockIdx.x * 256;
  if (g0 >= n) return;
  // exclusive sum of the bins, four per thread
  constexpr int K = kWorkBins / 256;
  const int *bins = S.bins[half ? 1 : 0];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int v[K], sum = 0;
#pragma unroll
  for (int i = 0; i < K; i++) v[i] = bins[K * threadIdx.x + i], sum += v[i];
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) warp_sum[w] = inc;
  __syncthreads();
  int run = inc - sum;
  for (int i = 0; i < w; i++) run += warp_sum[i];
#pragma unroll
  for (int i = 0; i < K; i++) first[K * threadIdx.x + i] = run, run += v[i];
  __syncthreads();
  const long k = g0 + threadIdx.x;
  if (k >= n) return;
  const long s = D.g_off + k;
  const int b = (half ? hbin : bin)[s];
  const int dest = first[b] + atomicAdd(&S.taken[half ? 1 : 0][b], 1);
  (half ? D.hgroups : D.groups)[dest] = (half ? uh : ug)[s];
  if (half) D.hzones[dest] = uz[s];
  (half ? D.hcen : D.gcen)[dest] = cen[s];
}

__global__ void collect_counts_kernel(const SysDesc *__restrict__ d, int R,
                                      const SysStats *__restrict__ st,
                                      const int *__restrict__ goff, const int *__restrict__ pos,
                                      SetupCounts *__restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  const SysDesc &D = d[r];
  out[r].bad = st[r].bad;
  out[r].cand = st[r].cand;
  out[r].hcand = st[r].hcand;
  out[r].nodd = st[r].nodd;
  out[r].must = st[r].must;
  out[r].ngroups = (int)sys_groups(D, goff);
  out[r].nnonempty = pos[D.b_off + D.nbt] - pos[D.b_off];
}

int bits_for(unsigned long long v) {  // bits to hold values < v
  int b = 1;
  while (b < 64 && (1ull << b) < v) b++;
  return b;
}

inline unsigned blocks_for(long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// Scratch buffers of the set-up, kept by the handle that owns a batch (the
// first) and reused by its next set-up.
enum Scratch {
  kPts, kBKey, kBKeyOut, kIota, kBPerm, kCKey, kSKey, kKeyOut, kCOrder, kSOrder, kBOrder,
  kBStart, kValues, kPos, kCStart, kSStart, kCPos, kGOff, kCen, kBins, kUGroups, kUHGroups,
  kUZones,
  kStats, kSysStats, kDesc, kOffs, kCub, kBPos, kCountsDev, kScratchCount
};
static_assert(kScratchCount <= kSetupScratch, "raise kSetupScratch");

#define SCK(call)                                                                         \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return record_error(h, NPME_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

template <typename P>
int scratch(npme_handle *h, Scratch i, size_t bytes, P **out) {
  const int rc = handle_buffer(h, &h->d_su[i], std::max<size_t>(bytes, 16));
  *out = (P *)h->d_su[i];
  return rc;
}

// CUB temporary storage of at least `bytes`
int cub_tmp(npme_handle *h, size_t bytes, void **out) {
  return scratch(h, kCub, std::max<size_t>(bytes, 256), out);
}

// stable radix sort of (key, value) pairs on bits [0, end_bit), ascending
template <typename K>
int sort_pairs(npme_handle *h, const K *kin, K *kout, const unsigned *vin, unsigned *vout,
               long n, int end_bit, cudaStream_t s) {
  size_t tb = 0;
  SCK(cub::DeviceRadixSort::SortPairs(nullptr, tb, kin, kout, vin, vout, (int)n, 0, end_bit, s));
  void *tmp;
  int rc;
  if ((rc = cub_tmp(h, tb, &tmp))) return rc;
  SCK(cub::DeviceRadixSort::SortPairs(tmp, tb, kin, kout, vin, vout, (int)n, 0, end_bit, s));
  return NPME_OK;
}

int exclusive_sum(npme_handle *h, const int *in, int *out, long n, cudaStream_t s) {
  size_t tb = 0;
  SCK(cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, (int)n, s));
  void *tmp;
  int rc;
  if ((rc = cub_tmp(h, tb, &tmp))) return rc;
  SCK(cub::DeviceScan::ExclusiveSum(tmp, tb, in, out, (int)n, s));
  return NPME_OK;
}

// Host side of one system: its binning geometry (and the handle's refine2),
// its sizes and its output buffers.
template <typename T>
int describe(npme_handle *h, SysDesc &D) {
  const long n = (long)h->n;
  const GridGeom &gr = h->grid;
  const double *R = h->box + 3, *L = h->box + 6;
  int rc;
  BinGeom &g = D.g;
  for (int a = 0; a < 3; a++) {
    g.N[a] = (double)gr.N[a], g.L[a] = L[a], g.R[a] = R[a];
    g.Nl[a] = gr.N[a], g.H[a] = gr.H[a], g.nb[a] = gr.nb[a];
  }
  g.P = gr.order;
  g.TL = kBrick + gr.order - 1;
  g.nkeys = 32 / ((int)(sizeof(T) / 4) * (h->complex_kernel ? 2 : 1));
  // direct-sum columns: edge e ~ (32 / density)^(1/3) over the bounding box
  // (degenerate axes are given a nominal thickness of Rdir / 4)
  const double Rd = h->p.Rdir;
  double vol = 1.0;
  for (int a = 0; a < 3; a++) vol *= std::max(h->bmax[a] - h->bmin[a], 0.25 * Rd);
  double e = std::cbrt(32.0 * vol / (double)n);
  e = std::max(e, 1e-3 * Rd);
  for (int a = 0; a < 2; a++) {
    const double ext = h->bmax[a] - h->bmin[a];
    g.nc[a] = std::max(1, std::min((int)std::ceil(ext / e), 1 << 14));
    g.edge[a] = std::max(ext / g.nc[a], 1e-12);
    g.ns[a] = g.nc[a] * kSourceSplit;
    g.sedge[a] = g.edge[a] / kSourceSplit;
    g.mn[a] = h->bmin[a];
  }
  {
    const double H = h->bmax[2] - h->bmin[2];
    g.zbits = std::max(8, std::min(kMaxZBits,
                                   (int)std::ceil(std::log2(std::max(1.0, 1024.0 * H / e)))));
    g.zmin = h->bmin[2];
    g.zscale = (double)((1u << g.zbits) - 1u) / std::max(H, 1e-300);
  }
  GroupGeom &gg = D.gg;
  gg.R = Rd, gg.R2 = Rd * Rd;
  for (int a = 0; a < 2; a++) gg.mn[a] = g.mn[a], gg.sedge[a] = g.sedge[a], gg.ns[a] = g.ns[a];
  gg.nc1 = g.nc[1];
  gg.zmin = g.zmin, gg.zscale = g.zscale, gg.zbits = g.zbits;
  // heads of offsets up to ~the group half-diagonal carry ~6e-8 e absolute
  // error; below r = e/4 the relative error would exceed ~1e-6, so refine
  h->refine2 = (0.25 * e) * (0.25 * e);
  D.n = n;
  D.nbt = gr.nb[0] * gr.nb[1] * gr.nb[2];
  D.ncol = (long)g.nc[0] * g.nc[1];
  D.nscol = (long)g.ns[0] * g.ns[1];
  h->n_bricks = D.nbt;
  // Upper bounds (the kernels read the actual counts on the device; the
  // host reads them once the set-up has completed):
  //   groups   <= n / 32 + non-empty columns <= n / 32 + min(n, ncol)
  //   segments <= groups x the fine columns that can be within Rdir of a group: it
  //               lies in one coarse column, so at most (edge + 2 Rdir) / sedge + 2
  //               per axis (the window's margin columns are not), two more for
  //               rounding
  //   non-empty bricks <= min(n, nbt)
  D.ngb = n / 32 + std::min(n, D.ncol) + 1;
  long wmax = 1;
  for (int a = 0; a < 2; a++)
    wmax *= std::min<long>(g.ns[a], (long)std::floor((g.edge[a] + 2.0 * Rd) / g.sedge[a]) + 4);
  D.wmax = wmax;
  D.full = needs_full_lists(h);
  const long nsb = D.ngb * wmax;
  if (nsb >= (1L << 31))  // int offsets in the group records
    return record_error(h, NPME_EINVAL, "too many direct-sum source segments (2^31)");
  // Zones leave an eighth of the pairs out (at density 1 and Rdir 8 a quarter of
  // the candidates reach one half of a group only) but cost shorter lists.  They
  // gain where a pair is expensive and the lists are long: FP64 1M 6,411 ->
  // 6,131 us, FP64 Helmholtz 62,500 1,088 -> 1,037, FP32 r^-0.5 500k 1,778 ->
  // 1,731, FP32 Helmholtz 250k 1,257 -> 1,239; FP32 1/r 1M 3,121 -> 3,168, and
  // with few groups, whose walks are split, 4,000 points 26 -> 41, 30,000 82 ->
  // 98.  Not for the walks that take all segments alike (one-sided, original Ewald in
  // FP64, caller kernels), nor where three segments per column would exceed the
  // offsets or the memory.
  const long min_points = sizeof(T) == 8 ? 32L * 4 * 148 : 32L * 20 * 148;
  const bool zoned_walk = !D.full && h->p.EwaldSplit == NPME_SPLIT_DERIVMATCH &&
                          (h->p.funcType == NPME_FUNC_RALPHA ||
                           h->p.funcType == NPME_FUNC_HELMHOLTZ ||
                           (sizeof(T) == 8 && h->p.funcType == NPME_FUNC_LAPLACE));
  D.zones = zoned_walk && n >= min_points && 3 * nsb < (1L << 31);
  if (D.zones && handle_buffer(h, (void **)&h->d_hsegs, sizeof(int2) * nsb * 3)) D.zones = false;
  const int C = h->complex_kernel ? 2 : 1;
  if ((rc = handle_buffer(h, &h->d_bpts, sizeof(BrickPoint<T>) * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_brick_start, sizeof(int) * (D.nbt + 1))) ||
      (rc = handle_buffer(h, (void **)&h->d_brick_list,
                          sizeof(int) * std::max<long>(1, std::min(n, D.nbt)))) ||
      (rc = handle_buffer(h, (void **)&h->d_odd_list,
                          sizeof(int) * std::max<long>(1, std::min(n, D.nbt)))) ||
      (rc = handle_buffer(h, (void **)&h->d_cperm, sizeof(uint32_t) * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_sperm, sizeof(uint32_t) * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_bperm, sizeof(uint32_t) * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_gpos, sizeof(double4) * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_spos, sizeof(double4) * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_hsegs, sizeof(int2) * nsb * (D.zones ? 3 : 1))) ||
      (rc = handle_buffer(h, (void **)&h->d_hzones, sizeof(int2) * D.ngb)) ||
      (rc = handle_buffer(h, (void **)&h->d_hgroups, sizeof(int4) * D.ngb)) ||
      (rc = handle_buffer(h, (void **)&h->d_hcen, sizeof(double4) * D.ngb)) ||
      (rc = handle_buffer(h, &h->d_qc, sizeof(T) * C * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_q_in, sizeof(double) * C * n)) ||
      (rc = handle_buffer(h, (void **)&h->d_V, sizeof(double) * 4 * C * n)))
    return rc;
  if (D.full && ((rc = handle_buffer(h, (void **)&h->d_segs, sizeof(int2) * nsb)) ||
                 (rc = handle_buffer(h, (void **)&h->d_groups, sizeof(int4) * D.ngb)) ||
                 (rc = handle_buffer(h, (void **)&h->d_gcen, sizeof(double4) * D.ngb))))
    return rc;
  // source-side sums of the pair-once walk start (and are kept) at zero
  if (h->fp32) {
    if ((rc = handle_buffer(h, (void **)&h->d_vsrc, sizeof(float4) * C * n))) return rc;
    cudaMemsetAsync(h->d_vsrc, 0, sizeof(float4) * C * n, h->stream);
  } else {
    if ((rc = handle_buffer(h, (void **)&h->d_vsrc64, sizeof(double) * 4 * C * n))) return rc;
    cudaMemsetAsync(h->d_vsrc64, 0, sizeof(double) * 4 * C * n, h->stream);
  }
  // grids
  const long *N = gr.N;
  const size_t Ntot = (size_t)N[0] * N[1] * N[2];
  const size_t Mtot = (size_t)(N[0] / 2 + 1) * (N[1] / 2 + 1) * (N[2] / 2 + 1);
  if (h->own_fft) {  // the octant, and half the box of spectrum rows
    const size_t K = h->complex_kernel ? N[2] : N[2] / 2 + 1;
    if ((rc = handle_buffer(h, &h->d_grid, sizeof(T) * C * (Ntot / 8))) ||
        (rc = handle_buffer(h, &h->d_kgrid,
                            sizeof(T) * 2 * (size_t)(N[0] / 2) * N[1] * ((K + 3) & ~size_t(3)))) ||
        (rc = handle_buffer(h, &h->d_G, sizeof(T) * C * Mtot)))
      return rc;
  } else if (h->complex_kernel) {
    if ((rc = handle_buffer(h, &h->d_grid, sizeof(T) * 2 * Ntot)) ||
        (rc = handle_buffer(h, &h->d_G, sizeof(T) * 2 * Mtot)))
      return rc;
  } else {
    if ((rc = handle_buffer(h, &h->d_grid, sizeof(T) * Ntot)) ||
        (rc = handle_buffer(h, &h->d_kgrid, sizeof(T) * 2 * (size_t)N[0] * N[1] * (N[2] / 2 + 1))) ||
        (rc = handle_buffer(h, &h->d_G, sizeof(T) * Mtot)))
      return rc;
  }
  D.coord = h->d_coord;
  D.bpts = h->d_bpts;
  D.brick_start = h->d_brick_start;
  D.brick_list = h->d_brick_list, D.odd_list = h->d_odd_list;
  D.cperm = h->d_cperm, D.sperm = h->d_sperm, D.bperm = h->d_bperm;
  D.gpos = h->d_gpos, D.spos = h->d_spos;
  D.segs = h->d_segs, D.hsegs = h->d_hsegs;
  D.groups = h->d_groups, D.hgroups = h->d_hgroups, D.hzones = h->d_hzones;
  D.gcen = h->d_gcen, D.hcen = h->d_hcen;
  h->d_dperm = h->d_sperm;  // direct-sum charges are gathered into the source order
  return NPME_OK;
}

// Brick order, direct-sum orders, warp groups and segment lists of R systems
// of one precision in one pass on stream s (h0 = hs[0] owns the scratch).
// Enqueued without waiting; the counts arrive in h0->h_counts with the
// caller's synchronisation.  `hook` runs when the systems' buffers are
// allocated and nothing of the geometry is enqueued yet.
template <typename T>
int geometry_batch(npme_handle **hs, int R, cudaStream_t s, const std::function<int()> &hook) {
  npme_handle *h = hs[0];
  int rc;
  std::vector<SysDesc> ds(R);
  long P = 0, B = 0, C = 0, S = 0, G = 0, gmax = 1, nbtmax = 1, ncolmax = 1, nscolmax = 1;
  int zf = 1;
  bool full = false;
  for (int r = 0; r < R; r++) {
    if ((rc = describe<T>(hs[r], ds[r]))) {
      if (hs[r] != h) h->err = hs[r]->err;
      return rc;
    }
    SysDesc &D = ds[r];
    D.p_off = P, D.b_off = B, D.c_off = C, D.s_off = S, D.g_off = G;
    P += D.n, B += D.nbt + 1, C += D.ncol + 1, S += D.nscol + 1, G += D.ngb;
    gmax = std::max(gmax, D.ngb), nbtmax = std::max(nbtmax, D.nbt);
    zf = std::max(zf, D.g.zbits), full = full || D.full;
    ncolmax = std::max(ncolmax, D.ncol), nscolmax = std::max(nscolmax, D.nscol);
    // the system's coordinates and buffers (on its own stream) come first
    if (hs[r]->stream != s) {
      SCK(cudaEventRecord(hs[r]->ev_fork, hs[r]->stream));
      SCK(cudaStreamWaitEvent(s, hs[r]->ev_fork, 0));
    }
  }
  if (hook && (rc = hook())) return rc;
  if (P >= (1L << 31) || B >= (1L << 31) || G >= (1L << 31))
    return record_error(h, NPME_EINVAL, "set-up batch too large for 32-bit indices");
  const int rbits = bits_for((unsigned long long)R);
  const int bbits = bits_for(nbtmax), cbits = bits_for(ncolmax), sbits = bits_for(nscolmax);
  if (rbits + bbits + 5 > 64 || rbits + sbits + zf > 64)
    return record_error(h, NPME_EINVAL, "set-up batch keys exceed 64 bits");

  // descriptors and the index-space starts (points, bricks, columns, fine
  // columns, groups), R each
  SysDesc *dd;
  long *offs;
  if ((rc = scratch(h, kDesc, sizeof(SysDesc) * R, &dd)) ||
      (rc = scratch(h, kOffs, sizeof(long) * 5 * R, &offs)))
    return rc;
  // staged in pinned memory: a copy from pageable memory would first wait
  // for everything enqueued on s
  static_assert(sizeof(SysDesc) % sizeof(long) == 0, "descriptor alignment");
  if ((rc = pinned_block(h, &h->h_desc, &h->desc_cap, (sizeof(SysDesc) + sizeof(long) * 5) * R)))
    return rc;
  SysDesc *hd = static_cast<SysDesc *>(h->h_desc);
  long *ho = reinterpret_cast<long *>(hd + R);
  for (int r = 0; r < R; r++) {
    hd[r] = ds[r];
    ho[r] = ds[r].p_off, ho[R + r] = ds[r].b_off, ho[2 * R + r] = ds[r].c_off;
    ho[3 * R + r] = ds[r].s_off, ho[4 * R + r] = ds[r].g_off;
  }
  SCK(cudaMemcpyAsync(dd, hd, sizeof(SysDesc) * R, cudaMemcpyHostToDevice, s));
  SCK(cudaMemcpyAsync(offs, ho, sizeof(long) * 5 * R, cudaMemcpyHostToDevice, s));
  const long *poff = offs, *boff = offs + R, *coff = offs + 2 * R, *soff = offs + 3 * R,
             *goffs = offs + 4 * R;

  BrickPoint<T> *pts;
  unsigned long long *bkey, *bkey_out, *ckey, *skey, *key_out;
  unsigned *iota, *border, *corder, *sorder, *border2, *bpos, *cpos;
  int *bstart, *pos, *cstart, *sstart, *goff, *bins;
  int4 *ug, *uh;
  int2 *uz;
  double4 *cen;
  SysStats *st;
  if ((rc = scratch(h, kPts, sizeof(BrickPoint<T>) * P, &pts)) ||
      (rc = scratch(h, kBKey, sizeof(unsigned long long) * P, &bkey)) ||
      (rc = scratch(h, kBKeyOut, sizeof(unsigned long long) * P, &bkey_out)) ||
      (rc = scratch(h, kCKey, sizeof(unsigned long long) * P, &ckey)) ||
      (rc = scratch(h, kSKey, sizeof(unsigned long long) * P, &skey)) ||
      (rc = scratch(h, kKeyOut, sizeof(unsigned long long) * P, &key_out)) ||
      (rc = scratch(h, kIota, sizeof(unsigned) * P, &iota)) ||
      (rc = scratch(h, kBPerm, sizeof(unsigned) * P, &border)) ||
      (rc = scratch(h, kBOrder, sizeof(unsigned) * P, &border2)) ||
      (rc = scratch(h, kCOrder, sizeof(unsigned) * P, &corder)) ||
      (rc = scratch(h, kSOrder, sizeof(unsigned) * P, &sorder)) ||
      (rc = scratch(h, kBPos, sizeof(unsigned) * P, &bpos)) ||
      (rc = scratch(h, kCPos, sizeof(unsigned) * P, &cpos)) ||
      (rc = scratch(h, kBStart, sizeof(int) * (B + 1), &bstart)) ||
      (rc = scratch(h, kPos, sizeof(int) * B, &pos)) ||
      (rc = scratch(h, kCStart, sizeof(int) * (C + 1), &cstart)) ||
      (rc = scratch(h, kSStart, sizeof(int) * (S + 1), &sstart)) ||
      (rc = scratch(h, kGOff, sizeof(int) * C, &goff)) ||
      (rc = scratch(h, kCen, sizeof(double4) * G, &cen)) ||
      (rc = scratch(h, kBins, sizeof(int) * 2 * G, &bins)) ||
      (rc = scratch(h, kUGroups, sizeof(int4) * G, &ug)) ||
      (rc = scratch(h, kUHGroups, sizeof(int4) * G, &uh)) ||
      (rc = scratch(h, kUZones, sizeof(int2) * G, &uz)) ||
      (rc = scratch(h, kSysStats, sizeof(SysStats) * R, &st)))
    return rc;

  // --- binning: records and keys of every point ---
  init_sys_stats_kernel<<<R, 256, 0, s>>>(dd, st);
  bin_kernel<T><<<blocks_for(P), 256, 0, s>>>(dd, poff, R, P, bbits, cbits, sbits, zf, pts, bkey,
                                              ckey, skey, iota, st);
  SCK(cudaGetLastError());

  // --- the three orders: (system, brick, bank, index) for the bricks,
  // (system, column, quantised z, index) for the direct sum's targets and
  // sources, one radix sort each (the sorted source keys take the place of the
  // unsorted target keys) ---
  if ((rc = sort_pairs(h, bkey, bkey_out, iota, border, P, rbits + bbits + 5, s)) ||
      (rc = sort_pairs(h, ckey, key_out, iota, corder, P, rbits + cbits + zf, s)) ||
      (rc = sort_pairs(h, skey, ckey, iota, sorder, P, rbits + sbits + zf, s)))
    return rc;
  starts_kernel<<<blocks_for(B + C + S + 3), 256, 0, s>>>(dd, R, boff, coff, soff, P, B, C, S,
                                                         bbits, cbits, sbits, zf, bkey_out,
                                                         key_out, ckey, bstart, cstart, sstart);
  if (std::max(B, C) <= kOneScan) {
    scans_kernel<<<2, 1024, 0, s>>>(bstart, (int)B, pos, cstart, (int)C, goff);
  } else {
    int *values;
    if ((rc = scratch(h, kValues, sizeof(int) * std::max(B, C), &values))) return rc;
    values_kernel<<<blocks_for(B), 256, 0, s>>>(NonEmpty{bstart}, B, values);
    if ((rc = exclusive_sum(h, values, pos, B, s))) return rc;
    values_kernel<<<blocks_for(C), 256, 0, s>>>(GroupsOf{cstart}, C, values);
    if ((rc = exclusive_sum(h, values, goff, C, s))) return rc;
  }
  round_place_kernel<<<blocks_for(B, kPlaceWarps), 32 * kPlaceWarps, 0, s>>>(bkey_out, border,
                                                                            bstart, B, border2);
  place_bricks_kernel<T><<<blocks_for(std::max(P, B)), 256, 0, s>>>(
      dd, poff, boff, R, P, B, border2, pts, bstart, pos, bpos);
  place_orders_kernel<T><<<blocks_for(P) + blocks_for(B, 8), 256, 0, s>>>(
      dd, poff, R, P, corder, sorder, bpos, cpos, blocks_for(P), boff, B, bstart, pos, st);
  SCK(cudaGetLastError());

  // --- warp groups and their source segments, heaviest groups first ---
  groups_kernel<<<blocks_for(32 * G), 256, 0, s>>>(dd, goffs, R, G, goff, cstart, sstart, ckey, zf,
                                                  sorder, cpos, ug, uh, uz, cen, bins,
                                                  bins + G, st);
  const dim3 og((unsigned)blocks_for(gmax), (unsigned)R, full ? 2 : 1);
  order_groups_kernel<<<og, 256, 0, s>>>(dd, goff, ug, uh, uz, cen, bins, bins + G, st);
  // the counts, for the host to read when the set-up has completed
  SetupCounts *dc;
  if ((rc = scratch(h, kCountsDev, sizeof(SetupCounts) * R, &dc))) return rc;
  if ((rc = pinned_block(h, &h->h_counts, &h->counts_cap, sizeof(SetupCounts) * R))) return rc;
  collect_counts_kernel<<<blocks_for(R, 64), 64, 0, s>>>(dd, R, st, goff, pos, dc);
  SCK(cudaMemcpyAsync(h->h_counts, dc, sizeof(SetupCounts) * R, cudaMemcpyDeviceToHost, s));
  SCK(cudaGetLastError());
  return NPME_OK;
}

}  // namespace

int device_bbox(npme_handle *h, const double *coord, double mn[3], double mx[3]) {
  const long n = (long)h->n;
  cudaStream_t s = h->stream;
  int rc;
  if ((rc = handle_buffer(h, (void **)&h->d_coord, sizeof(double) * 3 * n))) return rc;
  SCK(cudaMemcpyAsync(h->d_coord, coord, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s));
  if (n < kHostBoxPoints) {
    // small systems: one host pass costs less than a device reduction and
    // the wait for it
    for (int a = 0; a < 3; a++) mn[a] = 1e300, mx[a] = -1e300;
    for (long i = 0; i < n; i++)
      for (int a = 0; a < 3; a++) {
        const double x = coord[3 * i + a];
        if (!std::isfinite(x)) return record_error(h, NPME_EINVAL, "non-finite coordinate");
        mn[a] = std::min(mn[a], x);
        mx[a] = std::max(mx[a], x);
      }
    SCK(cudaGetLastError());
    return NPME_OK;
  }
  SetupStats *st;
  if ((rc = scratch(h, kStats, sizeof(SetupStats), &st))) return rc;
  init_stats_kernel<<<1, 1, 0, s>>>(st);
  const unsigned blocks = (unsigned)std::min<long>(blocks_for(n), 148 * 8);
  bbox_kernel<<<blocks, 256, 0, s>>>(h->d_coord, n, st);
  SCK(cudaGetLastError());
  SetupStats hs;
  SCK(cudaMemcpyAsync(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost, s));
  SCK(cudaStreamSynchronize(s));
  if (hs.nonfinite) return record_error(h, NPME_EINVAL, "non-finite coordinate");
  for (int a = 0; a < 3; a++) mn[a] = dkey_inv(hs.mn[a]), mx[a] = dkey_inv(hs.mx[a]);
  return NPME_OK;
}

int setup_geometry(npme_handle **hs, int R, cudaStream_t s, const std::function<int()> &hook) {
  return hs[0]->fp32 ? geometry_batch<float>(hs, R, s, hook)
                     : geometry_batch<double>(hs, R, s, hook);
}

int finish_setup(npme_handle *h, const npme_handle *owner, int r) {
  const SetupCounts &c = static_cast<const SetupCounts *>(owner->h_counts)[r];
  const long n = (long)h->n;
  if (c.bad < n) {
    // the axis of the first offending point, from its coordinates
    double x[3];
    SCK(cudaMemcpy(x, h->d_coord + 3 * c.bad, sizeof(x), cudaMemcpyDeviceToHost));
    const GridGeom &gr = h->grid;
    const double *R = h->box + 3, *L = h->box + 6;
    int axis = 0;
    for (int a = 0; a < 3; a++) {
      const double w = (double)gr.N[a] / L[a] * (x[a] - R[a]);
      const long ms = w < 0 ? (long)(-w) + 1 : (long)(-w);
      const long o = ms + gr.N[a] / 4;
      if (o < 0 || o + gr.order - 1 > gr.H[a] - 1) {
        axis = a;
        break;
      }
    }
    return record_error(h, NPME_EINVAL,
                        "point " + std::to_string(c.bad) + " has a B-spline stencil outside "
                        "the charge octant (axis " + std::to_string(axis) + ")");
  }
  h->n_nonempty = c.nnonempty;
  // odd bricks cost a launch of their own: not for a few that need not go (a system's edges)
  h->n_odd = c.must || 2 * c.nodd > c.nnonempty ? c.nodd : 0;
  h->n_groups = h->n_hgroups = c.ngroups;
  h->cand_per_point = (double)c.cand / (double)n;
  h->hcand_per_point = (double)c.hcand / (double)n;
  return NPME_OK;
}

}  // namespace npme
