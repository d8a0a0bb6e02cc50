// Batched CalcV: many set-up systems (different sizes, kernels, B-spline
// orders and FFT boxes) in one pass, one launch per stage and launch class.
//
// A launch class groups the systems a single kernel instantiation can serve:
//   gather, multiply        -> real / complex charges
//   spread, interpolation   -> (B-spline order, real / complex)
//   direct sum              -> identical pair-kernel coefficients (kernel,
//                              split, Rdir, nDeriv, alpha, k0); the
//                              coefficients stay in the parameter bank, as in
//                              the single-system launch
// Each class launch gets a device array of per-system descriptors and the
// prefix sums of its work units (points, bricks, transform CTAs, warp
// groups); a thread finds its system by binary search over the prefix.  The
// library's own transforms take all members of one kind in five launches; boxes with
// a length that has a prime factor above 5 run one by one with their handles' cuFFT
// plans.  FP32-bulk handles use
// the batch kernels; FP64 handles run their ordinary single-system path in
// the same stream order.  Results equal the single-system path's: the same
// bodies (bodies.cuh) run on the same data.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "batch.cuh"
#include "bodies.cuh"
#include "internal.h"

namespace npme {

template <bool CPLX>
__global__ void batch_gather_kernel(const BatchSys *__restrict__ sys,
                                    const long long *__restrict__ off, int count) {
  const long long total = off[count];
  for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < total;
       u += (long long)gridDim.x * blockDim.x) {
    const int s = find_sys(off, count, u);
    const BatchSys &S = sys[s];
    gather_body<float, CPLX>(S.q, S.dperm, S.qc, (long)(u - off[s]));
  }
}

// Zeroes the spread grids of a spread class; CTAs of kClearFloats floats each,
// off: prefix sums of the systems' CTAs.
constexpr long kClearFloats = 16384;
template <bool CPLX>
__global__ void __launch_bounds__(256) batch_clear_kernel(const BatchSys *__restrict__ sys,
                                                          const long long *__restrict__ off,
                                                          int count) {
  const int s = find_sys(off, count, blockIdx.x);
  const BatchSys &S = sys[s];
  const long n = (CPLX ? 2 : 1) * S.g1 * S.g2 * S.g3;  // even: so are the dimensions
  const long a = (blockIdx.x - off[s]) * kClearFloats, b = min(n, a + kClearFloats);
  for (long i = a + 2 * threadIdx.x; i < b; i += 512)
    *reinterpret_cast<float2 *>(S.grid + i) = make_float2(0.f, 0.f);
}

template <int P, bool CPLX>
__global__ void __launch_bounds__(256) batch_spread_kernel(const BatchSys *__restrict__ sys,
                                                           const long long *__restrict__ off,
                                                           int count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long u = blockIdx.x;
  const int s = find_sys(off, count, u);
  const BatchSys &S = sys[s];
  spread_brick<float, P, CPLX>(S.brick_list[u - off[s]], S.brick_start, S.bpts, S.q, S.grid,
                               S.nb2, S.nb3, S.g1, S.g2, S.g3, smem_raw, S.apart != 0);
}

// the odd bricks
template <int P, bool CPLX>
__global__ void __launch_bounds__(256, kSpreadOddCtas<float, P, CPLX>)
    batch_spread_odd_kernel(const BatchSys *__restrict__ sys, const long long *__restrict__ off,
                            int count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long u = blockIdx.x;
  const int s = find_sys(off, count, u);
  const BatchSys &S = sys[s];
  spread_brick_shared<float, P, CPLX>(S.odd_list[u - off[s]], S.brick_start, S.bpts, S.q, S.grid,
                                      S.nb2, S.nb3, S.g1, S.g2, S.g3, smem_raw);
}

// one warp per spectrum row of one system (units: rows)
template <bool CPLX>
__global__ void batch_multiply_kernel(const BatchSys *__restrict__ sys,
                                      const long long *__restrict__ off, int count) {
  const long long total = off[count];
  const int lane = threadIdx.x & 31;
  for (long long u = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; u < total;
       u += (gridDim.x * (long long)blockDim.x) >> 5) {
    const int s = find_sys(off, count, u);
    const BatchSys &S = sys[s];
    const int M2 = (int)(S.N2 / 2 + 1), M3 = (int)(S.N3 / 2 + 1);
    const int r = (int)(u - off[s]);
    if (CPLX)
      multiply_cplx_row<float>(reinterpret_cast<float2 *>(S.grid),
                               reinterpret_cast<const float2 *>(S.G), r, (int)S.N1, (int)S.N2,
                               (int)S.N3, M2, M3, lane);
    else
      multiply_real_row<float>(S.kgrid, S.G, r, (int)S.N1, (int)S.N2, (int)(S.N3 / 2 + 1), M2,
                               M3, lane);
  }
}

template <int P, bool CPLX>
__global__ void __launch_bounds__(256) batch_interp_kernel(const BatchSys *__restrict__ sys,
                                                           const long long *__restrict__ off,
                                                           int count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long u = blockIdx.x;
  const int s = find_sys(off, count, u);
  const BatchSys &S = sys[s];
  interp_brick_body<float, P, CPLX>(list_brick(S.brick_list[u - off[s]]), S.brick_start, S.bpts,
                                    S.grid, S.V, S.nb2, S.nb3, S.g1, S.g2, S.g3, S.c1, S.c2, S.c3,
                                    reinterpret_cast<float *>(smem_raw),
                                    S.fold ? (void *)S.vsrc : nullptr, S.vs, S.gs);
}

}  // namespace npme

using npme::BatchSys;

struct npme_batch {
  int device = 0;
  cudaStream_t stream2 = nullptr;
  cudaStream_t hi = nullptr;  // reciprocal chain: its CTAs go before the direct sums'
  // the direct-sum classes beyond the first run beside it
  static constexpr int kSide = 3;
  cudaStream_t side[kSide] = {};
  cudaEvent_t ev_side[kSide] = {}, ev_gather = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_done = nullptr;
  bool pending = false;  // ev_done recorded: buffers and members may be in use
  unsigned char *h_pinned = nullptr;  // host image of the descriptor block
  size_t h_cap = 0;
  unsigned char *d_block = nullptr;
  size_t d_cap = 0;
  std::string err;
  int launches = 0;
};

namespace {

int bfail(npme_batch *b, int code, const std::string &m) {
  if (b) b->err = m;
  return code;
}

// One launch class: the systems it serves and the prefix of its work units.
struct Class {
  std::vector<int> members;  // indices into the batch's FP32 handle list
  std::vector<long long> off;   // prefix of the class's work units
  size_t desc_at = 0, off_at = 0;  // byte offsets in the descriptor block
};

// The members whose transforms the library's own kernels run.
struct FftClass {
  std::vector<int> members;
  std::vector<long long> off;  // CTA prefixes of x, y and z
  long units[3] = {0, 0, 0};
  size_t smem[3] = {0, 0, 0};
  size_t desc_at = 0, off_at = 0;
};

size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

}  // namespace

extern "C" {

int npme_gpu_batch_create(int device, npme_batch **out) {
  if (!out) return NPME_EINVAL;
  *out = nullptr;
  npme_batch *b = new (std::nothrow) npme_batch;
  if (!b) return NPME_ENOMEM;
  b->device = device;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream2, cudaStreamNonBlocking);
  int prio_lo = 0, prio_hi = 0;
  if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi);
  if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&b->hi, cudaStreamNonBlocking, prio_hi);
  for (int i = 0; i < npme_batch::kSide && e == cudaSuccess; i++) {
    e = cudaStreamCreateWithFlags(&b->side[i], cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_side[i], cudaEventDisableTiming);
  }
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_gather, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_done, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    npme_gpu_batch_destroy(b);
    return NPME_ECUDA;
  }
  *out = b;
  return NPME_OK;
}

int npme_gpu_batch_destroy(npme_batch *b) {
  if (!b) return NPME_OK;
  cudaSetDevice(b->device);
  if (b->pending) cudaEventSynchronize(b->ev_done);
  if (b->stream2) cudaStreamSynchronize(b->stream2);
  if (b->hi) cudaStreamSynchronize(b->hi);
  for (int i = 0; i < npme_batch::kSide; i++)
    if (b->side[i]) cudaStreamSynchronize(b->side[i]);
  if (b->stream2) cudaStreamDestroy(b->stream2);
  if (b->hi) cudaStreamDestroy(b->hi);
  for (int i = 0; i < npme_batch::kSide; i++) {
    if (b->side[i]) cudaStreamDestroy(b->side[i]);
    if (b->ev_side[i]) cudaEventDestroy(b->ev_side[i]);
  }
  if (b->ev_gather) cudaEventDestroy(b->ev_gather);
  if (b->ev_fork) cudaEventDestroy(b->ev_fork);
  if (b->ev_join) cudaEventDestroy(b->ev_join);
  if (b->ev_done) cudaEventDestroy(b->ev_done);
  if (b->h_pinned) cudaFreeHost(b->h_pinned);
  if (b->d_block) cudaFree(b->d_block);
  delete b;
  return NPME_OK;
}

int npme_gpu_batch_sync(npme_batch *b) {
  if (!b) return NPME_EINVAL;
  if (cudaSetDevice(b->device) != cudaSuccess) return bfail(b, NPME_ECUDA, "cudaSetDevice");
  cudaError_t e = cudaSuccess;
  if (b->pending) e = cudaEventSynchronize(b->ev_done);
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream2);
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->hi);
  for (int i = 0; i < npme_batch::kSide && e == cudaSuccess; i++)
    e = cudaStreamSynchronize(b->side[i]);
  b->pending = false;
  if (e != cudaSuccess) return bfail(b, NPME_ECUDA, cudaGetErrorString(e));
  return NPME_OK;
}

int npme_gpu_batch_last_error(const npme_batch *b, char *buf, size_t len) {
  if (!b || !buf || len == 0) return NPME_EINVAL;
  strncpy(buf, b->err.c_str(), len - 1);
  buf[len - 1] = 0;
  return NPME_OK;
}

int npme_gpu_calcv_batch(npme_batch *b, npme_handle *const *hs, int count,
                         double *const *d_V, const double *const *d_q, void *stream) {
  using namespace npme;
  if (!b) return NPME_EINVAL;
  if (count < 0 || (count > 0 && (!hs || !d_V || !d_q)))
    return bfail(b, NPME_EINVAL, "bad batch arguments");
  if (count == 0) return NPME_OK;
  for (int i = 0; i < count; i++) {
    if (!hs[i] || !hs[i]->ready) return bfail(b, NPME_ESTATE, "batch member not set up");
    if (hs[i]->device != b->device) return bfail(b, NPME_EINVAL, "batch member on another device");
    if (!d_V[i] || !d_q[i]) return bfail(b, NPME_EINVAL, "null buffer in batch");
  }
  if (cudaSetDevice(b->device) != cudaSuccess) return bfail(b, NPME_ECUDA, "cudaSetDevice");
  const cudaStream_t user = (cudaStream_t)stream;
  b->launches = 0;

  // FP64 (plain) and caller-defined-kernel members take their ordinary path
  // in stream order
  std::vector<int> f32;
  for (int i = 0; i < count; i++) {
    if (hs[i]->fp32 && !hs[i]->user_kernel) {
      f32.push_back(i);
    } else {
      const int rc = npme_gpu_calcv_device(hs[i], d_V[i], d_q[i], stream);
      if (rc) return bfail(b, rc, "batch member: " + hs[i]->err);
      b->launches += hs[i]->launches;
    }
  }
  const int m = (int)f32.size();
  if (m == 0) {
    // the members' own CalcVs are on `stream`: npme_gpu_batch_sync waits for them
    if (cudaEventRecord(b->ev_done, user) != cudaSuccess)
      return bfail(b, NPME_ECUDA, "batch: event record failed");
    b->pending = true;
    return NPME_OK;
  }

  // descriptors
  std::vector<BatchSys> desc(m);
  for (int k = 0; k < m; k++) {
    const npme_handle *h = hs[f32[k]];
    BatchSys &S = desc[k];
    memset(&S, 0, sizeof(S));
    S.q = d_q[f32[k]];
    S.V = d_V[f32[k]];
    S.bpts = (const BrickPoint<float> *)h->d_bpts;
    S.cperm = h->d_cperm;
    S.dperm = h->d_dperm;
    S.qc = (float *)h->d_qc;
    S.brick_list = h->d_brick_list;
    S.odd_list = h->d_odd_list;
    S.apart = h->n_odd > 0;
    S.brick_start = h->d_brick_start;
    S.nb2 = (int)h->grid.nb[1];
    S.nb3 = (int)h->grid.nb[2];
    S.grid = (float *)h->d_grid;
    S.kgrid = (float2 *)h->d_kgrid;
    S.G = (const float *)h->d_G;
    S.N1 = h->grid.N[0], S.N2 = h->grid.N[1], S.N3 = h->grid.N[2];
    S.g1 = h->gd[0], S.g2 = h->gd[1], S.g3 = h->gd[2];
    const int P = h->grid.order;
    const double dw = npme::spline_scale(P) / npme::spline_scale(P - 1);
    S.c1 = (float)(h->grid.N[0] / h->box[6] * dw);
    S.c2 = (float)(h->grid.N[1] / h->box[7] * dw);
    S.c3 = (float)(h->grid.N[2] / h->box[8] * dw);
    S.gpos = h->d_gpos;
    S.spos = h->d_spos;
    S.groups = h->d_groups;
    S.gcen = h->d_gcen;
    S.segs = h->d_segs;
    S.hgroups = h->d_hgroups;
    S.hcen = h->d_hcen;
    S.hsegs = h->d_hsegs;
    S.hzones = h->d_hzones;
    S.vsrc = h->d_vsrc;
    S.bperm = h->d_bperm;
    S.refine2 = (float)h->refine2;
    S.fself_r = h->fself_r;
    S.fself_i = h->fself_i;
    S.fold = pairs_once(h) ? 1 : 0;
    const bool scaled =
        h->p.funcType != NPME_FUNC_HELMHOLTZ;
    const PairCoef<float> pc = make_pair_coef<float>(h);
    S.vs = scaled ? pc.vscale : 1.0;
    S.gs = scaled ? pc.gscale : 1.0;
  }

  // launch classes
  std::map<int, Class> clr;  // key: complex (members with the library's transforms)
  std::map<int, Class> gath, mult;                           // key: complex (mult: cuFFT members)
  std::map<int, FftClass> own;                               // key: complex
  std::map<std::pair<int, int>, Class> spr, odd;             // (order, complex); odd bricks
  typedef std::tuple<int, int, int, int, double, double, double, double, double> DKey;
  std::map<DKey, Class> dir;  // direct sums
  for (int k = 0; k < m; k++) {
    const npme_handle *h = hs[f32[k]];
    const int cx = h->complex_kernel ? 1 : 0;
    gath[cx].members.push_back(k);
    if (h->own_fft) own[cx].members.push_back(k), clr[cx].members.push_back(k);
    else mult[cx].members.push_back(k);
    spr[{h->grid.order, cx}].members.push_back(k);
    if (h->n_odd > 0) odd[{h->grid.order, cx}].members.push_back(k);
    const DKey key(pairs_once(h) ? 1 : 0, h->p.funcType, h->p.EwaldSplit, h->p.nDeriv,
                   h->p.Rdir, h->p.alpha, h->p.k0_r, h->p.k0_i, h->beta);
    dir[key].members.push_back(k);
  }
  auto units_gather = [&](int k) { return (long long)hs[f32[k]]->n; };
  auto units_spread = [&](int k) { return (long long)hs[f32[k]]->n_nonempty; };
  auto units_odd = [&](int k) { return (long long)hs[f32[k]]->n_odd; };
  auto units_mult = [&](int k) {  // spectrum rows
    const long *N = hs[f32[k]]->grid.N;
    return (long long)N[0] * N[1];
  };
  auto units_clear = [&](int k) {
    const npme_handle *h = hs[f32[k]];
    const long n = (h->complex_kernel ? 2 : 1) * h->gd[0] * h->gd[1] * h->gd[2];
    return (long long)((n + kClearFloats - 1) / kClearFloats);
  };
  auto units_dir = [&](int k) {
    const npme_handle *h = hs[f32[k]];
    return (long long)(pairs_once(h) ? h->n_hgroups : h->n_groups);
  };

  // descriptor block layout: for every class, its descriptors then offsets
  size_t bytes = 0;
  std::vector<Class *> all;
  auto lay = [&](Class &c, auto units) {
    c.off.assign(c.members.size() + 1, 0);
    for (size_t t = 0; t < c.members.size(); t++) c.off[t + 1] = c.off[t] + units(c.members[t]);
    c.desc_at = bytes;
    bytes = align16(bytes + sizeof(BatchSys) * c.members.size());
    c.off_at = bytes;
    bytes = align16(bytes + sizeof(long long) * c.off.size());
    all.push_back(&c);
  };
  for (auto &kv : gath) lay(kv.second, units_gather);
  for (auto &kv : clr) lay(kv.second, units_clear);
  for (auto &kv : mult) lay(kv.second, units_mult);
  for (auto &kv : spr) lay(kv.second, units_spread);  // spread and interpolation: bricks
  for (auto &kv : odd) lay(kv.second, units_odd);
  for (auto &kv : dir) lay(kv.second, units_dir);
  for (auto &kv : own) {  // transform descriptors, then the CTA prefixes of x, y and z
    FftClass &c = kv.second;
    const size_t n = c.members.size();
    c.off.assign(3 * (n + 1), 0);
    for (int a = 0; a < 3; a++) {
      long long *o = c.off.data() + a * (n + 1);
      c.smem[a] = 0;
      for (size_t t = 0; t < n; t++) {
        const FftJob &j = hs[f32[c.members[t]]]->fft;
        o[t + 1] = o[t] + (a == 0 ? j.ux : a == 1 ? j.uy : j.uz);
        c.smem[a] = std::max(c.smem[a], own_fft_smem(j, a, sizeof(float2)));
      }
      c.units[a] = o[n];
      if (c.units[a] >= (1LL << 31)) return bfail(b, NPME_EINVAL, "batch too large");
    }
    c.desc_at = bytes;
    bytes = align16(bytes + sizeof(FftJob) * n);
    c.off_at = bytes;
    bytes = align16(bytes + sizeof(long long) * c.off.size());
  }

  // the pinned staging buffer is reused: wait for the previous batch's copy
  if (b->pending) {
    cudaEventSynchronize(b->ev_done);
    b->pending = false;
  }
  if (bytes > b->h_cap) {
    if (b->h_pinned) cudaFreeHost(b->h_pinned);
    b->h_pinned = nullptr;
    b->h_cap = 0;
    // at least 1 MiB: a serving loop then never grows it (cudaMallocHost /
    // cudaFreeHost are slow and take driver locks other threads wait for)
    const size_t cap = std::max<size_t>(bytes * 2, size_t(1) << 20);
    if (cudaMallocHost((void **)&b->h_pinned, cap) != cudaSuccess)
      return bfail(b, NPME_ENOMEM, "pinned descriptor buffer");
    b->h_cap = cap;
  }
  if (bytes > b->d_cap) {
    if (b->d_block) cudaFree(b->d_block);
    b->d_block = nullptr;
    b->d_cap = 0;
    // the same floor: cudaFree waits for the whole device
    const size_t cap = std::max<size_t>(bytes * 2, size_t(1) << 20);
    if (cudaMalloc((void **)&b->d_block, cap) != cudaSuccess)
      return bfail(b, NPME_ENOMEM, "device descriptor buffer");
    b->d_cap = cap;
  }
  for (Class *c : all) {
    BatchSys *dd = (BatchSys *)(b->h_pinned + c->desc_at);
    for (size_t t = 0; t < c->members.size(); t++) dd[t] = desc[c->members[t]];
    memcpy(b->h_pinned + c->off_at, c->off.data(), sizeof(long long) * c->off.size());
  }
  for (auto &kv : own) {
    FftClass &c = kv.second;
    FftJob *dj = (FftJob *)(b->h_pinned + c.desc_at);
    for (size_t t = 0; t < c.members.size(); t++) dj[t] = hs[f32[c.members[t]]]->fft;
    memcpy(b->h_pinned + c.off_at, c.off.data(), sizeof(long long) * c.off.size());
  }
  cudaMemcpyAsync(b->d_block, b->h_pinned, bytes, cudaMemcpyHostToDevice, user);
  auto D = [&](const Class &c) { return (const BatchSys *)(b->d_block + c.desc_at); };
  auto O = [&](const Class &c) { return (const long long *)(b->d_block + c.off_at); };
  auto grid_of = [](long long units, int threads, int cap) {
    return (unsigned)std::max<long long>(1, std::min<long long>((units + threads - 1) / threads, cap));
  };

  // A failure from here on leaves with work of this call enqueued: all of its streams
  // join the caller's, and the source-side sums that no interpolation takes are cleared.
  auto leave = [&](const std::string &msg) {
    for (int i = 0; i <= npme_batch::kSide; i++) {
      cudaEvent_t ev = i < npme_batch::kSide ? b->ev_side[i] : b->ev_join;
      cudaEventRecord(ev, i < npme_batch::kSide ? b->side[i] : b->stream2);
      cudaStreamWaitEvent(b->hi, ev, 0);
    }
    for (int k = 0; k < m; k++) clear_source_sums(hs[f32[k]], b->hi);
    cudaEventRecord(b->ev_done, b->hi);
    cudaStreamWaitEvent(user, b->ev_done, 0);
    b->pending = true;
    cudaGetLastError();
    return bfail(b, NPME_ECUDA, "batch: " + msg);
  };

  // 1. gather, then 2. direct sums, on the second stream, beside the
  // reciprocal sums
  const cudaStream_t s = b->hi;  // the reciprocal chain
  cudaEventRecord(b->ev_fork, user);
  cudaStreamWaitEvent(s, b->ev_fork, 0);
  cudaStreamWaitEvent(b->stream2, b->ev_fork, 0);
  for (auto &kv : gath) {
    Class &c = kv.second;
    const unsigned g = grid_of(c.off.back(), 256, 148 * 16);
    const int m = (int)c.members.size();
    if (kv.first) batch_gather_kernel<true><<<g, 256, 0, b->stream2>>>(D(c), O(c), m);
    else batch_gather_kernel<false><<<g, 256, 0, b->stream2>>>(D(c), O(c), (int)c.members.size());
    b->launches++;
  }
  cudaEventRecord(b->ev_gather, b->stream2);
  int nclass = 0;  // direct-sum launches so far
  for (auto &kv : dir) {
    Class &c = kv.second;
    const npme_handle *h0 = hs[f32[c.members[0]]];
    const PairCoef<float> k = make_pair_coef<float>(h0);
    const long long ng = c.off.back();
    if (ng == 0) continue;
    // classes beyond the first on streams of their own: a class has its own
    // tail of late CTAs, which the others fill
    cudaStream_t ds = b->stream2;
    if (nclass > 0) {
      const int i = (nclass - 1) % npme_batch::kSide;
      ds = b->side[i];
      if (nclass <= npme_batch::kSide) cudaStreamWaitEvent(ds, b->ev_gather, 0);
    }
    launch_batch_direct(k, std::get<0>(kv.first) != 0, h0->p.alpha >= 0, D(c), O(c),
                        (int)c.members.size(), ng, ds);
    nclass++;
    b->launches++;
  }
  for (int i = 0; i < std::min(nclass - 1, (int)npme_batch::kSide); i++) {
    cudaEventRecord(b->ev_side[i], b->side[i]);
    cudaStreamWaitEvent(b->stream2, b->ev_side[i], 0);
  }
  cudaEventRecord(b->ev_join, b->stream2);
  // 3. spread (grids zeroed first)
  for (auto &kv : clr) {
    Class &c = kv.second;
    const unsigned g = (unsigned)c.off.back();
    if (kv.first) batch_clear_kernel<true><<<g, 256, 0, s>>>(D(c), O(c), (int)c.members.size());
    else batch_clear_kernel<false><<<g, 256, 0, s>>>(D(c), O(c), (int)c.members.size());
    b->launches++;
  }
  for (int k = 0; k < m; k++)
    if (!hs[f32[k]]->own_fft) grid_clear(hs[f32[k]], s);
  for (auto &kv : spr) {
    Class &c = kv.second;
    const long long nb = c.off.back();
    if (nb == 0) continue;
    const int P = kv.first.first;
    const bool cx = kv.first.second;
    const int cnt = (int)c.members.size();
#define NPME_BS(PP, CX)                                                                    \
  {                                                                                        \
    const size_t smem = spread_smem<float, PP, CX>();                                      \
    auto kern = batch_spread_kernel<PP, CX>;                                               \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    kern<<<(unsigned)nb, 256, smem, s>>>(D(c), O(c), cnt);                                 \
  }
#define NPME_BS_P(CX)                    \
  switch (P) {                           \
    case 4: NPME_BS(4, CX); break;       \
    case 6: NPME_BS(6, CX); break;       \
    case 8: NPME_BS(8, CX); break;       \
    case 10: NPME_BS(10, CX); break;     \
    case 12: NPME_BS(12, CX); break;     \
    case 14: NPME_BS(14, CX); break;     \
    case 16: NPME_BS(16, CX); break;     \
  }
    if (cx) { NPME_BS_P(true); } else { NPME_BS_P(false); }
#undef NPME_BS_P
#undef NPME_BS
    b->launches++;
  }
  for (auto &kv : odd) {
    Class &c = kv.second;
    const unsigned nb = (unsigned)c.off.back();
    const int cnt = (int)c.members.size();
    auto launch = [&](auto kern, size_t smem) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      kern<<<nb, 256, smem, s>>>(D(c), O(c), cnt);
      b->launches++;
    };
    const int P = kv.first.first;  // the others take odd bricks with the rest (kSpreadApart)
    static_assert(kSpreadApart<float, 6> && kSpreadApart<float, 8> && !kSpreadApart<float, 4>);
    if (P == 6 && kv.first.second)
      launch(batch_spread_odd_kernel<6, true>, SpreadOwner<float, 6, true>::kSharedBytes);
    else if (P == 6)
      launch(batch_spread_odd_kernel<6, false>, SpreadOwner<float, 6, false>::kSharedBytes);
    else if (P == 8 && kv.first.second)
      launch(batch_spread_odd_kernel<8, true>, SpreadOwner<float, 8, true>::kSharedBytes);
    else if (P == 8)
      launch(batch_spread_odd_kernel<8, false>, SpreadOwner<float, 8, false>::kSharedBytes);
  }
  {  // launch errors are checked before cuFFT runs
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return leave(cudaGetErrorString(e));
  }
  // 4. transforms and kernel multiply of the members with the library's own
  // transforms: five launches for all of one kind
  for (auto &kv : own) {
    FftClass &c = kv.second;
    own_convolve_batch((const FftJob *)(b->d_block + c.desc_at),
                       (const long long *)(b->d_block + c.off_at), (int)c.members.size(),
                       kv.first != 0, c.units, c.smem, s);
    b->launches += 5;
  }
  // the others: forward transforms
  for (int k = 0; k < m; k++) {
    npme_handle *h = hs[f32[k]];
    if (!h->own_fft && fft_forward(h, s)) return leave(h->err);
  }
  // 5. kernel multiply
  for (auto &kv : mult) {
    Class &c = kv.second;
    const unsigned g = grid_of(c.off.back(), 8, 148 * 16);  // 8 rows (warps) per CTA
    if (kv.first) batch_multiply_kernel<true><<<g, 256, 0, s>>>(D(c), O(c), (int)c.members.size());
    else batch_multiply_kernel<false><<<g, 256, 0, s>>>(D(c), O(c), (int)c.members.size());
    b->launches++;
  }
  {  // launch errors are checked before cuFFT runs
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return leave(cudaGetErrorString(e));
  }
  // 6. inverse transforms
  for (int k = 0; k < m; k++) {
    npme_handle *h = hs[f32[k]];
    if (!h->own_fft && fft_inverse(h, s)) return leave(h->err);
  }
  // 7. interpolation after the direct sums
  cudaStreamWaitEvent(s, b->ev_join, 0);
  for (auto &kv : spr) {
    Class &c = kv.second;
    const int P = kv.first.first;
    const bool cx = kv.first.second;
    const long long nb = c.off.back();
    if (nb == 0) continue;
    const int cnt = (int)c.members.size();
#define NPME_BI(PP, CX)                                                                    \
  {                                                                                        \
    constexpr int TL = kBrick + PP - 1;                                                    \
    const size_t smem = sizeof(float) * TL * TL * TL * (CX ? 2 : 1);                       \
    auto kern = batch_interp_kernel<PP, CX>;                                               \
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    kern<<<(unsigned)nb, 256, smem, s>>>(D(c), O(c), cnt);                                 \
  }
#define NPME_BI_P(CX)                   \
  switch (P) {                          \
    case 4: NPME_BI(4, CX); break;      \
    case 6: NPME_BI(6, CX); break;      \
    case 8: NPME_BI(8, CX); break;      \
    case 10: NPME_BI(10, CX); break;    \
    case 12: NPME_BI(12, CX); break;    \
    case 14: NPME_BI(14, CX); break;    \
    case 16: NPME_BI(16, CX); break;    \
  }
    if (cx) { NPME_BI_P(true); } else { NPME_BI_P(false); }
#undef NPME_BI_P
#undef NPME_BI
    b->launches++;
  }
  cudaEventRecord(b->ev_done, s);
  cudaStreamWaitEvent(user, b->ev_done, 0);
  b->pending = true;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return leave(cudaGetErrorString(e));
  return NPME_OK;
}

}  // extern "C"
