// The library's own transforms of the reciprocal sum (fft_own.cuh): plans,
// twiddle tables and launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "fft_own.cuh"
#include "internal.h"

namespace npme {

template <typename T, bool CPLX, int DIR>
__global__ void __launch_bounds__(kFftThreads) fft_z_kernel(const __grid_constant__ FftJob J) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  fft_z_body<T, CPLX, DIR>(J, blockIdx.x, fft_smem);
}
template <typename T, int DIR>
__global__ void __launch_bounds__(kFftThreads) fft_y_kernel(const __grid_constant__ FftJob J) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  fft_y_body<T, DIR>(J, blockIdx.x, fft_smem);
}
template <typename T, bool CPLX>
__global__ void __launch_bounds__(kFftThreads) fft_x_kernel(const __grid_constant__ FftJob J) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  fft_x_body<T, CPLX>(J, blockIdx.x, fft_smem);
}

// Batched passes (FP32): CTAs of all systems concatenated, off[s] the first
// CTA of system s.
__device__ __forceinline__ int fft_owner(const long long *__restrict__ off, int count, long u) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int m = (lo + hi + 1) >> 1;
    if (off[m] <= u) lo = m;
    else hi = m - 1;
  }
  return lo;
}
template <bool CPLX, int DIR>
__global__ void __launch_bounds__(kFftThreads)
    batch_fft_z_kernel(const FftJob *__restrict__ jobs, const long long *__restrict__ off,
                       int count) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  const int s = fft_owner(off, count, blockIdx.x);
  fft_z_body<float, CPLX, DIR>(jobs[s], blockIdx.x - off[s], fft_smem);
}
template <int DIR>
__global__ void __launch_bounds__(kFftThreads)
    batch_fft_y_kernel(const FftJob *__restrict__ jobs, const long long *__restrict__ off,
                       int count) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  const int s = fft_owner(off, count, blockIdx.x);
  fft_y_body<float, DIR>(jobs[s], blockIdx.x - off[s], fft_smem);
}
template <bool CPLX>
__global__ void __launch_bounds__(kFftThreads)
    batch_fft_x_kernel(const FftJob *__restrict__ jobs, const long long *__restrict__ off,
                       int count) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  const int s = fft_owner(off, count, blockIdx.x);
  fft_x_body<float, CPLX>(jobs[s], blockIdx.x - off[s], fft_smem);
}

namespace {

// Radices of N, as few as possible, then the smallest largest one, none above
// `largest`; an even one first (half of the line is zero at the start and
// unwanted at the end of the reverse order).  Empty when N has a factor other
// than 2, 3 and 5 or takes fewer than two passes.
std::vector<int> radices(long N, int largest = 16) {
  static const int kR[] = {16, 12, 10, 9, 8, 6, 5, 4, 3, 2};
  // products of at most `left` radices, none above cap
  struct Search {
    static bool run(long n, int left, int cap, std::vector<int> &out) {
      if (n == 1) return true;
      if (left == 0) return false;
      for (int r : kR) {
        if (r > cap || n % r) continue;
        out.push_back(r);
        if (run(n / r, left - 1, r, out)) return true;
        out.pop_back();
      }
      return false;
    }
  };
  std::vector<int> r;
  for (int passes = 2; passes <= 8; passes++)
    for (int i = 9; i >= 0 && kR[i] <= largest; i--) {
      r.clear();
      if (Search::run(N, passes, kR[i], r)) {
        if (r.size() < 2 || N % 2) r.clear();
        for (size_t k = 0; k < r.size(); k++)
          if (r[k] % 2 == 0) {
            std::swap(r[0], r[k]);
            break;
          }
        return r;
      }
    }
  r.clear();
  return r;
}

// Twiddle tables, one per (device, precision, length) for the whole process,
// like the FFT plans; never freed (16 KB at length 2,048 in FP32).
std::mutex g_tw_mu;
std::map<std::tuple<int, bool, long>, void *> g_tw;

// (On a stream and waited for: cudaMemcpy from pageable memory may return before the
// copy has arrived, and non-blocking streams do not wait for it.)
template <typename C>
cudaError_t make_table(long N, cudaStream_t s, void **out) {
  std::vector<C> t(N);
  for (long m = 0; m < N; m++) {
    const double a = -2.0 * M_PI * (double)m / (double)N;
    t[m].x = std::cos(a), t[m].y = std::sin(a);
  }
  void *d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(C) * N);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d, t.data(), sizeof(C) * N, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess && d) cudaFree(d), d = nullptr;
  *out = d;
  return e;
}

int twiddles(npme_handle *h, long N, const void **out) {
  std::lock_guard<std::mutex> lk(g_tw_mu);
  void *&d = g_tw[std::make_tuple(h->device, h->fp32, N)];
  if (!d) {
    const cudaError_t e = h->fp32 ? make_table<float2>(N, h->stream, &d)
                                   : make_table<double2>(N, h->stream, &d);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return record_error(h, NPME_ECUDA, std::string("FFT tables: ") + cudaGetErrorString(e));
    }
  }
  *out = d;
  return NPME_OK;
}

// Passes of a length-N transform whose twiddles are every `stride`-th entry
// of a table.
void make_axis(FftAxis &a, long N, int stride, bool fp32, bool reverse) {
  a.N = (int)N;
  a.np = 0;
  int Ns = 1;
  // radix 9 and more take two doubles too many per value for two resident CTAs
  // in FP64 (128 registers): 256^3 in FP64 235 us with them, 209 without
  std::vector<int> radix = radices(N, fp32 ? 16 : 8);
  if (reverse) std::reverse(radix.begin(), radix.end());
  for (int R : radix) {
    FftPass &p = a.p[a.np++];
    p.R = R, p.Ns = Ns;
    p.magic = (unsigned)(0xffffffffu / (unsigned)Ns) + 1u;  // not used for Ns = 1
    p.step = (int)(N / ((long)Ns * R)) * stride;
    Ns *= R;
  }
  a.twlen = (int)(N * stride);
}

}  // namespace

size_t own_fft_smem(const FftJob &j, int axis, size_t cbytes) {
  const FftAxis &a = axis == 0 ? j.x : axis == 1 ? j.y : j.z;
  const size_t B = (size_t)1 << a.lb;
  // twiddles and two buffers of the CTA's lines (along z padded)
  return cbytes * (a.twlen + 2 * (axis == 2 ? (size_t)(a.N + 1) * (B + 1) : (size_t)a.N * B));
}

// Shared memory of a CTA: at most about half of an SM's, so that two or more are
// resident, with 4 or 2 lines where 8 do not fit that; two lines of the greatest
// length (2,048) fit a CTA in FP64 (229,472 bytes along z, complex).
static constexpr size_t kFftSmem = 100 * 1024, kFftSmemMax = 226 * 1024;

bool own_fft_lengths(const long N[3]) {
  for (int a = 0; a < 3; a++)
    if (radices(N[a]).empty()) return false;
  return !radices(N[2] / 2).empty();
}

int own_fft_prepare(npme_handle *h) {
  FftJob &j = h->fft;
  j = FftJob{};
  const long *N = h->grid.N;
  for (int a = 0; a < 3; a++) j.N[a] = (int)N[a], j.H[a] = (int)(N[a] / 2);
  const bool cx = h->complex_kernel;
  j.K = cx ? j.N[2] : j.H[2] + 1;
  j.KP = (j.K + 3) & ~3;
  j.grid = h->d_grid, j.spec = h->d_kgrid, j.G = h->d_G;
  for (int r = 0; r < 2; r++) {
    make_axis(r ? j.xi : j.x, N[0], 1, h->fp32, r != 0);
    make_axis(r ? j.yi : j.y, N[1], 1, h->fp32, r != 0);
    make_axis(r ? j.zi : j.z, cx ? N[2] : N[2] / 2, cx ? 1 : 2, h->fp32, r != 0);
  }
  int rc;
  if ((rc = twiddles(h, N[0], &j.x.tw)) || (rc = twiddles(h, N[1], &j.y.tw)) ||
      (rc = twiddles(h, N[2], &j.z.tw)))
    return rc;
  const size_t cb = h->fp32 ? 8 : 16;
  FftAxis *ax[3] = {&j.x, &j.y, &j.z};
  const long lines[3] = {(long)j.N[1] * j.KP, (long)j.H[0] * j.KP, (long)j.H[0] * j.H[1]};
  long *units[3] = {&j.ux, &j.uy, &j.uz};
  for (int a = 0; a < 3; a++) {
    // 16 lines (128 bytes of a row in FP32), fewer when they do not fit or
    // when the pass would leave SMs without a CTA
    int lb = kFftMaxLines;
    for (ax[a]->lb = lb; lb > 1; lb--) {
      ax[a]->lb = lb;
      if (own_fft_smem(j, a, cb) <= kFftSmem && (lb <= 3 || (lines[a] >> lb) >= 148)) break;
    }
    ax[a]->lb = std::max(lb, 1);
    *units[a] = (lines[a] + (1L << ax[a]->lb) - 1) >> ax[a]->lb;
  }
  j.xi.lb = j.x.lb, j.yi.lb = j.y.lb, j.zi.lb = j.z.lb;
  j.xi.tw = j.x.tw, j.yi.tw = j.y.tw, j.zi.tw = j.z.tw;
  return NPME_OK;
}

namespace {

// The kernels' shared-memory limit, raised once per kernel and device.
template <class K>
void raise_limit(K kern) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, bool> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  bool &d = done[std::make_pair(dev, (const void *)kern)];
  if (!d) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFftSmemMax);
  d = true;
}

template <typename T, bool CPLX>
void convolve(const FftJob &j, int part, cudaStream_t s) {
  const size_t cb = sizeof(Cx<T>);
  const size_t mx = own_fft_smem(j, 0, cb), my = own_fft_smem(j, 1, cb), mz = own_fft_smem(j, 2, cb);
  auto zf = fft_z_kernel<T, CPLX, -1>;
  auto zi = fft_z_kernel<T, CPLX, 1>;
  auto yf = fft_y_kernel<T, -1>;
  auto yi = fft_y_kernel<T, 1>;
  auto xx = fft_x_kernel<T, CPLX>;
  raise_limit(zf), raise_limit(zi), raise_limit(yf), raise_limit(yi), raise_limit(xx);
  if (part == 0) {
    zf<<<(unsigned)j.uz, kFftThreads, mz, s>>>(j);
    yf<<<(unsigned)j.uy, kFftThreads, my, s>>>(j);
  } else if (part == 1) {
    xx<<<(unsigned)j.ux, kFftThreads, mx, s>>>(j);
  } else {
    yi<<<(unsigned)j.uy, kFftThreads, my, s>>>(j);
    zi<<<(unsigned)j.uz, kFftThreads, mz, s>>>(j);
  }
}

template <bool CPLX>
void convolve_batch(const FftJob *jobs, const long long *offs, int count, const long units[3],
                    const size_t smem[3], cudaStream_t s) {
  // offs: the CTA prefixes of x, y and z, count + 1 each
  const long long *ox = offs, *oy = offs + count + 1, *oz = offs + 2 * (count + 1);
  auto zf = batch_fft_z_kernel<CPLX, -1>;
  auto zi = batch_fft_z_kernel<CPLX, 1>;
  auto yf = batch_fft_y_kernel<-1>;
  auto yi = batch_fft_y_kernel<1>;
  auto xx = batch_fft_x_kernel<CPLX>;
  raise_limit(zf), raise_limit(zi), raise_limit(yf), raise_limit(yi), raise_limit(xx);
  zf<<<(unsigned)units[2], kFftThreads, smem[2], s>>>(jobs, oz, count);
  yf<<<(unsigned)units[1], kFftThreads, smem[1], s>>>(jobs, oy, count);
  xx<<<(unsigned)units[0], kFftThreads, smem[0], s>>>(jobs, ox, count);
  yi<<<(unsigned)units[1], kFftThreads, smem[1], s>>>(jobs, oy, count);
  zi<<<(unsigned)units[2], kFftThreads, smem[2], s>>>(jobs, oz, count);
}

}  // namespace

void own_convolve(npme_handle *h, int part, cudaStream_t s) {
  if (h->fp32) {
    if (h->complex_kernel) convolve<float, true>(h->fft, part, s);
    else convolve<float, false>(h->fft, part, s);
  } else {
    if (h->complex_kernel) convolve<double, true>(h->fft, part, s);
    else convolve<double, false>(h->fft, part, s);
  }
  h->launches += part == 1 ? 1 : 2;
}

void own_convolve_batch(const FftJob *jobs, const long long *offs, int count, bool cplx,
                        const long units[3], const size_t smem[3], cudaStream_t s) {
  if (cplx) convolve_batch<true>(jobs, offs, count, units, smem, s);
  else convolve_batch<false>(jobs, offs, count, units, smem, s);
}

}  // namespace npme
