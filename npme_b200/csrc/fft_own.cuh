// The reciprocal sum's transforms for FFT lengths with factors 2, 3 and 5,
// written for the charge octant.
//
// Charges and theta live on the octant H1 x H2 x H3 (H = N/2) of the
// zero-padded N1 x N2 x N3 box, so each axis is transformed only for the
// lines that can be nonzero or are read: z for the H1 H2 rows of the octant,
// y for the H1 slabs, x for all lines; the upper halves of the inputs are
// zeros that are never loaded and the upper halves of the outputs are never
// stored.  The transform along x, the multiply by the kernel transform G and
// the inverse along x are one kernel (fft_x_kernel): the spectrum crosses
// memory four times in all, half the box each, where three-dimensional
// library transforms around a multiply kernel move the whole box eight times.
//
// Storage: grid [H1][H2][H3] (real, or complex for complex kernels); spectrum
// [H1][N2][KP], K = N3/2 + 1 values (real kernels) or N3 per row, rows padded
// to a multiple of 4 values (32-byte sectors).  All passes but z work in
// place on the spectrum: a CTA reads all of its lines before it writes them.
//
// One CTA of 256 threads transforms a batch of B lines (B a power of two)
// held in shared memory as [element][line], so that consecutive threads touch
// consecutive lines: Stockham passes of radix 16, 12, 10, 9, 8, 6, 5, 4, 3 and
// 2, two buffers, one barrier per pass; nearly every length up to 256 takes two
// passes, i.e. crosses shared memory once.  Along x and y, consecutive lines are
// consecutive in memory, and the first pass loads from and the last pass stores
// to global memory directly; along z the rows are loaded and stored element by element
// (coalesced) with a padded line pitch in shared memory, and real rows are
// transformed as complex ones of half the length.
#pragma once

#include "internal.h"

namespace npme {

constexpr int kFftThreads = 256;
constexpr int kFftMaxLines = 4;  // log2 of the lines per CTA at most

template <typename T>
using Cx = typename Vec2<T>::type;

template <typename T>
__device__ __forceinline__ Cx<T> cx(T a, T b) {
  Cx<T> v;
  v.x = a, v.y = b;
  return v;
}
template <typename C>
__device__ __forceinline__ C cadd(C a, C b) {
  a.x += b.x, a.y += b.y;
  return a;
}
template <typename C>
__device__ __forceinline__ C csub(C a, C b) {
  a.x -= b.x, a.y -= b.y;
  return a;
}
// a * b, or a * conj(b) for the inverse transform (twiddles are stored for
// the forward one)
template <int DIR, typename C>
__device__ __forceinline__ C ctw(C a, C b) {
  C r;
  if (DIR < 0) {
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
  } else {
    r.x = a.x * b.x + a.y * b.y;
    r.y = a.y * b.x - a.x * b.y;
  }
  return r;
}
// a * exp(DIR i pi / 2)
template <int DIR, typename C>
__device__ __forceinline__ C cmuli(C a) {
  C r;
  if (DIR < 0) r.x = a.y, r.y = -a.x;
  else r.x = -a.y, r.y = a.x;
  return r;
}

// a * exp(DIR i phi), c = cos phi, s = sin phi
template <int DIR, typename C, typename T>
__device__ __forceinline__ C crot(C a, T c, T s) {
  C r;
  r.x = a.x * c - T(DIR) * a.y * s;
  r.y = a.y * c + T(DIR) * a.x * s;
  return r;
}

template <typename T, int DIR, int R>
__device__ __forceinline__ void dft(Cx<T> (&v)[R]);

// DFT of length A B, A and B coprime, without twiddles (Good-Thomas): input
// (B n1 + A n2) mod A B, output k with k mod A = k1, k mod B = k2.
template <typename T, int DIR, int A, int B>
__device__ __forceinline__ void dft_coprime(Cx<T> (&v)[A * B]) {
  Cx<T> y[A][B];
#pragma unroll
  for (int n2 = 0; n2 < B; n2++) {
    Cx<T> t[A];
#pragma unroll
    for (int n1 = 0; n1 < A; n1++) t[n1] = v[(B * n1 + A * n2) % (A * B)];
    dft<T, DIR, A>(t);
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) y[k1][n2] = t[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; k1++) dft<T, DIR, B>(y[k1]);
#pragma unroll
  for (int k = 0; k < A * B; k++) v[k] = y[k % A][k % B];
}

// In-place DFT of R values, natural order, sign DIR.
template <typename T, int DIR, int R>
__device__ __forceinline__ void dft(Cx<T> (&v)[R]) {
  using C = Cx<T>;
  if constexpr (R == 2) {
    const C a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  } else if constexpr (R == 4) {
    const C a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]),
            d = cmuli<DIR>(csub(v[1], v[3]));
    v[0] = cadd(a, c), v[1] = cadd(b, d), v[2] = csub(a, c), v[3] = csub(b, d);
  } else if constexpr (R == 8) {
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft<T, DIR, 4>(e);
    dft<T, DIR, 4>(o);
    const T h = T(0.70710678118654752440);
    // exp(DIR i pi k / 4) o[k]
    const C o1 = cx<T>(h * (o[1].x - DIR * o[1].y), h * (o[1].y + DIR * o[1].x));
    const C o2 = cmuli<DIR>(o[2]);
    const C o3 = cx<T>(-h * (o[3].x + DIR * o[3].y), h * (DIR * o[3].x - o[3].y));
    v[0] = cadd(e[0], o[0]), v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], o1), v[5] = csub(e[1], o1);
    v[2] = cadd(e[2], o2), v[6] = csub(e[2], o2);
    v[3] = cadd(e[3], o3), v[7] = csub(e[3], o3);
  } else if constexpr (R == 3) {
    const T s = T(DIR * 0.86602540378443864676);
    const C a = cadd(v[1], v[2]), b = csub(v[1], v[2]);
    const C m = cx<T>(v[0].x - T(0.5) * a.x, v[0].y - T(0.5) * a.y);
    v[0] = cadd(v[0], a);
    v[1] = cx<T>(m.x - s * b.y, m.y + s * b.x);
    v[2] = cx<T>(m.x + s * b.y, m.y - s * b.x);
  } else if constexpr (R == 6) {
    dft_coprime<T, DIR, 2, 3>(v);
  } else if constexpr (R == 10) {
    dft_coprime<T, DIR, 2, 5>(v);
  } else if constexpr (R == 12) {
    dft_coprime<T, DIR, 4, 3>(v);
  } else if constexpr (R == 9) {
    // exp(i 2 pi m / 9), m = 1, 2, 4
    const T c[3] = {T(0.76604444311897803520), T(0.17364817766693034885),
                    T(-0.93969262078590838405)};
    const T s[3] = {T(0.64278760968653932632), T(0.98480775301220805937),
                    T(0.34202014332566873304)};
    C y[3][3];
#pragma unroll
    for (int n = 0; n < 3; n++) {
      C t[3] = {v[n], v[n + 3], v[n + 6]};
      dft<T, DIR, 3>(t);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int m = n * k;
        y[k][n] = m == 0 ? t[k] : crot<DIR>(t[k], c[m == 4 ? 2 : m - 1], s[m == 4 ? 2 : m - 1]);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      dft<T, DIR, 3>(y[k]);
#pragma unroll
      for (int n = 0; n < 3; n++) v[k + 3 * n] = y[k][n];
    }
  } else if constexpr (R == 16) {
    const T h = T(0.70710678118654752440), a = T(0.92387953251128675613),
            b = T(0.38268343236508977173);
    // exp(i pi m / 8), m = 1, 2, 3, 4, 6, 9
    const T c[10] = {1, a, h, b, 0, 0, -h, 0, 0, -a}, s[10] = {0, b, h, a, 1, 0, h, 0, 0, -b};
    C y[4][4];
#pragma unroll
    for (int n = 0; n < 4; n++) {
      C t[4] = {v[n], v[n + 4], v[n + 8], v[n + 12]};
      dft<T, DIR, 4>(t);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int m = n * k;
        y[k][n] = m == 0 ? t[k] : m == 4 ? cmuli<DIR>(t[k]) : crot<DIR>(t[k], c[m], s[m]);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      dft<T, DIR, 4>(y[k]);
#pragma unroll
      for (int n = 0; n < 4; n++) v[k + 4 * n] = y[k][n];
    }
  } else {
    static_assert(R == 5, "radix 2-6, 8-10, 12 or 16");
    const T c1 = T(0.30901699437494742410), c2 = T(-0.80901699437494742410);
    const T s1 = T(DIR * 0.95105651629515357212), s2 = T(DIR * 0.58778525229247312917);
    const C a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
    const C a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
    const C m1 = cx<T>(v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y);
    const C m2 = cx<T>(v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y);
    const C n1 = cx<T>(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y);
    const C n2 = cx<T>(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y);
    v[0] = cadd(v[0], cadd(a1, a2));
    v[1] = cx<T>(m1.x - n1.y, m1.y + n1.x), v[4] = cx<T>(m1.x + n1.y, m1.y - n1.x);
    v[2] = cx<T>(m2.x - n2.y, m2.y + n2.x), v[3] = cx<T>(m2.x + n2.y, m2.y - n2.x);
  }
}

// Largest radix first; even radices only where half of the line is zero or
// unwanted (HIN, HOUT below).
#define NPME_FFT_EVEN(CASE) CASE(16) CASE(12) CASE(10) CASE(8) CASE(6) CASE(4) CASE(2)
#define NPME_FFT_ALL(CASE) NPME_FFT_EVEN(CASE) CASE(9) CASE(5) CASE(3)

// One Stockham pass over a line: butterfly j reads elements j + r N/R and
// writes (j / Ns) Ns R + j mod Ns + r Ns; element n is at src[n ss], dst[n ds].
// HIN (first pass): the elements from N/2 on are zeros that are not read.  HOUT
// (last pass): those from N/2 on are not written.  Both are half of the
// butterfly's values for an even radix, known at compile time.
template <typename T, int DIR, int R, bool HIN, bool HOUT, class SS, class DS>
__device__ __forceinline__ void fft_pass_r(const FftPass &p, int N, int j0, int dj, const Cx<T> *tw,
                                           const Cx<T> *src, SS ss, Cx<T> *dst, DS ds) {
  static_assert(R % 2 == 0 || (!HIN && !HOUT), "even radix");
  const int nb = N / R;
  for (int j = j0; j < nb; j += dj) {
    const int q = p.Ns == 1 ? j : (int)__umulhi((unsigned)j, p.magic), k = j - q * p.Ns;
    Cx<T> v[R];
    const Cx<T> *in = src + j * ss;
    const SS sstep = nb * ss;
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (HIN && r >= R / 2) {
        v[r] = Cx<T>{};
      } else {
        v[r] = *in;
        in += sstep;
      }
    }
    if (!HIN && p.Ns > 1) {
      const Cx<T> *t = tw;
      const int step = k * p.step;
#pragma unroll
      for (int r = 1; r < R; r++) {
        t += step;
        v[r] = ctw<DIR>(v[r], *t);
      }
    }
    dft<T, DIR, R>(v);
    Cx<T> *out = dst + (q * p.Ns * R + k) * ds;
    const DS dstep = p.Ns * ds;
#pragma unroll
    for (int r = 0; r < (HOUT ? R / 2 : R); r++) {
      *out = v[r];
      out += dstep;
    }
  }
}

template <typename T, int DIR, bool HIN, bool HOUT, class SS, class DS>
__device__ __forceinline__ void fft_pass(const FftPass &p, int N, int j0, int dj, const Cx<T> *tw,
                                         const Cx<T> *src, SS ss, Cx<T> *dst, DS ds) {
#define NPME_FFT_CASE(RR) \
  case RR: fft_pass_r<T, DIR, RR, HIN, HOUT>(p, N, j0, dj, tw, src, ss, dst, ds); break;
  if constexpr (HIN || HOUT) {
    switch (p.R) { NPME_FFT_EVEN(NPME_FFT_CASE) }
  } else {
    switch (p.R) { NPME_FFT_ALL(NPME_FFT_CASE) }
  }
#undef NPME_FFT_CASE
}

// The last forward pass, a pointwise multiply and the first inverse pass in
// registers: the last pass (Ns = N / R) of butterfly j writes elements j + r
// N/R, which are the ones that the first pass of a transform with radix R
// reads for its butterfly j.  mul(n, v): the product at element n.
template <typename T, int R, class Mul>
__device__ __forceinline__ void fft_turn_r(const FftPass &p, int N, int j0, int dj,
                                           const Cx<T> *tw, const Cx<T> *src, Cx<T> *dst,
                                           int pitch, const Mul &mul) {
  const int nb = N / R;
  for (int j = j0; j < nb; j += dj) {
    Cx<T> v[R];
    const Cx<T> *in = src + j * pitch, *t = tw;
    const int sstep = nb * pitch, step = j * p.step;
#pragma unroll
    for (int r = 0; r < R; r++) {
      v[r] = *in;
      in += sstep;
    }
#pragma unroll
    for (int r = 1; r < R; r++) {
      t += step;
      v[r] = ctw<-1>(v[r], *t);
    }
    dft<T, -1, R>(v);
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = mul(j + r * nb, v[r]);
    dft<T, 1, R>(v);
    Cx<T> *out = dst + j * R * pitch;
#pragma unroll
    for (int r = 0; r < R; r++) {
      *out = v[r];
      out += pitch;
    }
  }
}

template <typename T, class Mul>
__device__ __forceinline__ void fft_turn(const FftPass &p, int N, int j0, int dj,
                                         const Cx<T> *tw, const Cx<T> *src, Cx<T> *dst, int pitch,
                                         const Mul &mul) {
#define NPME_FFT_CASE(RR) \
  case RR: fft_turn_r<T, RR>(p, N, j0, dj, tw, src, dst, pitch, mul); break;
  switch (p.R) { NPME_FFT_ALL(NPME_FFT_CASE) }
#undef NPME_FFT_CASE
}

// Passes [from, to) of a transform in shared memory (the thread's line at cur,
// the other buffer at other), a barrier after each; returns the buffer that
// holds the result.  Dead lines only meet the barriers.
template <typename T, int DIR>
__device__ __forceinline__ Cx<T> *fft_middle(const FftAxis &a, int from, int to, int j0, int dj,
                                             const Cx<T> *tw, Cx<T> *cur, Cx<T> *other, int pitch,
                                             bool live = true) {
  for (int i = from; i < to; i++) {
    if (live) fft_pass<T, DIR, false, false>(a.p[i], a.N, j0, dj, tw, cur, pitch, other, pitch);
    __syncthreads();
    Cx<T> *t = cur;
    cur = other;
    other = t;
  }
  return cur;
}

template <typename T>
__device__ __forceinline__ void load_twiddles(const FftAxis &a, Cx<T> *tw) {
  const Cx<T> *g = static_cast<const Cx<T> *>(a.tw);
  for (int i = threadIdx.x; i < a.twlen; i += kFftThreads) tw[i] = g[i];
}

// Lines along y (DIR: forward from H2 to N2 elements, inverse from N2 to H2)
// in place on the spectrum; unit u: lines u B ... of the H1 KP lines.
template <typename T, int DIR>
__device__ __forceinline__ void fft_y_body(const FftJob &J, long u, unsigned char *smem) {
  using C = Cx<T>;
  const FftAxis &a = DIR < 0 ? J.y : J.yi;
  const int B = 1 << a.lb;
  C *tw = reinterpret_cast<C *>(smem), *s0 = tw + a.twlen, *s1 = s0 + (long)a.N * B;
  const int b = threadIdx.x & (B - 1), j0 = threadIdx.x >> a.lb, dj = kFftThreads >> a.lb;
  const int line = (int)(u << a.lb) + b;
  const int x = line / J.KP, k = line - x * J.KP;
  const bool live = x < J.H[0] && k < J.K;
  C *g = static_cast<C *>(J.spec) + (long)x * J.N[1] * J.KP + k;
  const long st = J.KP;
  load_twiddles<T>(a, tw);
  if (live) fft_pass<T, DIR, DIR<0, false>(a.p[0], a.N, j0, dj, tw, g, st, s0 + b, B);
  __syncthreads();
  const C *in = fft_middle<T, DIR>(a, 1, a.np - 1, j0, dj, tw, s0 + b, s1 + b, B, live);
  if (live) fft_pass<T, DIR, false, (DIR > 0)>(a.p[a.np - 1], a.N, j0, dj, tw, in, B, g, st);
}

// Lines along x: forward, times G, inverse, in place on the spectrum; unit
// u: lines u B ... of the N2 KP lines.  The inverse runs the forward's radices
// in reverse order (J.xi).  CPLX: complex kernel.
template <typename T, bool CPLX>
__device__ __forceinline__ void fft_x_body(const FftJob &J, long u, unsigned char *smem) {
  using C = Cx<T>;
  const FftAxis &a = J.x, &ai = J.xi;
  const int B = 1 << a.lb;
  C *tw = reinterpret_cast<C *>(smem), *s0 = tw + a.twlen, *s1 = s0 + (long)a.N * B;
  const int b = threadIdx.x & (B - 1), j0 = threadIdx.x >> a.lb, dj = kFftThreads >> a.lb;
  const int line = (int)(u << a.lb) + b;
  const int N1 = J.N[0], N2 = J.N[1], N3 = J.N[2];
  const int k2 = line / J.KP, k3 = line - k2 * J.KP;
  const bool live = k2 < N2 && k3 < J.K;
  C *g = static_cast<C *>(J.spec) + line;
  const long st = (long)N2 * J.KP;
  const int M2 = N2 / 2 + 1, M3 = N3 / 2 + 1;
  const int f2 = min(k2, N2 - k2), f3 = min(k3, N3 - k3);
  const long gst = (long)M2 * M3;
  using GT = typename std::conditional<CPLX, C, T>::type;
  const GT *G = static_cast<const GT *>(J.G) + ((long)f2 * M3 + f3);  // read for live lines
  load_twiddles<T>(a, tw);
  if (live) fft_pass<T, -1, true, false>(a.p[0], N1, j0, dj, tw, g, st, s0 + b, B);
  __syncthreads();
  C *cur = fft_middle<T, -1>(a, 1, a.np - 1, j0, dj, tw, s0 + b, s1 + b, B, live);
  C *out = cur == s0 + b ? s1 + b : s0 + b;
  if (live)
    fft_turn<T>(a.p[a.np - 1], N1, j0, dj, tw, cur, out, B, [=](int n, C v) {
      const GT w = G[min(n, N1 - n) * gst];
      if constexpr (CPLX) return cx<T>(v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x);
      else return cx<T>(v.x * w, v.y * w);
    });
  __syncthreads();
  const C *in = fft_middle<T, 1>(ai, 1, ai.np - 1, j0, dj, tw, out, cur, B, live);
  if (live) fft_pass<T, 1, false, true>(ai.p[ai.np - 1], N1, j0, dj, tw, in, B, g, st);
}

// Rows along z; unit u: rows u B ... of the H1 H2 rows.  Forward: the grid's
// row (H3 values) to the spectrum's (K values); inverse: back.  Real kernels
// transform the row as H3 complex values (x_2j, x_2j+1): with Z their
// transform and w = exp(-2 pi i k / N3), X_k = (Z_k + Z*_{H-k}) / 2 - i w
// (Z_k - Z*_{H-k}) / 2, and back Z_k = X_k + X*_{H-k} + i w* (X_k - X*_{H-k}).
template <typename T, bool CPLX, int DIR>
__device__ __forceinline__ void fft_z_body(const FftJob &J, long u, unsigned char *smem) {
  using C = Cx<T>;
  __shared__ long srow[1 << kFftMaxLines];   // the rows' places in the spectrum
  const FftAxis &a = DIR < 0 ? J.z : J.zi;  // length N3 (complex kernels) or H3
  const int B = 1 << a.lb, P = B + 1, L = a.N, H3 = J.H[2];
  C *tw = reinterpret_cast<C *>(smem), *s0 = tw + a.twlen, *s1 = s0 + (long)(L + 1) * P;
  const int b = threadIdx.x & (B - 1), j0 = threadIdx.x >> a.lb, dj = kFftThreads >> a.lb;
  const int row0 = (int)(u << a.lb), rows = min(B, J.H[0] * J.H[1] - row0);
  const bool live = b < rows;
  // grid rows as complex values: H3 (complex kernels) or H3 / 2 pairs
  const int gl = CPLX ? H3 : H3 / 2;
  C *grid = static_cast<C *>(J.grid) + (long)row0 * gl, *spec = static_cast<C *>(J.spec);
  if (threadIdx.x < rows) {
    const int row = row0 + threadIdx.x, x = row / J.H[1];
    srow[threadIdx.x] = ((long)x * J.N[1] + (row - x * J.H[1])) * J.KP;
  }
  load_twiddles<T>(a, tw);
  // element i of row r of the batch -> (r, i), i fastest
  auto sweep = [&](int len, auto f) {
    const unsigned m = 0xffffffffu / (unsigned)len + 1;  // ceil(2^32 / len), len > 1
    for (int t = threadIdx.x; t < len * rows; t += kFftThreads) {
      const int r = (int)__umulhi((unsigned)t, m);
      f(r, t - r * len, t);
    }
  };
  if (DIR < 0) {
    // the rows are contiguous in the grid
    sweep(gl, [&](int r, int i, int t) { s0[i * P + r] = grid[t]; });
    __syncthreads();
    if (live) fft_pass<T, -1, true, false>(a.p[0], L, j0, dj, tw, s0 + b, P, s1 + b, P);
    __syncthreads();
    const C *Z = fft_middle<T, -1>(a, 1, a.np, j0, dj, tw, s1 + b, s0 + b, P, live) - b;
    if (CPLX) {
      sweep(L, [&](int r, int k, int) { spec[srow[r] + k] = Z[k * P + r]; });
    } else {
      sweep(L + 1, [&](int r, int k, int) {
        const C z = Z[(k == L ? 0 : k) * P + r], m = Z[(k == 0 ? 0 : L - k) * P + r];
        const C e = cx<T>(T(0.5) * (z.x + m.x), T(0.5) * (z.y - m.y));
        const C d = cx<T>(T(0.5) * (z.x - m.x), T(0.5) * (z.y + m.y));
        const C w = tw[k];  // table of the length-N3 transform
        // -i w d
        const C wd = cx<T>(w.x * d.x - w.y * d.y, w.x * d.y + w.y * d.x);
        spec[srow[r] + k] = cx<T>(e.x + wd.y, e.y - wd.x);
      });
    }
  } else {
    __syncthreads();
    if (CPLX) {
      sweep(L, [&](int r, int k, int) { s0[k * P + r] = spec[srow[r] + k]; });
    } else {
      sweep(L + 1, [&](int r, int k, int) { s1[k * P + r] = spec[srow[r] + k]; });
      __syncthreads();
      sweep(L, [&](int r, int k, int) {
        const C z = s1[k * P + r], m = s1[(L - k) * P + r];
        const C e = cx<T>(z.x + m.x, z.y - m.y), d = cx<T>(z.x - m.x, z.y + m.y);
        const C w = tw[k];
        // i w* d
        const C wd = cx<T>(w.x * d.x + w.y * d.y, w.x * d.y - w.y * d.x);
        s0[k * P + r] = cx<T>(e.x - wd.y, e.y + wd.x);
      });
    }
    __syncthreads();
    C *in = fft_middle<T, 1>(a, 0, a.np - 1, j0, dj, tw, s0 + b, s1 + b, P, live);
    C *out = in == s0 + b ? s1 + b : s0 + b;
    if (live) fft_pass<T, 1, false, true>(a.p[a.np - 1], L, j0, dj, tw, in, P, out, P);
    __syncthreads();
    const C *Z = out - b;
    sweep(gl, [&](int r, int i, int t) { grid[t] = Z[i * P + r]; });
  }
}

}  // namespace npme
