// rgf_gw_fft.cu -- FFT form of the GW loop's energy convolutions, as the
// production loop with energy <-> (i,j) redistribution computes them
// (green_rgf_solve_gw_ephoton_3d_ijs, src/green_rgf.f90:1397-1473 for the
// polarization, :1598-1678 for the self-energy; corr1d2 / conv1d2 with
// method 'fft', src/fft_mod.f90:56-89, :175-212, each a zero-padded
// circular convolution by do_mkl_dfti_conv, :214-234).
//
// The reference forms, for every banded (i,j) element and block ix, one
// length-(2n-1) FFT correlation per (k, q) pair and sums them over k.  Here
// the sums over k move into frequency space: per (i,j, ix) "line" the
// (ky, kz, energy) array of each operand gets one 3-D FFT (energy axis
// zero-padded to N >= 2n-1 with no prime factor above 7), the k - q index
// ikd = k - q + nk/2 - 1 (mod nk) per axis makes the k sums circular
// correlations (P) or convolutions (Sigma) over the k-grid, so
//   P^(p)     = X^(p) Y^(-p) exp(-2 pi i p.s/nk) / (nk N) * dE_P
//   Sigma^(p) = G^(p) W^(p)  exp(+2 pi i p.s/nk) / (nk N) * dE_S
// and one inverse 3-D FFT per output gives every q (or k) at once.  The
// window read back is the 'fft' paths' one: P(p) at energy shift
// b = p - 1 - n/2, Sigma(e) from W placed at nop = -(n/2-1) .. n/2-1.
//
// Up to nen = 4096 (N = 8192) the transforms are this library's own, and the
// energy axis never leaves the SM between transform, product and inverse:
//   k_forward   the k-grid transform of every operand (nen values a line and
//               k, before any padding), one read and one write;
//   line_*      per (line, k-frequency): the energy transforms of all operands
//               one after another (registers + one shared buffer,
//               rgf_fft_smem.cuh), the products, the inverse transforms and
//               the window; spectra that wait for a partner go to scratch of
//               the resident CTAs (L2);
//   k_inverse   the inverse k-grid transform of the windows with the phases.
// Longer axes, and k-grids for which own_log finds it faster, take the form
// below it: cuFFT's 3-D transforms (Z2Z, batched, stream-ordered) with separate packing,
// product and window kernels.
//
// Arrays: the *_by_blocks layout (nen, nk, nx, nij) complex(8) on the device,
// energy fastest, ik = ikz + nkz (iky) (0-based).  nen must be even.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <vector>

#include "rgf_fft_cache.h"
#include "rgf_fft_smem.cuh"
#include "rgf_internal.h"

namespace {

thread_local char g_fft_err[256];

int fft_fail(int code, const char* msg) {
  std::snprintf(g_fft_err, sizeof(g_fft_err), "%s", msg);
  return code;
}

// smallest m' >= m with no prime factor above 7
int64_t nice_length(int64_t m) {
  for (int64_t n = m;; n++) {
    int64_t r = n;
    for (int64_t p : {2, 3, 5, 7})
      while (r % p == 0) r /= p;
    if (r == 1) return n;
  }
}

struct Dims {
  int64_t nen, nky, nkz, nk, N;
};

// buf[b][k][m] (m < N) from line lines[b] of A: mode 0 the series zero-padded,
// mode 1 its conjugate, mode 2 W placed by energy shift (nop = m for
// m < n/2, nop = m - N for m >= N - (n/2 - 1); W index nop + n/2 - 1).
__global__ void pack_kernel(const double2* __restrict__ A, const int64_t* __restrict__ lines, int64_t nlines,
                            Dims d, int mode, double2* __restrict__ buf) {
  const int64_t total = nlines * d.nk * d.N;
  const int64_t h = d.nen / 2;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = t % d.N, r = t / d.N;
    const int64_t k = r % d.nk, b = r / d.nk;
    const double2* src = A + (lines[b] * d.nk + k) * d.nen;
    double2 v = make_double2(0.0, 0.0);
    if (mode == 2) {
      if (m < h) v = src[m + h - 1];
      else if (m >= d.N - (h - 1)) v = src[m - d.N + h - 1];
    } else if (m < d.nen) {
      v = src[m];
      if (mode == 1) v.y = -v.y;
    }
    buf[t] = v;
  }
}

__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 ca(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// P in frequency space, in place over the x-side buffers:
//   xl <- ph (xl ygt~),  xg <- ph (xg ylt~),  xr <- ph (xl ycr~ + xr ylt~)
// with y~ the y-side spectra at negated (ky, kz, energy) frequencies and
// ph[k] the shift phase times the normalisation and dE.
__global__ void corr_freq_kernel(double2* __restrict__ xl, double2* __restrict__ xg, double2* __restrict__ xr,
                                 const double2* __restrict__ ygt, const double2* __restrict__ ylt,
                                 const double2* __restrict__ ycr, const double2* __restrict__ ph, int64_t nlines,
                                 Dims d) {
  const int64_t total = nlines * d.nk * d.N;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = t % d.N, r = t / d.N;
    const int64_t k = r % d.nk, b = r / d.nk;
    const int64_t ky = k / d.nkz, kz = k % d.nkz;
    const int64_t kn = ((d.nky - ky) % d.nky) * d.nkz + (d.nkz - kz) % d.nkz;
    const int64_t tn = (b * d.nk + kn) * d.N + (d.N - m) % d.N;
    const double2 p = ph[k];
    const double2 a = xl[t], g = xg[t], rr = xr[t];
    const double2 yl = ylt[tn];
    xl[t] = cm(p, cm(a, ygt[tn]));
    xg[t] = cm(p, cm(g, yl));
    xr[t] = cm(p, ca(cm(a, ycr[tn]), cm(rr, yl)));
  }
}

// Sigma in frequency space, in place over the G-side buffers:
//   gl <- ph gl wl,  gg <- ph gg wg,  gr <- ph (gl wr + gr wl + gr wr)
__global__ void conv_freq_kernel(double2* __restrict__ gl, double2* __restrict__ gg, double2* __restrict__ gr,
                                 const double2* __restrict__ wl, const double2* __restrict__ wg,
                                 const double2* __restrict__ wr, const double2* __restrict__ ph, int64_t nlines,
                                 Dims d) {
  const int64_t total = nlines * d.nk * d.N;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = (t / d.N) % d.nk;
    const double2 p = ph[k];
    const double2 a = gl[t], g = gg[t], rr = gr[t], l = wl[t], w = wr[t];
    gl[t] = cm(p, cm(a, l));
    gg[t] = cm(p, cm(g, wg[t]));
    gr[t] = cm(p, ca(ca(cm(a, w), cm(rr, l)), cm(rr, w)));
  }
}

// outputs of the lines of a chunk: P(o) = buf[(o - n/2) mod N] (mode 0) or
// Sigma(e) = buf[e] with Sigma^R = (Re, Im(Sigma^> - Sigma^<) / 2) (mode 1)
__global__ void unpack_kernel(const double2* __restrict__ b0, const double2* __restrict__ b1,
                              const double2* __restrict__ b2, const int64_t* __restrict__ lines, int64_t nlines,
                              Dims d, int mode, double2* __restrict__ o0, double2* __restrict__ o1,
                              double2* __restrict__ o2) {
  const int64_t total = nlines * d.nk * d.nen;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = t % d.nen, r = t / d.nen;
    const int64_t k = r % d.nk, b = r / d.nk;
    const int64_t src = (b * d.nk + k) * d.N +
                        (mode == 0 ? ((e - d.nen / 2) % d.N + d.N) % d.N : e);
    const int64_t dst = (lines[b] * d.nk + k) * d.nen + e;
    const double2 v0 = b0[src], v1 = b1[src];
    double2 v2 = b2[src];
    if (mode == 1) v2.y = (v1.y - v0.y) / 2.0;
    o0[dst] = v0;
    o1[dst] = v1;
    o2[dst] = v2;
  }
}

// ------------------------------------------------------------ own transforms
namespace own {

using rgf::fft::add;
using rgf::fft::mul;
using rgf::fft::mulc;

constexpr int kMinLog = 5, kMaxLog = 12;   // log2 of M, half the circular length

// DFT of x[0], x[S], ... (L values), exp(-2 pi i) forward, + inverse.
template <int L, int S, bool INV>
__device__ __forceinline__ void dft_small(double2* x) {
  if constexpr (L == 2) {
    const double2 a = x[0], b = x[S];
    x[0] = add(a, b);
    x[S] = rgf::fft::sub(a, b);
  } else if constexpr (L == 4) {
    rgf::fft::dft4<INV>(x[0], x[S], x[2 * S], x[3 * S]);
  }
}

template <int NKY, int NKZ, bool INV>
__device__ __forceinline__ void dft_k(double2 (&x)[NKY * NKZ]) {
#pragma unroll
  for (int y = 0; y < NKY; y++) dft_small<NKZ, 1, INV>(x + y * NKZ);
#pragma unroll
  for (int z = 0; z < NKZ; z++) dft_small<NKY, NKZ, INV>(x + z);
}

struct Six {
  const double2* a[6];
};
struct Three {
  double2* a[3];
};

// k-grid transform of operand blockIdx.z of the lines of a chunk into
// kb[op][line][k][energy]; bit op of `conj`: of its conjugate.  One thread an
// energy with its nk values in registers: bound by one read and one write.
template <int NKY, int NKZ>
__global__ void __launch_bounds__(256) k_forward(Six in, const int64_t* __restrict__ lines, int64_t nl, Dims d,
                                                 unsigned conj, double2* __restrict__ kb) {
  constexpr int NK = NKY * NKZ;
  const int op = blockIdx.z;
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x, b = blockIdx.y;
  if (e >= d.nen) return;
  const double2* src = in.a[op] + lines[b] * NK * d.nen + e;
  double2* dst = kb + ((size_t)op * nl + b) * NK * d.nen + e;
  const double sg = (conj >> op) & 1 ? -1.0 : 1.0;
  double2 x[NK];
#pragma unroll
  for (int k = 0; k < NK; k++) {
    const double2 v = src[k * d.nen];
    x[k] = make_double2(v.x, sg * v.y);
  }
  dft_k<NKY, NKZ, false>(x);
#pragma unroll
  for (int k = 0; k < NK; k++) dst[k * d.nen] = x[k];
}

// Windows pb[v][line][k-frequency][energy] times ph -> outputs of the lines.
// fix: Sigma^R's imaginary part is (Im Sigma^> - Im Sigma^<) / 2.
template <int NKY, int NKZ>
__global__ void __launch_bounds__(128) k_inverse(Three out, const int64_t* __restrict__ lines, int64_t nl, Dims d,
                                                 bool fix, const double2* __restrict__ ph,
                                                 const double2* __restrict__ pb) {
  constexpr int NK = NKY * NKZ;
  const int64_t e = (int64_t)blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
  if (e >= d.nen) return;
  double diff[NK];
#pragma unroll
  for (int k = 0; k < NK; k++) diff[k] = 0.0;
#pragma unroll
  for (int v = 0; v < 3; v++) {
    const double2* src = pb + ((size_t)v * nl + b) * NK * d.nen + e;
    double2* dst = out.a[v] + lines[b] * NK * d.nen + e;
    double2 x[NK];
#pragma unroll
    for (int k = 0; k < NK; k++) x[k] = mul(src[k * d.nen], ph[k]);
    dft_k<NKY, NKZ, true>(x);
#pragma unroll
    for (int k = 0; k < NK; k++) {
      if (v == 0) diff[k] = -x[k].y;
      else if (v == 1) diff[k] += x[k].y;
      else if (fix) x[k].y = diff[k] / 2.0;
      dst[k * d.nen] = x[k];
    }
  }
}

// The same two for any k-grid: a tile of 32 energies in shared memory, the
// two axes one after another as sums over the axis (tables of the nky-th and
// nkz-th roots behind the ph table).
constexpr int kTileE = 32;
__device__ __forceinline__ void dft_tile(double2* cur, double2* nxt, const double2* wy, const double2* wz, int nky,
                                         int nkz, bool inv) {
  const int nk = nky * nkz;
  for (int q = threadIdx.x; q < nk * kTileE; q += blockDim.x) {   // along kz
    const int e = q % kTileE, k = q / kTileE, y = k / nkz, z = k % nkz;
    double2 a = make_double2(0.0, 0.0);
    for (int i = 0; i < nkz; i++) {
      const double2 w = wz[(i * z) % nkz], v = cur[(y * nkz + i) * kTileE + e];
      a = add(a, inv ? mulc(v, w) : mul(v, w));
    }
    nxt[q] = a;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nk * kTileE; q += blockDim.x) {   // along ky
    const int e = q % kTileE, k = q / kTileE, y = k / nkz, z = k % nkz;
    double2 a = make_double2(0.0, 0.0);
    for (int i = 0; i < nky; i++) {
      const double2 w = wy[(i * y) % nky], v = nxt[(i * nkz + z) * kTileE + e];
      a = add(a, inv ? mulc(v, w) : mul(v, w));
    }
    cur[q] = a;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) k_forward_any(Six in, const int64_t* __restrict__ lines, int64_t nl, Dims d,
                                                     unsigned conj, const double2* __restrict__ ph,
                                                     double2* __restrict__ kb) {
  extern __shared__ __align__(16) double2 sh[];
  const int nk = (int)d.nk, op = blockIdx.z;
  const int64_t e0 = (int64_t)blockIdx.x * kTileE, b = blockIdx.y;
  const double2* src = in.a[op] + lines[b] * nk * d.nen;
  double2* dst = kb + ((size_t)op * nl + b) * nk * d.nen;
  const double sg = (conj >> op) & 1 ? -1.0 : 1.0;
  for (int q = threadIdx.x; q < nk * kTileE; q += blockDim.x) {
    const int64_t e = e0 + q % kTileE;
    const double2 v = e < d.nen ? src[(q / kTileE) * d.nen + e] : make_double2(0.0, 0.0);
    sh[q] = make_double2(v.x, sg * v.y);
  }
  __syncthreads();
  dft_tile(sh, sh + nk * kTileE, ph + nk, ph + nk + d.nky, (int)d.nky, (int)d.nkz, false);
  for (int q = threadIdx.x; q < nk * kTileE; q += blockDim.x) {
    const int64_t e = e0 + q % kTileE;
    if (e < d.nen) dst[(q / kTileE) * d.nen + e] = sh[q];
  }
}

__global__ void __launch_bounds__(256) k_inverse_any(Three out, const int64_t* __restrict__ lines, int64_t nl, Dims d,
                                                     bool fix, const double2* __restrict__ ph,
                                                     const double2* __restrict__ pb) {
  extern __shared__ __align__(16) double2 sh[];
  const int nk = (int)d.nk;
  double* diff = (double*)(sh + 2 * nk * kTileE);
  const int64_t e0 = (int64_t)blockIdx.x * kTileE, b = blockIdx.y;
  for (int v = 0; v < 3; v++) {
    const double2* src = pb + ((size_t)v * nl + b) * nk * d.nen;
    double2* dst = out.a[v] + lines[b] * nk * d.nen;
    for (int q = threadIdx.x; q < nk * kTileE; q += blockDim.x) {
      const int64_t e = e0 + q % kTileE;
      sh[q] = e < d.nen ? mul(src[(q / kTileE) * d.nen + e], ph[q / kTileE]) : make_double2(0.0, 0.0);
    }
    __syncthreads();
    dft_tile(sh, sh + nk * kTileE, ph + nk, ph + nk + d.nky, (int)d.nky, (int)d.nkz, true);
    for (int q = threadIdx.x; q < nk * kTileE; q += blockDim.x) {
      const int64_t e = e0 + q % kTileE;
      double2 x = sh[q];
      if (v == 0) diff[q] = -x.y;
      else if (v == 1) diff[q] += x.y;
      else if (fix) x.y = diff[q] / 2.0;
      if (e < d.nen) dst[(q / kTileE) * d.nen + e] = x;
    }
    __syncthreads();
  }
}

// Energy transforms, products and windows of (line, k-frequency) tasks.
// The circular length is N = 2 M with M = 2^LOGM >= nen, and a task does its
// even and its odd frequencies one after the other, each a problem of length
// M: X[2f] is the M-point transform of x[n] + x[n + M], X[2f + 1] that of
// (x[n] - x[n + M]) exp(-2 pi i n / N), and the result is E[n] +- exp(2 pi i
// n / N) O[n] (n < M, n + M), of which the window needs one sign per n.  The
// padding is then never transformed, M = 4096 takes two exchanges instead of
// the three of 8192, and two CTAs fit an SM, so one exchanges while the other
// computes.  Measured (1 B200, nen = 4096, 4 x 4 k-grid, 140 lines, P and
// Sigma): cuFFT's 3-D form 9.8 ms; own transforms of N = 8192, one CTA an SM
// 5.1 ms (these kernels 3.2 of it, the zeros outside the band 1.2); halves of
// M = 4096 with the zeros written beside them 4.5 ms.
//
// NT = M / 16 threads a task, G tasks side by side in a CTA of at least 128
// threads.  kb: operands [op][line][k][energy]; pb: windows [v][line][k]
// [energy]; scr: three half spectra for each task in work (L2).  The
// conjugate of the correlation's second operands was transformed, so their
// spectra at negated frequencies are conjugates at the same ones:
//   P^< = G^< conj(Y^>),  P^> = G^> conj(Y^<),
//   P^R = G^< conj(G^R) + G^R conj(Y^<)      (the second operand conj(G^R))
// and Sigma^R = G^< W^R + G^R (W^< + W^R).  Operands: P: G^<, G^>, G^R, Y^>,
// Y^<; Sigma: G^<, G^>, G^R, W^<, W^>, W^R.
// w: the twiddle table, w2: exp(-2 pi i n / N), n < M.
template <int LOGM>
struct Line {
  using C = rgf::fft::Cfg<LOGM>;
  static constexpr int kThreads = C::NT < 128 ? 128 : C::NT;
  static constexpr int G = kThreads / C::NT;
  static constexpr int kPerSm = 512 / kThreads;         // 128 registers a thread
  static constexpr size_t smem = sizeof(double2) * G * C::SMEM;
};

template <int LOGM, int MODE>
__global__ void __launch_bounds__(Line<LOGM>::kThreads, Line<LOGM>::kPerSm)
line_kernel(int64_t nl, Dims d, const double2* __restrict__ w, const double2* __restrict__ w2,
            const double2* __restrict__ kb, double2* __restrict__ pb, double2* __restrict__ scr) {
  using C = rgf::fft::Cfg<LOGM>;
  constexpr int M = C::M, NT = C::NT, G = Line<LOGM>::G;
  extern __shared__ __align__(16) double2 sh[];
  const int grp = threadIdx.x / NT, t = threadIdx.x % NT;
  double2* buf = sh + grp * C::SMEM;
  double2* s1 = scr + ((size_t)blockIdx.x * G + grp) * 3 * M + t;
  double2 *s2 = s1 + M, *s3 = s2 + M;
  const int nen = (int)d.nen, h = nen / 2;
  const int64_t total = nl * d.nk, op_stride = total * nen;
  const double2 zero = make_double2(0.0, 0.0);
  double2 x[16];
  for (int64_t base = (int64_t)blockIdx.x * G; base < total; base += (int64_t)gridDim.x * G) {
    const int64_t task = base + grp;
    const bool on = task < total;
    const double2* in = kb + task * nen;
    double2* out = pb + task * nen;
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
      auto load = [&](int op, bool shifted) {
        const double2* src = in + op * op_stride;
#pragma unroll
        for (int m = 0; m < 16; m++) {
          const int i = t + NT * m;
          double2 v = zero;
          if (!shifted) {              // a series, zero-padded
            if (on && i < nen) v = __ldcg(src + i);
          } else if (i < h) {          // W by its energy shift: n >= 0 first,
            if (on) v = __ldcg(src + i + h - 1);
          } else if (i > M - h) {      // n < 0 at the end of N (x[n + M])
            if (on) v = __ldcg(src + i - M + h - 1);
            if (half) v = make_double2(-v.x, -v.y);
          }
          x[m] = v;
        }
        if (half)
#pragma unroll
          for (int m = 0; m < 16; m++) x[m] = mul(x[m], w2[t + NT * m]);
      };
      auto keep = [&](double2* s) {
#pragma unroll
        for (int m = 0; m < 16; m++) __stcg(s + NT * m, x[m]);
      };
      // one transform of each direction in the code: a loop over the operands
#pragma unroll 1
      for (int step = 0; step < (MODE == 0 ? 5 : 6); step++) {
        int v = -1;                    // output of this step
        if constexpr (MODE == 0) {
          load(step == 0 ? 4 : (step == 1 ? 1 : (step == 2 ? 2 : (step == 3 ? 0 : 3))), false);
          rgf::fft::transform<LOGM, false>(x, buf, w, t);
          if (step == 0) {
            keep(s1);                  // Y^<
          } else if (step == 1) {
#pragma unroll
            for (int m = 0; m < 16; m++) x[m] = mulc(x[m], __ldcg(s1 + NT * m));
            v = 1;
          } else if (step == 2) {
            keep(s2);                  // G^R
          } else if (step == 3) {
            keep(s3);                  // G^<
#pragma unroll
            for (int m = 0; m < 16; m++) {
              const double2 gr = __ldcg(s2 + NT * m);
              x[m] = add(mulc(x[m], gr), mulc(gr, __ldcg(s1 + NT * m)));
            }
            v = 2;
          } else {
#pragma unroll
            for (int m = 0; m < 16; m++) x[m] = mulc(__ldcg(s3 + NT * m), x[m]);
            v = 0;
          }
        } else {
          load(step == 0 ? 4 : (step == 1 ? 1 : (step == 2 ? 3 : (step == 3 ? 5 : (step == 4 ? 0 : 2)))),
               step == 0 || step == 2 || step == 3);
          rgf::fft::transform<LOGM, false>(x, buf, w, t);
          if (step == 0 || step == 2) {
            keep(s1);                  // W^>, then W^<
          } else if (step == 1) {
#pragma unroll
            for (int m = 0; m < 16; m++) x[m] = mul(x[m], __ldcg(s1 + NT * m));
            v = 1;
          } else if (step == 3) {
            keep(s2);                  // W^R
          } else if (step == 4) {
            keep(s3);                  // G^<
#pragma unroll
            for (int m = 0; m < 16; m++) x[m] = mul(x[m], __ldcg(s1 + NT * m));
            v = 0;
          } else {
#pragma unroll
            for (int m = 0; m < 16; m++) {
              const double2 wr = __ldcg(s2 + NT * m);
              x[m] = add(mul(__ldcg(s3 + NT * m), wr), mul(x[m], add(__ldcg(s1 + NT * m), wr)));
            }
            v = 2;
          }
        }
        if (v < 0) continue;
        rgf::fft::transform<LOGM, true>(x, buf, w, t);
        if (!on) continue;
        double2* dst = out + v * op_stride;
#pragma unroll
        for (int m = 0; m < 16; m++) {
          const int i = t + NT * m;
          // P(o): energy shift o - h, negative ones at n + M (minus sign)
          const bool up = MODE == 0 && i >= M - h;
          const int o = MODE == 1 ? i : (up ? i - (M - h) : (i < h ? i + h : nen));
          if (o >= nen) continue;
          if (half == 0) {
            __stcg(dst + o, x[m]);
          } else {
            const double2 e = __ldcg(dst + o), q = mulc(x[m], w2[i]);
            __stcg(dst + o, up ? rgf::fft::sub(e, q) : add(e, q));
          }
        }
      }
    }
  }
}

}  // namespace own

struct Plan {
  cufftHandle h = 0;
  bool created = false, ok = false;
  Plan(const Dims& d, int64_t batch, cudaStream_t st) {
    int n[3], rank = 0;
    if (d.nky > 1) n[rank++] = (int)d.nky;
    if (d.nkz > 1) n[rank++] = (int)d.nkz;
    n[rank++] = (int)d.N;
    created = cufftPlanMany(&h, rank, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_Z2Z, (int)batch) == CUFFT_SUCCESS;
    ok = created && cufftSetStream(h, st) == CUFFT_SUCCESS;
  }
  ~Plan() { if (created) cufftDestroy(h); }
  bool run(double2* buf, int dir) const {
    return cufftExecZ2Z(h, (cufftDoubleComplex*)buf, (cufftDoubleComplex*)buf, dir) == CUFFT_SUCCESS;
  }
};

// Kept in the context between calls (a GW loop calls these every
// iteration): the cuFFT plans of the last shape and the device scratch, so a
// call neither re-plans nor re-allocates.  Freed with the context.
struct FftCache {
  rgf::FftKeys keys;                       // what scratch, full and part belong to
  std::unique_ptr<struct Plan> full, part;
  void* scratch = nullptr;
  double2* roots[own::kMaxLog + 1] = {};   // own transforms: exp(-2 pi i n / 2M), n < M, then the twiddles
  int roots_dev = -1;
  cudaStream_t fill = nullptr;             // zeroes the elements outside the band beside the transforms
  cudaEvent_t fill_from = nullptr;
  int fill_dev = -1;
  void close_fill() {
    if (fill) cudaStreamDestroy(fill);
    if (fill_from) cudaEventDestroy(fill_from);
    fill = nullptr;
    fill_from = nullptr;
  }
  ~FftCache();
  static void destroy(void* p) { delete static_cast<FftCache*>(p); }
};

FftCache::~FftCache() {
  full.reset();
  part.reset();
  for (double2* r : roots)
    if (r) cudaFree(r);
  close_fill();
  if (scratch) {
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(keys.scratch_dev);
    cudaFree(scratch);
    cudaSetDevice(cur);
  }
}

// cache->scratch of at least `need` bytes on device dev
int reserve_scratch(FftCache* cache, int dev, size_t need, cudaStream_t st) {
  if (cache->keys.scratch_fits(dev, need)) return RGF_OK;
  cudaError_t e = cudaStreamSynchronize(st);   // earlier calls may still use the old scratch
  if (cache->scratch) cudaFree(cache->scratch);
  cache->scratch = nullptr;
  cache->keys.set_scratch(dev, 0);
  if (e == cudaSuccess) e = cudaMalloc(&cache->scratch, need);
  if (e != cudaSuccess) {
    cudaGetLastError();
    cache->scratch = nullptr;
    return fft_fail(RGF_E_NOMEM, "device scratch for the transforms");
  }
  cache->keys.set_scratch(dev, need);
  return RGF_OK;
}

// exp(-2 pi i num / den), rounded once
double2 unit_root(int64_t num, int64_t den) {
  const long double th = 2.0L * 3.14159265358979323846264338327950288L * (long double)num / (long double)den;
  return make_double2((double)cosl(th), (double)-sinl(th));
}

// ---- the library's own transforms
using LineFn = void (*)(int64_t, Dims, const double2*, const double2*, const double2*, double2*, double2*);
struct LineLaunch {
  LineFn fn[2];
  int threads, group, per_sm;
  size_t smem;
};
template <int LOGM>
LineLaunch line_launch() {
  using L = own::Line<LOGM>;
  return LineLaunch{{own::line_kernel<LOGM, 0>, own::line_kernel<LOGM, 1>}, L::kThreads, L::G, L::kPerSm, L::smem};
}
LineLaunch line_launch_for(int logm) {
  switch (logm) {
    case 5: return line_launch<5>();
    case 6: return line_launch<6>();
    case 7: return line_launch<7>();
    case 8: return line_launch<8>();
    case 9: return line_launch<9>();
    case 10: return line_launch<10>();
    case 11: return line_launch<11>();
    default: return line_launch<12>();
  }
}

// Where the own form pays (P + Sigma, 112 lines, ms, cuFFT form / own, 1 B200).
// k-grids with both axes of 1, 2 or 4 points have their transform in registers
// and win at every length (1 x 1: 130 energies 0.21 / 0.18, 2050 0.36 / 0.28,
// 4096 0.51 / 0.34; 4 x 4: 0.53 / 0.22, 3.64 / 2.13, 7.1 / 2.8).  Other grids
// sum their axes directly, at nky + nkz terms a value, against cuFFT:
//   one axis:  130 energies, 1 x 7 0.36 / 0.26;  258, 1 x 3 0.34 / 0.30, 1 x 11
//     0.50 / 0.52;  512, 1 x 3 0.37 / 0.38;  1026, 1 x 3 0.57 / 0.66;  2050,
//     1 x 8 1.5 / 2.1;  512, 1 x 64 2.6 / 6.6
//   two axes:  258, 3 x 3 0.60 / 0.44, 5 x 5 0.94 / 0.93;  512, 4 x 6 1.41 /
//     1.18, 5 x 7 1.70 / 1.80;  514, 5 x 5 1.42 / 1.60;  2050, 3 x 3 2.0 / 2.7
//     (energies padded to the next power of two);  1000, 4 x 6 2.7 / 2.2, 3 x 4
//     1.38 / 1.35;  4096, 3 x 4 5.5 / 4.8
// So: one axis up to 8 points and 256 energies; two axes up to 10 points
// together, and 512 energies or a count that fills its power of two.
bool any_grid_pays(const Dims& d, int64_t M) {
  if (d.nky == 1 || d.nkz == 1) return d.nk <= 8 && M <= 256;
  return d.nky + d.nkz <= 10 && (M <= 512 || 32 * d.nen > 31 * M);
}
// log2 M, or 0 where the cuFFT form is taken
int own_log(const Dims& d) {
  auto small = [](int64_t n) { return n == 1 || n == 2 || n == 4; };
  const bool registers = small(d.nky) && small(d.nkz);
  for (int l = own::kMinLog; l <= own::kMaxLog; l++)
    if ((int64_t(1) << l) >= d.nen) return registers || any_grid_pays(d, int64_t(1) << l) ? l : 0;
  return 0;
}

template <int NKY, int NKZ>
void launch_k(bool forward, const own::Six& in, const own::Three& out, const int64_t* lines, int64_t nl, const Dims& d,
              int nops, unsigned conj, bool fix, const double2* ph, double2* kb, const double2* pb, cudaStream_t st) {
  if (forward)
    own::k_forward<NKY, NKZ><<<dim3((unsigned)((d.nen + 255) / 256), (unsigned)nl, (unsigned)nops), 256, 0, st>>>(
        in, lines, nl, d, conj, kb);
  else
    own::k_inverse<NKY, NKZ><<<dim3((unsigned)((d.nen + 127) / 128), (unsigned)nl), 128, 0, st>>>(out, lines, nl, d,
                                                                                                fix, ph, pb);
}

void k_transform(bool forward, const own::Six& in, const own::Three& out, const int64_t* lines, int64_t nl,
                 const Dims& d, int nops, unsigned conj, bool fix, const double2* ph, double2* kb, const double2* pb,
                 cudaStream_t st) {
#define RGF_K_CASE(Y, Z) \
  if (d.nky == Y && d.nkz == Z) return launch_k<Y, Z>(forward, in, out, lines, nl, d, nops, conj, fix, ph, kb, pb, st)
  RGF_K_CASE(1, 1);
  RGF_K_CASE(1, 2);
  RGF_K_CASE(2, 1);
  RGF_K_CASE(2, 2);
  RGF_K_CASE(1, 4);
  RGF_K_CASE(4, 1);
  RGF_K_CASE(2, 4);
  RGF_K_CASE(4, 2);
  RGF_K_CASE(4, 4);
#undef RGF_K_CASE
  const size_t tile = (size_t)d.nk * own::kTileE * sizeof(double2);
  const unsigned ge = (unsigned)((d.nen + own::kTileE - 1) / own::kTileE);
  if (forward)   // at most 25 k-points: 32 KB of shared memory
    own::k_forward_any<<<dim3(ge, (unsigned)nl, (unsigned)nops), 256, 2 * tile, st>>>(in, lines, nl, d, conj, ph, kb);
  else
    own::k_inverse_any<<<dim3(ge, (unsigned)nl), 256, 2 * tile + tile / 2, st>>>(out, lines, nl, d, fix, ph, pb);
}

// ph: the nk phases, then the nky-th and nkz-th roots.
int run_own(FftCache* cache, int dev, int mode, const Dims& d, int logm, const std::vector<int64_t>& lines,
            const std::vector<double2>& ph, const double2* const in[6], double2* const out[3], cudaStream_t st) {
  const int64_t M = int64_t(1) << logm;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const LineLaunch L = line_launch_for(logm);
  const int nops = mode == 0 ? 5 : 6;
  const size_t per_line = (size_t)(nops + 3) * d.nk * d.nen;   // values
  const int64_t nl = (int64_t)lines.size();
  int64_t chunk = (int64_t)(((size_t)1 << 30) / sizeof(double2) / per_line);
  if (const char* env = std::getenv("RGF_GW_FFT_CHUNK")) {
    const long v = std::atol(env);
    if (v > 0) chunk = v;
  }
  chunk = chunk < 1 ? 1 : (chunk > nl ? nl : chunk);
  if (chunk > 65535) chunk = 65535;                             // grid y
  // scratch for the CTAs that work, not more than a chunk keeps busy: short
  // calls need little memory
  const int64_t ctas = std::min((int64_t)sms * L.per_sm, (chunk * d.nk + L.group - 1) / L.group);
  const size_t scr = (size_t)ctas * L.group * 3 * M;
  int rc = reserve_scratch(cache, dev, sizeof(double2) * (per_line * chunk + scr + ph.size()) + sizeof(int64_t) * nl, st);
  if (rc) return rc;
  if (cache->roots_dev != dev) {
    for (double2*& r : cache->roots) {
      if (r) cudaFree(r);
      r = nullptr;
    }
    cache->roots_dev = dev;
  }
  if (!cache->roots[logm]) {
    std::vector<double2> r((size_t)M);
    for (int64_t n = 0; n < M; n++) r[n] = unit_root(n, 2 * M);
    r.resize((size_t)M + rgf::fft::table(logm, [](int, long long, long long) {}));
    rgf::fft::table(logm, [&](int k, long long num, long long den) { r[M + k] = unit_root(num, den); });
    double2* p = nullptr;
    if (cudaMalloc(&p, sizeof(double2) * r.size()) != cudaSuccess) {
      cudaGetLastError();
      return fft_fail(RGF_E_NOMEM, "table of roots");
    }
    if (cudaMemcpy(p, r.data(), sizeof(double2) * r.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
      cudaFree(p);
      return fft_fail(RGF_E_CUDA, "table of roots");
    }
    cache->roots[logm] = p;
  }
  double2* kb = (double2*)cache->scratch;
  double2* pb = kb + (size_t)nops * chunk * d.nk * d.nen;
  double2* d_scr = pb + (size_t)3 * chunk * d.nk * d.nen;
  double2* d_ph = d_scr + scr;
  int64_t* d_lines = (int64_t*)(d_ph + ph.size());
  cudaError_t ce = cudaMemcpyAsync(d_lines, lines.data(), sizeof(int64_t) * nl, cudaMemcpyHostToDevice, st);
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(d_ph, ph.data(), sizeof(double2) * ph.size(), cudaMemcpyHostToDevice, st);
  // the host vectors must outlive the asynchronous copies from them
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  if (ce == cudaSuccess && L.smem > 48 * 1024)
    ce = cudaFuncSetAttribute(L.fn[mode], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
  if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  own::Six src;
  for (int a = 0; a < 6; a++) src.a[a] = in[a];
  const own::Three dst{{out[0], out[1], out[2]}};
  const unsigned conj = mode == 0 ? 0x18u : 0u;                 // Y^>, Y^<
  for (int64_t c0 = 0; c0 < nl; c0 += chunk) {
    const int64_t nb = (nl - c0) < chunk ? (nl - c0) : chunk;
    const int64_t tasks = nb * d.nk, need = (tasks + L.group - 1) / L.group;
    k_transform(true, src, dst, d_lines + c0, nb, d, nops, conj, false, d_ph, kb, pb, st);
    L.fn[mode]<<<(unsigned)(need < ctas ? need : ctas), L.threads, L.smem, st>>>(
        nb, d, cache->roots[logm] + M, cache->roots[logm], kb, pb, d_scr);
    k_transform(false, src, dst, d_lines + c0, nb, d, nops, conj, mode == 1, d_ph, kb, pb, st);
    ce = cudaGetLastError();
    if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  }
  ce = cudaStreamSynchronize(st);
  if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  return RGF_OK;
}

unsigned grid_for(int64_t total) {
  const int64_t g = (total + 255) / 256;
  return (unsigned)(g < 148 * 32 ? (g < 1 ? 1 : g) : 148 * 32);
}

// mode 0: polarization (x: in[0..2], y: in[3..5]); mode 1: self-energy
// (G: in[0..2], W: in[3..5]).
int run_fft_form(rgf_ctx* ctx, int mode, int64_t nm, int64_t nx, int64_t nen, int64_t nky, int64_t nkz,
                 int64_t ndiag, int64_t nij, int64_t first_ij, double dEn, double spindeg,
                 const double2* const in[6], double2* const out[3], cudaStream_t st) {
  g_fft_err[0] = 0;
  if (nm < 1 || nx < 1 || nen < 2 || (nen % 2) != 0 || nky < 1 || nkz < 1 || ndiag < 0 || nij < 0 ||
      first_ij < 1)
    return fft_fail(RGF_E_ARG, "invalid dimensions (nen must be even and >= 2, first_ij >= 1)");
  for (int a = 0; a < 6; a++)
    if (!in[a]) return fft_fail(RGF_E_ARG, "NULL input array");
  for (int a = 0; a < 3; a++)
    if (!out[a]) return fft_fail(RGF_E_ARG, "NULL output array");
  Dims d;
  d.nen = nen;
  d.nky = nky;
  d.nkz = nkz;
  d.nk = nky * nkz;
  d.N = nice_length(2 * nen - 1);
  if (d.N > (1 << 30) || d.nky > (1 << 20) || d.nkz > (1 << 20))
    return fft_fail(RGF_E_UNSUPPORTED, "transform length out of range");
  const size_t series = (size_t)d.nk * nen;
  // banded lines (i, ix), line = i * nx + ix (src/green_rgf.f90:1401-1408)
  std::vector<int64_t> lines;
  for (int64_t i = 0; i < nij; i++) {
    const int64_t g = i + first_ij;
    const int64_t col = (g - 1) / nm + 1, row = (g - 1) % nm + 1;
    const int64_t lo = row - ndiag > 1 ? row - ndiag : 1, hi = row + ndiag < nm ? row + ndiag : nm;
    if (col < lo || col > hi) continue;
    for (int64_t ix = 0; ix < nx; ix++) lines.push_back(i * nx + ix);
  }
  if (lines.empty()) {
    // nothing but zeros, in stream order: the one form of the call that a
    // stream capture can hold
    for (int a = 0; a < 3; a++) {
      const cudaError_t e = cudaMemsetAsync(out[a], 0, sizeof(double2) * series * nx * nij, st);
      if (e != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(e));
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &cap);
    if (e == cudaSuccess && cap == cudaStreamCaptureStatusNone) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? RGF_OK : fft_fail(RGF_E_CUDA, cudaGetErrorString(e));
  }
  // elements outside the band are zero, as in the reference's zeroed buffers:
  // the runs of elements between banded ones, or everything where the runs
  // are many
  std::vector<std::pair<int64_t, int64_t>> gaps;
  for (size_t q = 0; q <= lines.size(); q += nx) {   // lines come in runs of nx
    const int64_t from = q == 0 ? 0 : lines[q - nx] / nx + 1, to = q < lines.size() ? lines[q] / nx : nij;
    if (to > from) gaps.push_back({from, to});
  }
  if (gaps.size() > 64) gaps.assign(1, {0, nij});
  int dev = 0;
  cudaGetDevice(&dev);
  FftCache* cache = static_cast<FftCache*>(rgf::ctx_ext_cache(ctx));
  if (!cache) {
    cache = new FftCache();
    rgf::ctx_set_ext_cache(ctx, cache, &FftCache::destroy);
  }
  // the zeros are bound by HBM writes, the transforms by the SMs: they run
  // beside each other, ordered after the caller's earlier work and complete
  // before the call returns, whichever way it does
  if (cache->fill_dev != dev) {
    cache->close_fill();
    if (cudaStreamCreateWithFlags(&cache->fill, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&cache->fill_from, cudaEventDisableTiming) != cudaSuccess) {
      cache->close_fill();
      return fft_fail(RGF_E_CUDA, "fill stream");
    }
    cache->fill_dev = dev;
  }
  struct FillDone {
    cudaStream_t s;
    ~FillDone() { cudaStreamSynchronize(s); }
  } fill_done{cache->fill};
  cudaError_t fe = cudaEventRecord(cache->fill_from, st);
  if (fe == cudaSuccess) fe = cudaStreamWaitEvent(cache->fill, cache->fill_from, 0);
  for (int a = 0; a < 3 && fe == cudaSuccess; a++)
    for (const auto& r : gaps) {
      fe = cudaMemsetAsync(out[a] + series * nx * r.first, 0, sizeof(double2) * series * nx * (r.second - r.first),
                           cache->fill);
      if (fe != cudaSuccess) break;
    }
  // a single run over everything includes the lines: they are written after it
  if (fe == cudaSuccess && gaps.size() == 1 && gaps[0].first == 0 && gaps[0].second == nij)
    fe = cudaStreamSynchronize(cache->fill);
  if (fe != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(fe));
  // the k-shift phase with the normalisation and dE folded in
  const double kPi = 3.14159265359;   // the reference's pi (src/green_rgf.f90:23)
  double2 dE;
  if (mode == 0) dE = make_double2(0.0, -1.0 * dEn / 2.0 / kPi * spindeg / (double)d.nk);
  else dE = make_double2(0.0, dEn / 2.0 / kPi / (double)d.nk);
  const int logm = own_log(d);
  if (logm) d.N = int64_t(2) << logm;
  const double norm = 1.0 / ((double)d.nk * (double)d.N);
  const double sgn = mode == 0 ? -1.0 : 1.0;
  const int64_t sy = nky > 1 ? ((nky / 2 - 1) % nky + nky) % nky : 0;
  const int64_t sz = nkz > 1 ? ((nkz / 2 - 1) % nkz + nkz) % nkz : 0;
  std::vector<double2> ph(d.nk);
  for (int64_t k = 0; k < d.nk; k++) {
    const int64_t ky = k / nkz, kz = k % nkz;
    const double th = sgn * 2.0 * M_PI * ((double)(ky * sy) / (double)nky + (double)(kz * sz) / (double)nkz);
    const double2 e = make_double2(std::cos(th) * norm, std::sin(th) * norm);
    ph[k] = make_double2(e.x * dE.x - e.y * dE.y, e.x * dE.y + e.y * dE.x);
  }
  if (logm) {
    for (int64_t n : {nky, nkz})
      for (int64_t m = 0; m < n; m++) ph.push_back(unit_root(m, n));
    return run_own(cache, dev, mode, d, logm, lines, ph, in, out, st);
  }
  // chunk of lines: six spectra of nk x N complex values each
  const size_t per_line = 6 * (size_t)d.nk * d.N * sizeof(double2);
  int64_t chunk = (int64_t)((size_t)4 << 30) / (int64_t)per_line;
  if (const char* env = std::getenv("RGF_GW_FFT_CHUNK")) {
    const long v = std::atol(env);
    if (v > 0) chunk = v;
  }
  if (chunk < 1) chunk = 1;
  if (chunk > (int64_t)lines.size()) chunk = (int64_t)lines.size();
  const int64_t cap = (int64_t)(0x7fffffff / ((size_t)d.nk * d.N));
  if (chunk > cap) chunk = cap;
  if (chunk < 1) return fft_fail(RGF_E_UNSUPPORTED, "one line exceeds the transform size limit");
  const int64_t nl = (int64_t)lines.size();
  const size_t need = per_line * chunk + sizeof(int64_t) * lines.size() + sizeof(double2) * d.nk;
  const int rc = reserve_scratch(cache, dev, need, st);
  if (rc) return rc;
  const int64_t tail = nl % chunk;
  const rgf::FftPlanKey key{dev, nky, nkz, d.N, chunk, tail};
  if (!cache->keys.plans_fit(key)) {
    cache->keys.drop_plans();
    cache->full.reset(new Plan(d, chunk, st));
    cache->part.reset(tail ? new Plan(d, tail, st) : nullptr);
    if (!cache->full->ok || (tail && !cache->part->ok)) {
      cache->full.reset();
      cache->part.reset();
      return fft_fail(RGF_E_CUDA, "cuFFT plan");
    }
    cache->keys.set_plans(key);
  }
  if (cufftSetStream(cache->full->h, st) != CUFFT_SUCCESS ||
      (cache->part && cufftSetStream(cache->part->h, st) != CUFFT_SUCCESS))
    return fft_fail(RGF_E_CUDA, "cuFFT stream");
  const size_t spec = (size_t)chunk * d.nk * d.N;
  double2* buf[6];
  for (int a = 0; a < 6; a++) buf[a] = (double2*)cache->scratch + a * spec;
  // the phases before the line numbers: an odd count of those would leave
  // 16-byte values at an odd multiple of 8
  double2* d_ph = (double2*)cache->scratch + 6 * spec;
  int64_t* d_lines = (int64_t*)(d_ph + d.nk);
  cudaError_t ce = cudaMemcpyAsync(d_lines, lines.data(), sizeof(int64_t) * lines.size(), cudaMemcpyHostToDevice, st);
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(d_ph, ph.data(), sizeof(double2) * d.nk, cudaMemcpyHostToDevice, st);
  if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  // the host vectors must outlive the asynchronous copies from them
  ce = cudaStreamSynchronize(st);
  if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  for (int64_t c0 = 0; c0 < nl; c0 += chunk) {
    const int64_t nb = (nl - c0) < chunk ? (nl - c0) : chunk;
    const Plan& plan = nb == chunk ? *cache->full : *cache->part;
    const int64_t* L = d_lines + c0;
    const int64_t tot = nb * d.nk * d.N;
    for (int a = 0; a < 6; a++) {
      const int pm = mode == 0 ? (a == 5 ? 1 : 0) : (a >= 3 ? 2 : 0);
      pack_kernel<<<grid_for(tot), 256, 0, st>>>(in[a], L, nb, d, pm, buf[a]);
      if (!plan.run(buf[a], CUFFT_FORWARD)) return fft_fail(RGF_E_CUDA, "cuFFT forward transform");
    }
    if (mode == 0)
      corr_freq_kernel<<<grid_for(tot), 256, 0, st>>>(buf[0], buf[1], buf[2], buf[3], buf[4], buf[5], d_ph, nb, d);
    else
      conv_freq_kernel<<<grid_for(tot), 256, 0, st>>>(buf[0], buf[1], buf[2], buf[3], buf[4], buf[5], d_ph, nb, d);
    for (int a = 0; a < 3; a++)
      if (!plan.run(buf[a], CUFFT_INVERSE)) return fft_fail(RGF_E_CUDA, "cuFFT inverse transform");
    unpack_kernel<<<grid_for(nb * d.nk * nen), 256, 0, st>>>(buf[0], buf[1], buf[2], L, nb, d, mode, out[0],
                                                             out[1], out[2]);
    ce = cudaGetLastError();
    if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  }
  ce = cudaStreamSynchronize(st);
  if (ce != cudaSuccess) return fft_fail(RGF_E_CUDA, cudaGetErrorString(ce));
  return RGF_OK;
}

}  // namespace

extern "C" const char* rgf_gw_fft_last_error(void) { return g_fft_err; }

extern "C" int rgf_gw_polarization_fft(rgf_ctx* ctx, int64_t nm, int64_t nx, int64_t nen, int64_t nky,
                                       int64_t nkz, int64_t ndiag, int64_t nij, int64_t first_ij, double dEn,
                                       double spindeg, const rgf_c16* G_lesser, const rgf_c16* G_greater,
                                       const rgf_c16* G_r, const rgf_c16* G_lesser_t,
                                       const rgf_c16* G_greater_t, rgf_c16* P_lesser, rgf_c16* P_greater,
                                       rgf_c16* P_retarded, void* stream) {
  if (!ctx) return fft_fail(RGF_E_ARG, "NULL context");
  // x side: G^<, G^>, G^R; y side: G^>_t, G^<_t, conj(G^R)
  const double2* in[6] = {(const double2*)G_lesser, (const double2*)G_greater, (const double2*)G_r,
                          (const double2*)G_greater_t, (const double2*)G_lesser_t, (const double2*)G_r};
  double2* out[3] = {(double2*)P_lesser, (double2*)P_greater, (double2*)P_retarded};
  return run_fft_form(ctx, 0, nm, nx, nen, nky, nkz, ndiag, nij, first_ij, dEn, spindeg, in, out, (cudaStream_t)stream);
}

extern "C" int rgf_gw_self_energy_fft(rgf_ctx* ctx, int64_t nm, int64_t nx, int64_t nen, int64_t nky,
                                      int64_t nkz, int64_t ndiag, int64_t nij, int64_t first_ij, double dEn,
                                      const rgf_c16* G_lesser, const rgf_c16* G_greater, const rgf_c16* G_r,
                                      const rgf_c16* W_lesser, const rgf_c16* W_greater,
                                      const rgf_c16* W_retarded, rgf_c16* Sigma_lesser_new,
                                      rgf_c16* Sigma_greater_new, rgf_c16* Sigma_r_new, void* stream) {
  if (!ctx) return fft_fail(RGF_E_ARG, "NULL context");
  const double2* in[6] = {(const double2*)G_lesser, (const double2*)G_greater, (const double2*)G_r,
                          (const double2*)W_lesser, (const double2*)W_greater, (const double2*)W_retarded};
  double2* out[3] = {(double2*)Sigma_lesser_new, (double2*)Sigma_greater_new, (double2*)Sigma_r_new};
  return run_fft_form(ctx, 1, nm, nx, nen, nky, nkz, ndiag, nij, first_ij, dEn, 1.0, in, out, (cudaStream_t)stream);
}
