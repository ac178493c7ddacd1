// rgf_fft_smem.cuh -- complex FP64 FFTs of M = 2^5 .. 2^12 points by the
// threads of one CTA, with the data in registers (16 points a thread) and
// shared memory used only to exchange them between stages.
//
// Stockham (self-sorting) radix-16 stages, the last one of radix 2, 4, 8 or
// 16: with NT = M / 16 threads, thread t starts from the points t + NT m
// (m = 0..15) and ends with the points t + NT m of the result, so a forward
// transform, a pointwise product and an inverse transform follow one another
// in registers.  At a stage with Ns = the product of the earlier radices, a
// butterfly j takes points j + r M/R, multiplies them by
// exp(-+2 pi i r (j mod Ns) / (Ns R)) and leaves point r at
// (j / Ns) Ns R + j mod Ns + r Ns.  Twiddles come from a table laid out as
// the threads read it (stage, then r, then j mod Ns), every value rounded
// once from extended precision: forming some of them as products of others
// cost 1.7x in error.
#pragma once
#include <cuda_runtime.h>

namespace rgf {
namespace fft {

__device__ __forceinline__ double2 mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a conj(b)
__device__ __forceinline__ double2 mulc(double2 a, double2 b) {
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// -i a (forward) or +i a (inverse)
template <bool INV>
__device__ __forceinline__ double2 quarter(double2 a) {
  return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}
template <bool INV>
__device__ __forceinline__ double2 twiddle(double2 a, double2 w) { return INV ? mulc(a, w) : mul(a, w); }

template <bool INV>
__device__ __forceinline__ void dft4(double2& a, double2& b, double2& c, double2& d) {
  const double2 s = add(a, c), t = sub(a, c), u = add(b, d), v = quarter<INV>(sub(b, d));
  a = add(s, u);
  b = add(t, v);
  c = sub(s, u);
  d = sub(t, v);
}

// x[r] (r = 0..15) -> its 16-point transform, in natural order.
template <bool INV>
__device__ __forceinline__ void dft16(double2 (&x)[16]) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
#pragma unroll
  for (int i = 0; i < 4; i++) dft4<INV>(x[i], x[i + 4], x[i + 8], x[i + 12]);
  // element i of the group k (x[i + 4 k]) times exp(-2 pi i i k / 16)
  const double2 w1 = make_double2(c1, -s1), w3 = make_double2(s1, -c1);
  auto eighth = [](double2 a) {   // exp(-+ 2 pi i / 8)
    return INV ? make_double2(h * (a.x - a.y), h * (a.x + a.y)) : make_double2(h * (a.x + a.y), h * (a.y - a.x));
  };
  x[5] = twiddle<INV>(x[5], w1);
  x[6] = eighth(x[6]);
  x[7] = twiddle<INV>(x[7], w3);
  x[9] = eighth(x[9]);
  x[10] = quarter<INV>(x[10]);
  x[11] = quarter<INV>(eighth(x[11]));
  x[13] = twiddle<INV>(x[13], w3);
  x[14] = quarter<INV>(eighth(x[14]));
  x[15] = twiddle<INV>(x[15], make_double2(-c1, s1));
#pragma unroll
  for (int k = 0; k < 4; k++) dft4<INV>(x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
  // x[4 k + m] is output k + 4 m
  auto swap = [](double2& a, double2& b) { const double2 t = a; a = b; b = t; };
  swap(x[1], x[4]);
  swap(x[2], x[8]);
  swap(x[3], x[12]);
  swap(x[6], x[9]);
  swap(x[7], x[13]);
  swap(x[11], x[14]);
}

template <bool INV>
__device__ __forceinline__ void dft8(double2& a0, double2& a1, double2& a2, double2& a3, double2& a4, double2& a5,
                                     double2& a6, double2& a7) {
  constexpr double h = 0.70710678118654752440;
  dft4<INV>(a0, a2, a4, a6);
  dft4<INV>(a1, a3, a5, a7);
  a3 = INV ? make_double2(h * (a3.x - a3.y), h * (a3.x + a3.y)) : make_double2(h * (a3.x + a3.y), h * (a3.y - a3.x));
  a5 = quarter<INV>(a5);
  a7 = quarter<INV>(INV ? make_double2(h * (a7.x - a7.y), h * (a7.x + a7.y))
                        : make_double2(h * (a7.x + a7.y), h * (a7.y - a7.x)));
  // even part e_k in a0, a2, a4, a6; odd part o_k in a1, a3, a5, a7
  const double2 e0 = a0, e1 = a2, e2 = a4, e3 = a6, o0 = a1, o1 = a3, o2 = a5, o3 = a7;
  a0 = add(e0, o0);
  a1 = add(e1, o1);
  a2 = add(e2, o2);
  a3 = add(e3, o3);
  a4 = sub(e0, o0);
  a5 = sub(e1, o1);
  a6 = sub(e2, o2);
  a7 = sub(e3, o3);
}

// Shared position of point n: one unused value per 16 keeps the first
// stage's stores (16 apart) on distinct banks.
__device__ __forceinline__ int pos(int n) { return n + (n >> 4); }

template <int LOGM>
struct Cfg {
  static constexpr int M = 1 << LOGM, NT = M / 16;
  static constexpr int S16 = LOGM / 4;                  // radix-16 stages
  static constexpr int LAST = 1 << (LOGM % 4);          // radix of the last stage (1: none)
  static constexpr int SMEM = M + M / 16;               // values of shared memory
};

// Twiddle table of a transform length: for each stage after the first, r =
// 1 .. R-1 and i = 0 .. Ns-1, exp(-2 pi i r i / (Ns R)).  fill(k, num, den)
// is called for entry k = exp(-2 pi i num / den); returns the entries.
template <class F>
inline int table(int logm, F&& fill) {
  int k = 0, left = logm;
  long long ns = 1;
  while (left > 0) {
    const int lr = left >= 4 ? 4 : left;
    const long long R = 1ll << lr;
    if (ns > 1)
      for (long long r = 1; r < R; r++)
        for (long long i = 0; i < ns; i++) fill(k++, r * i, ns * R);
    ns *= R;
    left -= lr;
  }
  return k;
}

// One transform by the NT threads of a group (t = 0..NT-1), every thread of
// the CTA calling it; buf: the group's shared memory; w: the table.
template <int LOGM, bool INV>
__device__ __forceinline__ void transform(double2 (&x)[16], double2* buf, const double2* __restrict__ w, int t) {
  using C = Cfg<LOGM>;
  constexpr int NT = C::NT;
  // the twiddles are the same for every transform of a task; keeping them
  // all in registers across transforms would spill, so each reads them again
  asm volatile("" : "+l"(w));
#pragma unroll
  for (int s = 0; s < C::S16; s++) {
    const int Ns = 1 << (4 * s);
    const int jm = t & (Ns - 1);
    if (s > 0) {
#pragma unroll
      for (int r = 1; r < 16; r++) x[r] = twiddle<INV>(x[r], w[(r - 1) * Ns + jm]);
      w += 15 * Ns;
    }
    dft16<INV>(x);
    if (s + 1 < C::S16 || C::LAST > 1) {
      const int base = ((t >> (4 * s)) << (4 * s + 4)) + jm;
      __syncthreads();
#pragma unroll
      for (int r = 0; r < 16; r++) buf[pos(base + r * Ns)] = x[r];
      __syncthreads();
#pragma unroll
      for (int r = 0; r < 16; r++) x[r] = buf[pos(t + r * NT)];
    }
  }
  // last stage: 16 / LAST butterflies a thread, j = t + NT b (b < 16 / LAST),
  // points j + r M / LAST = t + NT (b + r 16 / LAST), so it works in place
  if constexpr (C::LAST > 1) {
    constexpr int B = 16 / C::LAST, Ns = C::M / C::LAST;
#pragma unroll
    for (int b = 0; b < B; b++) {
#pragma unroll
      for (int r = 1; r < C::LAST; r++) x[b + r * B] = twiddle<INV>(x[b + r * B], w[(r - 1) * Ns + t + NT * b]);
      if constexpr (C::LAST == 2) {
        const double2 p = x[b], q = x[b + 8];
        x[b] = add(p, q);
        x[b + 8] = sub(p, q);
      } else if constexpr (C::LAST == 4) {
        dft4<INV>(x[b], x[b + 4], x[b + 8], x[b + 12]);
      } else {
        dft8<INV>(x[b], x[b + 2], x[b + 4], x[b + 6], x[b + 8], x[b + 10], x[b + 12], x[b + 14]);
      }
    }
  }
}

}  // namespace fft
}  // namespace rgf
