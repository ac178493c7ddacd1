// rgf_gw.cu -- the energy/k convolutions of the GW loop of
// green_rgf_solve_gw_3d (src/green_rgf.f90:2944-3092):
//
//   P^<_ij(w)  = dE_P sum_k sum_E G^<_ij(E,k) G^>_ji(E-w,k-q)
//   P^>_ij(w)  = dE_P sum_k sum_E G^>_ij(E,k) G^<_ji(E-w,k-q)
//   P^R_ij(w)  = dE_P sum_k sum_E G^<_ij(E,k) conj(G^R_ij(E-w,k-q)) + G^R_ij(E,k) G^<_ji(E-w,k-q)
//   S^<>_ij(E) = dE_S sum_w sum_q G^<>_ij(E-w,k-q) W^<>_ij(w,q)
//   S^R_ij(E)  = dE_S sum_w sum_q G^<_ij W^R_ij + G^R_ij W^<_ij + G^R_ij W^R_ij
//
// for |i - j| <= ndiag, dE_P = -i dE/(2 pi) spindeg/nk, dE_S = i dE/(2 pi)/nk,
// followed for S by the reference's Sigma^R imaginary part from
// Sigma^> - Sigma^<, symmetrisation, mixing into the running self-energies
// and the edge-block copies.  These are direct sums, as in the reference:
// every output element is accumulated by one thread in a
// fixed order (P: k then E; S: q then w).  Layout (nm,nm,nx,nen,nk) column-major, k = kz + ky*nkz.
//
// Three passes: the banded elements are gathered into series contiguous in
// energy, the sums run on those with R outputs a thread in registers, and a
// scatter pass writes the caller's arrays (for S with the post-processing).
// Where the device has no memory left for the series of one block, the sums
// run on the caller's arrays as they are (gw_*_direct_kernel, no scratch).
#include <algorithm>
#include <cstdio>
#include <type_traits>

#include "rgf_device.cuh"
#include "rgf_internal.h"

namespace {

constexpr double kPiGW = 3.14159265359;  // green_rgf.f90:23

struct GWDims {
  int64_t nm, nx, nen, nky, nkz, ndiag, nopmax;
  __device__ __forceinline__ size_t at(int64_t i, int64_t j, int64_t ix, int64_t ie, int64_t ik) const {
    return (size_t)i + (size_t)nm * ((size_t)j + (size_t)nm * ((size_t)ix + (size_t)nx * ((size_t)ie + (size_t)nen * ik)));
  }
  // 0-based k - q with the reference's nk/2 shift (green_rgf.f90:2968-2977)
  __device__ __forceinline__ int64_t kd(int64_t ik, int64_t iq) const {
    const int64_t iky = ik / nkz, ikz = ik % nkz, iqy = iq / nkz, iqz = iq % nkz;
    int64_t ikzd = ikz - iqz + nkz / 2, ikyd = iky - iqy + nky / 2;   // 0-based: the reference's value - 1
    ikzd -= 1;
    ikyd -= 1;
    if (ikzd < 0) ikzd += nkz;
    if (ikzd >= nkz) ikzd -= nkz;
    if (ikyd < 0) ikyd += nky;
    if (ikyd >= nky) ikyd -= nky;
    if (nky == 1) ikyd = 0;
    if (nkz == 1) ikzd = 0;
    return ikzd + ikyd * nkz;
  }
};

struct Arrays3 {          // three arrays in the caller's layout
  const double2* a[3];
};
struct Lines3 {           // the same as lines (double or double2 values)
  void* a[3];
};

__device__ __forceinline__ double2 gread(const double2* G, size_t k, int imag_only) {
  const double2 v = G[k];
  return imag_only ? make_double2(0.0 * v.x, v.y) : v;
}

__device__ __forceinline__ double2 cfma(double2 acc, double2 a, double2 b) {
  return rgf::cadd(acc, rgf::cmul(a, b));
}
// acc += a b; a double stands for the imaginary number i a
__device__ __forceinline__ void cfma_to(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
__device__ __forceinline__ void cfma_to(double2& acc, double a, double2 b) {
  acc.x = fma(-a, b.y, acc.x);
  acc.y = fma(a, b.x, acc.y);
}

// One output of the polarization, summed in the reference's own order and
// with its complex products (k, then E).  The tiled kernels use it for lines
// that hold an infinity or a NaN, where leaving a term out is not the same as
// adding a zero, and the direct kernels for every element.
__device__ __noinline__ void p_reference_sum(const GWDims& d, int imag_only, int64_t nop, int64_t i, int64_t j,
                                             int64_t ix, int64_t iq, Arrays3 G, double2 out[3]) {
  const double2 *GL = G.a[0], *GG = G.a[1], *GR = G.a[2];
  const int64_t nk = d.nky * d.nkz;
  double2 al = rgf::czero(), ag = rgf::czero(), ar = rgf::czero();
  const int64_t lo = (nop + 1 > 1 ? nop + 1 : 1) - 1;  // 0-based E range [lo, hi)
  const int64_t hi = d.nen < d.nen + nop ? d.nen : d.nen + nop;
  for (int64_t ik = 0; ik < nk; ik++) {
    const int64_t ikd = d.kd(ik, iq);
    for (int64_t ie = lo; ie < hi; ie++) {
      const size_t a = d.at(i, j, ix, ie, ik);
      const size_t bt = d.at(j, i, ix, ie - nop, ikd);
      const size_t b = d.at(i, j, ix, ie - nop, ikd);
      const double2 gl = gread(GL, a, imag_only), gg = gread(GG, a, imag_only), gr = gread(GR, a, imag_only);
      const double2 glt = gread(GL, bt, imag_only);
      al = cfma(al, gl, gread(GG, bt, imag_only));
      ag = cfma(ag, gg, glt);
      ar = rgf::cadd(ar, rgf::cadd(rgf::cmul(gl, rgf::cconj(gread(GR, b, imag_only))), rgf::cmul(gr, glt)));
    }
  }
  out[0] = al;
  out[1] = ag;
  out[2] = ar;
}

// One output of the self-energy in the reference's order (w, then q).
__device__ __noinline__ void s_reference_sum(const GWDims& d, int imag_only, int64_t ie1, int64_t i, int64_t j,
                                             int64_t ix, int64_t ik, Arrays3 G, Arrays3 W, double2 out[3]) {
  const double2 *GL = G.a[0], *GG = G.a[1], *GR = G.a[2], *WL = W.a[0], *WG = W.a[1], *WR = W.a[2];
  const int64_t nk = d.nky * d.nkz;
  double2 al = rgf::czero(), ag = rgf::czero(), ar = rgf::czero();
  for (int64_t nop = -d.nopmax; nop <= d.nopmax; nop++) {
    if (!(ie1 > (nop > 1 ? nop : 1) && ie1 < d.nen + nop)) continue;   // green_rgf.f90:3034
    const int64_t iop = nop + d.nen / 2 - 1;
    for (int64_t iq = 0; iq < nk; iq++) {
      const size_t g = d.at(i, j, ix, ie1 - nop - 1, d.kd(ik, iq));
      const size_t w = d.at(i, j, ix, iop, iq);
      const double2 gl = gread(GL, g, imag_only), gr = gread(GR, g, imag_only);
      const double2 wl = WL[w], wr = WR[w];
      al = cfma(al, gl, wl);
      ag = cfma(ag, gread(GG, g, imag_only), WG[w]);
      ar = rgf::cadd(ar, rgf::cadd(rgf::cadd(rgf::cmul(gl, wr), rgf::cmul(gr, wl)), rgf::cmul(gr, wr)));
    }
  }
  out[0] = al;
  out[1] = ag;
  out[2] = ar;
}

// ---------------------------------------------------------------- band lines
// The sums run along energy, the arrays have energy at stride nm^2 nx, so the
// banded elements are first gathered into "lines": series of one element
// (i, j, ix), contiguous in energy, line = (ix - ix0) * slots + slot, slot =
// i + nm (j - i + nd) (nd = min(ndiag, nm - 1), slots = nm (2 nd + 1); the
// few slots whose j lies outside the block stay unused).  A lines array is
// [line][k][energy].
struct Lines {
  int64_t nd, slots, ix0;
  __host__ __device__ int64_t slot(int64_t i, int64_t j, int64_t nm) const { return i + nm * (j - i + nd); }
};

constexpr int kPackP = 64, kPackE = 32;   // elements x energies of a gather tile

// Gathers three arrays into lines: the imaginary parts (IMAG) or the whole
// values.  A CTA takes kPackP consecutive elements of the block x kPackE
// energies of one (ix, k), so it reads contiguous runs and writes runs along
// energy through shared memory.  flags[line] is set when a line holds an
// infinity or a NaN.
template <bool IMAG>
__global__ void __launch_bounds__(256) gw_pack_kernel(GWDims d, Lines L, Arrays3 src, Lines3 dst,
                                                       int* __restrict__ flags) {
  using T = std::conditional_t<IMAG, double, double2>;
  __shared__ T tile[kPackP][kPackE + 1];
  const int64_t n2 = d.nm * d.nm, nk = d.nky * d.nkz;
  const int64_t p0 = (int64_t)blockIdx.x * kPackP;
  const int64_t ik = blockIdx.z % nk, ixl = blockIdx.z / nk;
  auto band = [&](int64_t p, int64_t& slot) {
    if (p >= n2) return false;
    const int64_t i = p % d.nm, j = p / d.nm;
    slot = L.slot(i, j, d.nm);
    return i - j <= L.nd && j - i <= L.nd;
  };
  int64_t slot;
  const int lp = threadIdx.x % kPackP;
  const bool mine = band(p0 + lp, slot);
  if (!__syncthreads_or(mine)) return;
  for (int64_t e0 = (int64_t)blockIdx.y * kPackE; e0 < d.nen; e0 += (int64_t)gridDim.y * kPackE)
    for (int v = 0; v < 3; v++) {
      if (mine) {
        bool bad = false;
        for (int le = threadIdx.x / kPackP; le < kPackE; le += 256 / kPackP) {
          const int64_t e = e0 + le;
          if (e >= d.nen) break;
          const double2 x = src.a[v][p0 + lp + n2 * ((L.ix0 + ixl) + d.nx * (e + d.nen * ik))];
          bad |= !(isfinite(x.x) && isfinite(x.y));
          if constexpr (IMAG) tile[lp][le] = x.y;
          else tile[lp][le] = x;
        }
        if (bad) flags[ixl * L.slots + slot] = 1;
      }
      __syncthreads();
      for (int q = threadIdx.x; q < kPackP * kPackE; q += 256) {
        const int le = q % kPackE, pp = q / kPackE;
        int64_t sl;
        if (e0 + le < d.nen && band(p0 + pp, sl))
          ((T*)dst.a[v])[((ixl * L.slots + sl) * nk + ik) * d.nen + e0 + le] = tile[pp][le];
      }
      __syncthreads();
    }
}

// ---------------------------------------------------------------- sums
// Both sums are correlations along energy: output n of a line is
// sum_u x(u) v(u - n), v a series that slides by one per step and per output.
// A thread owns R consecutive outputs; at step u it needs v(u - n) for its R
// outputs, of which R - 1 were already used at the step before, so it keeps
// them in registers (slot (u - r) mod R for output r) and loads one new value
// per series and step.  x(u) is the same for the whole CTA (a broadcast
// read).  Tiles of TILE outputs x kSteps steps are staged in shared memory,
// whatever nen is; v's position is padded by one per R values, so the lanes'
// reads (R apart) fall on distinct banks.  The bound is the FP64 pipe: per
// step and thread 32 multiply-adds against 6-7 shared loads.  Series are
// finite here (other lines take the reference sum), so values outside a
// series are zeros in shared memory instead of conditions in the loop.
// Measured (1 B200, 1965 MHz) at nk = 4, nen = 512, nx = 10, nm = 16,
// ndiag = 3, imaginary G: P 7.7 -> 1.64 ms, Sigma 12.6 -> 1.80 ms (complex
// products on values staged whole, one output a thread, before), i.e. 15 and
// 16 TFLOP/s of real multiply-adds; gathers 0.32 ms, scatters 0.18 ms.
constexpr int kSteps = 64;

template <bool IMAG>
struct GwCfg {
  static constexpr int TILE = IMAG ? 512 : 256;        // outputs a CTA
  static constexpr int RP = IMAG ? 8 : 4;              // outputs a thread, polarization
  static constexpr int RS = 4;                         // self-energy
  static constexpr int TP = TILE / RP, TS = TILE / RS;  // threads
  static constexpr int kPerSm = IMAG ? 5 : 6;          // CTAs of gw_p_kernel an SM: bounds its registers
};

template <int R>
__device__ __forceinline__ constexpr int vpos(int t) { return t + t / R; }
template <int R, int TILE>
constexpr int vlen() { return kSteps + TILE + (kSteps + TILE) / R + 1; }

// Adds a chunk's sums to the running ones and clears them: sums of kSteps
// terms added up have a smaller rounding error than one chain over all
// terms.  The running sums sit in shared memory (one column a thread), which
// the chunk's 32 kSteps multiply-adds hide.
template <int N, int NT>
__device__ __forceinline__ void flush(double (&run)[N][NT], double* part) {
#pragma unroll
  for (int k = 0; k < N; k++) {
    run[k][threadIdx.x] += part[k];
    part[k] = 0.0;
  }
}

// Polarization of one (line, q), outputs nop of tile blockIdx.x:
//   P^<(n) = sum_k sum_e G^<(e, k) G^>t(e - n, k - q), and the two others.
// With purely imaginary G every product is one real multiply-add.  G: the
// lines of G^<, G^>, G^R; out: lines [line][q][energy of n].
template <bool IMAG>
__global__ void __launch_bounds__(GwCfg<IMAG>::TP, GwCfg<IMAG>::kPerSm) gw_p_kernel(GWDims d, Lines L, double2 scale, int imag_only,
                                                               Arrays3 src, Lines3 G, Lines3 out,
                                                               const int* __restrict__ flags) {
  using T = std::conditional_t<IMAG, double, double2>;
  constexpr int R = GwCfg<IMAG>::RP, NT = GwCfg<IMAG>::TP, kTile = GwCfg<IMAG>::TILE;
  constexpr int V = IMAG ? 1 : 2;                      // doubles per value
  __shared__ T xs[3][kSteps];
  __shared__ T vs[3][vlen<R, kTile>()];
  __shared__ double run[3 * R * V][NT];
  const int64_t nk = d.nky * d.nkz, nen = d.nen;
  const int64_t slot = blockIdx.y, i = slot % d.nm, j = i - L.nd + slot / d.nm;
  if (j < 0 || j >= d.nm) return;                      // uniform over the CTA
  const int64_t iq = blockIdx.z % nk, ixl = blockIdx.z / nk;
  const int64_t line = ixl * L.slots + slot, lineT = ixl * L.slots + L.slot(j, i, d.nm);
  const int64_t n0 = -d.nopmax + (int64_t)blockIdx.x * kTile;
  const int tid = threadIdx.x, q0 = R * tid;
  const size_t orow = (size_t)(line * nk + iq) * nen + nen / 2 - 1;
  if (flags[line] | flags[lineT]) {
    for (int r = 0; r < R; r++) {
      const int64_t nop = n0 + q0 + r;
      if (nop > d.nopmax) break;
      double2 a[3];
      p_reference_sum(d, imag_only, nop, i, j, L.ix0 + ixl, iq, src, a);
      for (int v = 0; v < 3; v++) ((double2*)out.a[v])[orow + nop] = rgf::cmul(a[v], scale);
    }
    return;
  }
  T acc[3][R];
  T (&al)[R] = acc[0], (&ag)[R] = acc[1], (&ar)[R] = acc[2];
#pragma unroll
  for (int r = 0; r < R; r++) al[r] = ag[r] = ar[r] = T{};
#pragma unroll
  for (int k = 0; k < 3 * R * V; k++) run[k][tid] = 0.0;
  // n = 0: with imaginary G that is symmetric in (i, j), diagonal elements
  // among them, P^R is a difference of equal sums (of equal products where
  // k - q = k), i.e. zero or the rounding of the reference's order.  It is
  // formed in that order, product by product, beside the chains of
  // multiply-adds: the threads form a chunk's terms, one each, and the thread
  // that owns the output adds them up during the next chunk (P + Sigma at the
  // sizes above 4.0 ms; formed and added by the owner alone 4.3).
  static_assert(NT == kSteps, "a term a thread");
  __shared__ T term[2][kSteps];
  const bool zero_here = n0 <= 0 && n0 + kTile > 0;
  const bool owner = zero_here && n0 + q0 <= 0 && n0 + q0 + R > 0;
  const int rz = (int)(-n0) - q0;
  int chunk = 0;                                       // chunks done
  T pr0{};
  auto add_terms = [&](int c) {
#pragma unroll 8
    for (int u = 0; u < kSteps; u++) {
      if constexpr (IMAG) pr0 += term[c & 1][u];
      else pr0 = rgf::cadd(pr0, term[c & 1][u]);
    }
  };
  for (int64_t ik = 0; ik < nk; ik++) {
    const size_t xrow = (size_t)(line * nk + ik) * nen;
    const size_t vrow = (size_t)(line * nk + d.kd(ik, iq)) * nen, vrowT = (size_t)(lineT * nk + d.kd(ik, iq)) * nen;
    for (int64_t e0 = 0; e0 < nen; e0 += kSteps) {
      const int64_t vb = e0 - n0 - (kTile - 1);        // energy of position 0 of the sliding series
      if (vb >= nen || vb + kTile - 1 + kSteps <= 0) continue;
      __syncthreads();
      for (int t = tid; t < kSteps; t += NT)
#pragma unroll
        for (int v = 0; v < 3; v++) xs[v][t] = e0 + t < nen ? ((const T*)G.a[v])[xrow + e0 + t] : T{};
      for (int t = tid; t < kTile - 1 + kSteps; t += NT) {
        const bool in = vb + t >= 0 && vb + t < nen;
        vs[0][vpos<R>(t)] = in ? ((const T*)G.a[1])[vrowT + vb + t] : T{};   // G^>t
        vs[1][vpos<R>(t)] = in ? ((const T*)G.a[0])[vrowT + vb + t] : T{};   // G^<t
        vs[2][vpos<R>(t)] = in ? ((const T*)G.a[2])[vrow + vb + t] : T{};    // G^R
      }
      __syncthreads();
      if (owner && chunk > 0) add_terms(chunk - 1);
      T w0[R], w1[R], w2[R];
#pragma unroll
      for (int r = 1; r < R; r++) {
        const int p = vpos<R>(kTile - 1 - q0 - r);
        w0[(R - r) % R] = vs[0][p];
        w1[(R - r) % R] = vs[1][p];
        w2[(R - r) % R] = vs[2][p];
      }
#pragma unroll 1
      for (int u0 = 0; u0 < kSteps; u0 += R) {
#pragma unroll
        for (int c = 0; c < R; c++) {
          const int p = vpos<R>(u0 + c + kTile - 1 - q0);
          w0[c] = vs[0][p];
          w1[c] = vs[1][p];
          w2[c] = vs[2][p];
          const T xl = xs[0][u0 + c], xg = xs[1][u0 + c], xr = xs[2][u0 + c];
#pragma unroll
          for (int r = 0; r < R; r++) {
            const int m = (c - r + R) % R;
            if constexpr (IMAG) {
              al[r] = fma(-xl, w0[m], al[r]);          // (i a)(i b) = -a b
              ag[r] = fma(-xg, w1[m], ag[r]);
              ar[r] = fma(xl, w2[m], fma(-xr, w1[m], ar[r]));
            } else {
              cfma_to(al[r], xl, w0[m]);
              cfma_to(ag[r], xg, w1[m]);
              cfma_to(ar[r], xl, rgf::cconj(w2[m]));
              cfma_to(ar[r], xr, w1[m]);
            }
          }
        }
      }
      flush(run, reinterpret_cast<double*>(acc));
      if (zero_here) {
        const int p = vpos<R>(tid + kTile - 1 + (int)n0);
        if constexpr (IMAG)
          term[chunk & 1][tid] = __dsub_rn(__dmul_rn(xs[0][tid], vs[2][p]), __dmul_rn(xs[2][tid], vs[1][p]));
        else
          term[chunk & 1][tid] =
              rgf::cadd(rgf::cmul(xs[0][tid], rgf::cconj(vs[2][p])), rgf::cmul(xs[2][tid], vs[1][p]));
        chunk++;
      }
    }
  }
  if (chunk > 0) {                                     // uniform over the CTA
    __syncthreads();
    if (owner) add_terms(chunk - 1);
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int64_t nop = n0 + q0 + r;
    if (nop > d.nopmax) break;
#pragma unroll
    for (int v = 0; v < 3; v++) {
      double2 z = make_double2(run[(v * R + r) * V][tid], IMAG ? 0.0 : run[(v * R + r) * V + V - 1][tid]);
      if (v == 2 && owner && r == rz) {
        if constexpr (IMAG) z.x = pr0;
        else z = pr0;
      }
      ((double2*)out.a[v])[orow + nop] = rgf::cmul(z, scale);
    }
  }
}

// Self-energy of one (line, k), energies of tile blockIdx.x:
//   S^<(E) = sum_q sum_n G^<(E - n, k - q) W^<(n, q), and the two others;
// G^R W^< + G^R W^R is formed as G^R (W^< + W^R).  The sums leave out the
// first output energy and G's last one, as the reference's do (:3034).
template <bool IMAG>
__global__ void __launch_bounds__(GwCfg<IMAG>::TS) gw_s_kernel(GWDims d, Lines L, double2 scale, int imag_only,
                                                               Arrays3 gsrc, Arrays3 wsrc, Lines3 G, Lines3 W,
                                                               Lines3 out, const int* __restrict__ gflags,
                                                               const int* __restrict__ wflags) {
  using T = std::conditional_t<IMAG, double, double2>;
  constexpr int R = GwCfg<IMAG>::RS, NT = GwCfg<IMAG>::TS, kTile = GwCfg<IMAG>::TILE;
  __shared__ double2 xs[4][kSteps];                    // W^<, W^>, W^R, W^< + W^R
  __shared__ T vs[3][vlen<R, kTile>()];
  __shared__ double run[6 * R][NT];
  const int64_t nk = d.nky * d.nkz, nen = d.nen, h = nen / 2 - 1;
  const int64_t slot = blockIdx.y, i = slot % d.nm, j = i - L.nd + slot / d.nm;
  if (j < 0 || j >= d.nm) return;
  const int64_t ik = blockIdx.z % nk, ixl = blockIdx.z / nk;
  const int64_t line = ixl * L.slots + slot;
  const int64_t t0 = (int64_t)blockIdx.x * kTile;      // first energy of the tile
  const int tid = threadIdx.x, q0 = R * tid;
  const size_t orow = (size_t)(line * nk + ik) * nen;
  if (gflags[line] | wflags[line]) {
    for (int r = 0; r < R; r++) {
      const int64_t e = t0 + q0 + r;
      if (e >= nen) break;
      double2 a[3];
      s_reference_sum(d, imag_only, e + 1, i, j, L.ix0 + ixl, ik, gsrc, wsrc, a);
      for (int v = 0; v < 3; v++) ((double2*)out.a[v])[orow + e] = rgf::cmul(a[v], scale);
    }
    return;
  }
  double2 acc[3][R];
  double2 (&al)[R] = acc[0], (&ag)[R] = acc[1], (&ar)[R] = acc[2];
#pragma unroll
  for (int r = 0; r < R; r++) al[r] = ag[r] = ar[r] = rgf::czero();
#pragma unroll
  for (int k = 0; k < 6 * R; k++) run[k][tid] = 0.0;
  for (int64_t iq = 0; iq < nk; iq++) {
    const size_t wrow = (size_t)(line * nk + iq) * nen + h, grow = (size_t)(line * nk + d.kd(ik, iq)) * nen;
    for (int64_t c0 = -d.nopmax; c0 <= d.nopmax; c0 += kSteps) {
      const int64_t vb = t0 - c0 + kTile - 1;          // G energy of position 0 (positions run down)
      if (vb < 0 || vb - (kTile - 1 + kSteps) >= nen - 1) continue;
      __syncthreads();
      for (int t = tid; t < kSteps; t += NT) {
        const bool in = c0 + t <= d.nopmax;
        const double2 wl = in ? ((const double2*)W.a[0])[wrow + c0 + t] : rgf::czero();
        const double2 wr = in ? ((const double2*)W.a[2])[wrow + c0 + t] : rgf::czero();
        xs[0][t] = wl;
        xs[1][t] = in ? ((const double2*)W.a[1])[wrow + c0 + t] : rgf::czero();
        xs[2][t] = wr;
        xs[3][t] = rgf::cadd(wl, wr);
      }
      for (int t = tid; t < kTile - 1 + kSteps; t += NT) {
        const int64_t e = vb - t;
        const bool in = e >= 0 && e < nen - 1;
#pragma unroll
        for (int v = 0; v < 3; v++) vs[v][vpos<R>(t)] = in ? ((const T*)G.a[v])[grow + e] : T{};
      }
      __syncthreads();
      T w0[R], w1[R], w2[R];
#pragma unroll
      for (int r = 1; r < R; r++) {
        const int p = vpos<R>(kTile - 1 - q0 - r);
        w0[(R - r) % R] = vs[0][p];
        w1[(R - r) % R] = vs[1][p];
        w2[(R - r) % R] = vs[2][p];
      }
#pragma unroll 1
      for (int u0 = 0; u0 < kSteps; u0 += R) {
#pragma unroll
        for (int c = 0; c < R; c++) {
          const int p = vpos<R>(u0 + c + kTile - 1 - q0);
          w0[c] = vs[0][p];
          w1[c] = vs[1][p];
          w2[c] = vs[2][p];
          const double2 xl = xs[0][u0 + c], xg = xs[1][u0 + c], xr = xs[2][u0 + c], xt = xs[3][u0 + c];
#pragma unroll
          for (int r = 0; r < R; r++) {
            const int m = (c - r + R) % R;
            cfma_to(al[r], w0[m], xl);
            cfma_to(ag[r], w1[m], xg);
            cfma_to(ar[r], w0[m], xr);
            cfma_to(ar[r], w2[m], xt);
          }
        }
      }
      flush(run, reinterpret_cast<double*>(acc));
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int64_t e = t0 + q0 + r;
    if (e >= nen) break;
#pragma unroll
    for (int v = 0; v < 3; v++) {
      const double2 z = make_double2(run[2 * (v * R + r)][tid], run[2 * (v * R + r) + 1][tid]);
      ((double2*)out.a[v])[orow + e] = rgf::cmul(e == 0 ? rgf::czero() : z, scale);
    }
  }
}

// ---------------------------------------------------------------- scatter
constexpr int kOutP = 16, kOutE = 32;   // elements x energies of a scatter tile

// P lines -> the caller's arrays, every element of the blocks ix0.. written:
// zero outside the band and outside the window of energy offsets.
__global__ void __launch_bounds__(256) gw_p_scatter_kernel(GWDims d, Lines L, Lines3 P, Lines3 out) {
  __shared__ double2 tile[3][kOutP][kOutE + 1];
  const int64_t n2 = d.nm * d.nm, nk = d.nky * d.nkz;
  const int64_t p0 = (int64_t)blockIdx.x * kOutP;
  const int64_t iq = blockIdx.z % nk, ixl = blockIdx.z / nk;
  const int64_t lo = d.nen / 2 - 1 - d.nopmax, hi = d.nen / 2 - 1 + d.nopmax;
  for (int64_t e0 = (int64_t)blockIdx.y * kOutE; e0 < d.nen; e0 += (int64_t)gridDim.y * kOutE) {
    for (int q = threadIdx.x; q < kOutP * kOutE; q += 256) {
      const int le = q % kOutE, lp = q / kOutE;
      const int64_t p = p0 + lp, e = e0 + le, i = p % d.nm, j = p / d.nm;
      const bool in = p < n2 && i - j <= L.nd && j - i <= L.nd && e >= lo && e <= hi;
#pragma unroll
      for (int v = 0; v < 3; v++)
        tile[v][lp][le] = in ? ((const double2*)P.a[v])[((ixl * L.slots + L.slot(i, j, d.nm)) * nk + iq) * d.nen + e]
                             : rgf::czero();
    }
    __syncthreads();
    for (int q = threadIdx.x; q < kOutP * kOutE; q += 256) {
      const int lp = q % kOutP, le = q / kOutP;
      const int64_t p = p0 + lp, e = e0 + le;
      if (p >= n2 || e >= d.nen) continue;
      const size_t o = (size_t)p + (size_t)n2 * ((L.ix0 + ixl) + (size_t)d.nx * (e + (size_t)d.nen * iq));
#pragma unroll
      for (int v = 0; v < 3; v++) ((double2*)out.a[v])[o] = tile[v][lp][le];
    }
    __syncthreads();
  }
}

// New values of elements (i, j) and (j, i) -> what is mixed in at both:
// Sigma^R's imaginary part from Sigma^> - Sigma^<, symmetrisation
// (green_rgf.f90:3068-3081).
__device__ __forceinline__ void s_post(const double2 (&a)[3], const double2 (&b)[3], double2 (&out)[3]) {
  auto sym = [](double2 x, double2 y) { return make_double2((x.x + y.x) / 2.0, (x.y + y.y) / 2.0); };
  out[0] = sym(a[0], b[0]);
  out[1] = sym(a[1], b[1]);
  out[2] = sym(make_double2(a[2].x, (a[1].y - a[0].y) / 2.0), make_double2(b[2].x, (b[1].y - b[0].y) / 2.0));
}

// Element p of block ix at (energy, k) = row / nx: mixing (:3083-3085) and the
// edge-block copies (:3087-3092) in the same pass.  Blocks 1, 2 repeat block 3
// and blocks nx-1, nx block nx-2, so only the blocks in between are summed and
// each writes its own copies.
__device__ __forceinline__ void s_mix(const GWDims& d, const Lines3& S, double alpha, int64_t p, int64_t ix, size_t row,
                                      const double2 (&nv)[3]) {
  const bool all = d.nx < 5;                            // every block repeats block 3
  const int64_t d0 = all ? 0 : (ix == 2 ? 0 : ix), d1 = all ? d.nx - 1 : (ix == d.nx - 3 ? d.nx - 1 : ix);
  const size_t n2 = (size_t)(d.nm * d.nm);
#pragma unroll
  for (int v = 0; v < 3; v++) {
    double2* A = (double2*)S.a[v];
    const double2 s = A[(size_t)p + n2 * (ix + row)];
    const double2 r = rgf::cadd(s, rgf::cscale(rgf::csub(nv[v], s), alpha));
    for (int64_t b = d0; b <= d1; b++) A[(size_t)p + n2 * (b + row)] = r;
  }
}

// Sigma lines (N: S^<, S^>, S^R) -> the running self-energies (s_post, s_mix).
// have = false: the window of offsets is empty and every new value is zero.
__global__ void __launch_bounds__(256, 3) gw_s_scatter_kernel(GWDims d, Lines L, double alpha, bool have, Lines3 N,
                                                           Lines3 S) {
  __shared__ double2 tile[3][kOutP][kOutE + 1];
  const int64_t n2 = d.nm * d.nm, nk = d.nky * d.nkz;
  const int64_t p0 = (int64_t)blockIdx.x * kOutP;
  const int64_t ik = blockIdx.z % nk, ixl = blockIdx.z / nk, ix = L.ix0 + ixl;
  for (int64_t e0 = (int64_t)blockIdx.y * kOutE; e0 < d.nen; e0 += (int64_t)gridDim.y * kOutE) {
    for (int q = threadIdx.x; q < kOutP * kOutE; q += 256) {
      const int le = q % kOutE, lp = q / kOutE;
      const int64_t p = p0 + lp, e = e0 + le, i = p % d.nm, j = p / d.nm;
      double2 nv[3] = {rgf::czero(), rgf::czero(), rgf::czero()};
      if (have && p < n2 && i - j <= L.nd && j - i <= L.nd && e < d.nen) {
        const size_t a = (size_t)((ixl * L.slots + L.slot(i, j, d.nm)) * nk + ik) * d.nen + e;
        const size_t b = (size_t)((ixl * L.slots + L.slot(j, i, d.nm)) * nk + ik) * d.nen + e;
        double2 na[3], nb[3];
#pragma unroll
        for (int v = 0; v < 3; v++) {
          na[v] = ((const double2*)N.a[v])[a];
          nb[v] = ((const double2*)N.a[v])[b];
        }
        s_post(na, nb, nv);
      }
#pragma unroll
      for (int v = 0; v < 3; v++) tile[v][lp][le] = nv[v];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < kOutP * kOutE; q += 256) {
      const int lp = q % kOutP, le = q / kOutP;
      const int64_t p = p0 + lp, e = e0 + le;
      if (p >= n2 || e >= d.nen) continue;
      const double2 nv[3] = {tile[0][lp][le], tile[1][lp][le], tile[2][lp][le]};
      s_mix(d, S, alpha, p, ix, (size_t)d.nx * (e + (size_t)d.nen * ik), nv);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- no scratch
// The sums on the caller's arrays, one output a thread, in the reference's
// order: for calls that find no memory for the series of one block.
constexpr int kDirectThreads = 128;

// grid: x = chunks of offsets, y = slot of the band, z = k-point + nk * block;
// the rest of the arrays was zeroed
__global__ void __launch_bounds__(kDirectThreads) gw_p_direct_kernel(GWDims d, Lines L, double2 scale, int imag_only,
                                                                     Arrays3 G, Lines3 out) {
  const int64_t nk = d.nky * d.nkz, iq = blockIdx.z % nk, ix = blockIdx.z / nk;
  const int64_t i = blockIdx.y % d.nm, j = i - L.nd + blockIdx.y / d.nm;
  const int64_t nop = -d.nopmax + (int64_t)blockIdx.x * kDirectThreads + threadIdx.x;
  if (j < 0 || j >= d.nm || nop > d.nopmax) return;
  double2 a[3];
  p_reference_sum(d, imag_only, nop, i, j, ix, iq, G, a);
  for (int v = 0; v < 3; v++) ((double2*)out.a[v])[d.at(i, j, ix, nop + d.nen / 2 - 1, iq)] = rgf::cmul(a[v], scale);
}

// grid: x = chunks of energies, y = elements of the block (strided), z =
// k-point + nk * (block - ix0); a thread owns elements (i, j) and (j, i)
__global__ void __launch_bounds__(kDirectThreads) gw_s_direct_kernel(GWDims d, Lines L, double2 scale, double alpha,
                                                                     bool have, int imag_only, Arrays3 G, Arrays3 W,
                                                                     Lines3 S) {
  const int64_t nk = d.nky * d.nkz, ik = blockIdx.z % nk, ix = L.ix0 + blockIdx.z / nk;
  const int64_t e = (int64_t)blockIdx.x * kDirectThreads + threadIdx.x;
  if (e >= d.nen) return;
  const size_t row = (size_t)d.nx * (e + (size_t)d.nen * ik);
  for (int64_t p = blockIdx.y; p < d.nm * d.nm; p += gridDim.y) {
    const int64_t i = p % d.nm, j = p / d.nm;
    if (i > j) continue;
    double2 nv[3] = {rgf::czero(), rgf::czero(), rgf::czero()};
    if (have && j - i <= L.nd) {
      double2 a[3], b[3];
      s_reference_sum(d, imag_only, e + 1, i, j, ix, ik, G, W, a);
      s_reference_sum(d, imag_only, e + 1, j, i, ix, ik, G, W, b);
#pragma unroll
      for (int v = 0; v < 3; v++) {
        a[v] = rgf::cmul(a[v], scale);
        b[v] = rgf::cmul(b[v], scale);
      }
      s_post(a, b, nv);
    }
    s_mix(d, S, alpha, p, ix, row, nv);
    if (i != j) s_mix(d, S, alpha, j + d.nm * i, ix, row, nv);
  }
}

bool on_device(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// A device view of a caller array: the array itself if it is device memory,
// else a staged copy (copied in if `in`, back to the host by `finish` if `out`).
struct View {
  void* host = nullptr;
  void* dev = nullptr;
  size_t bytes = 0;
  bool own = false, out = false;
  cudaError_t open(void* p, size_t n, bool in, bool o, cudaStream_t st) {
    bytes = n;
    out = o;
    if (on_device(p)) { dev = p; return cudaSuccess; }
    host = p;
    own = true;
    cudaError_t e = cudaMalloc(&dev, n);
    if (e == cudaSuccess && in) e = cudaMemcpyAsync(dev, p, n, cudaMemcpyHostToDevice, st);
    return e;
  }
  cudaError_t finish(cudaStream_t st) {
    return (own && out) ? cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st) : cudaSuccess;
  }
  ~View() { if (own && dev) cudaFree(dev); }
};

thread_local char g_gw_err[256];

int gw_fail(int code, const char* msg) {
  std::snprintf(g_gw_err, sizeof(g_gw_err), "%s", msg);
  return code;
}

// Scratch of one call (the context's, kept between calls up to kWorkBytes):
// the lines of as many blocks ix as fit kWorkBytes, at least one, and a flag
// per line.  The calls return with their stream drained, so the next one may
// reuse it.
struct Workspace {
  static constexpr size_t kWorkBytes = size_t(256) << 20;
  rgf_ctx* ctx = nullptr;
  int64_t nd = 0, slots = 0, nix = 0;
  size_t per_line = 0;
  char* base = nullptr;      // NULL: no memory for one block's lines
  int* flags = nullptr;

  ~Workspace() {
    if (ctx) rgf::ctx_scratch_trim(ctx, kWorkBytes);
  }
  // bytes_per_value: of all the lines arrays together
  void open(rgf_ctx* c, const GWDims& d, int64_t ix0, int64_t ix1, size_t bytes_per_value, int nflags) {
    ctx = c;
    nd = std::min(d.ndiag, d.nm - 1);
    slots = d.nm * (2 * nd + 1);
    per_line = (size_t)d.nky * d.nkz * d.nen;
    const size_t per_ix = ((size_t)slots * per_line * bytes_per_value + 255) & ~size_t(255);
    const size_t flag_bytes = sizeof(int) * (size_t)nflags * slots;
    nix = std::max<int64_t>(1, std::min<int64_t>(ix1 - ix0, (int64_t)(kWorkBytes / (per_ix + flag_bytes))));
    void* p = nullptr;
    if (!rgf::ctx_scratch(ctx, (per_ix + flag_bytes) * nix, &p)) {
      nix = 1;
      if (!rgf::ctx_scratch(ctx, per_ix + flag_bytes, &p)) return;
    }
    base = (char*)p;
    flags = (int*)(base + per_ix * nix);
  }
  // three lines arrays of `val`-byte values for n blocks, after `before` bytes
  // per value (the 16-byte ones first, which keeps them aligned)
  Lines3 take(size_t val, int64_t n, size_t before) const {
    const size_t len = (size_t)slots * n * per_line;
    char* p = base + len * before;
    return Lines3{{p, p + len * val, p + 2 * len * val}};
  }
  // CTAs along energy: a tile each, or several where the grid's limit is met
  static unsigned energy_tiles(const GWDims& d, int tile) {
    return (unsigned)std::min<int64_t>((d.nen + tile - 1) / tile, 65535);
  }
  void pack(const GWDims& d, const Lines& L, int64_t n, bool imag, const Arrays3& src, const Lines3& dst, int* fl,
            cudaStream_t st) const {
    cudaMemsetAsync(fl, 0, sizeof(int) * (size_t)n * slots, st);
    const dim3 grid((unsigned)((d.nm * d.nm + kPackP - 1) / kPackP), energy_tiles(d, kPackE),
                    (unsigned)(n * d.nky * d.nkz));
    if (imag) gw_pack_kernel<true><<<grid, 256, 0, st>>>(d, L, src, dst, fl);
    else gw_pack_kernel<false><<<grid, 256, 0, st>>>(d, L, src, dst, fl);
  }
  dim3 out_grid(const GWDims& d, int64_t n) const {
    return dim3((unsigned)((d.nm * d.nm + kOutP - 1) / kOutP), energy_tiles(d, kOutE),
                (unsigned)(n * d.nky * d.nkz));
  }
};

int check_dims(int64_t nm, int64_t nx, int64_t nen, int64_t nky, int64_t nkz, int64_t ndiag) {
  if (nm < 1 || nm > 4096 || nx < 3 || nen < 1 || nky < 1 || nkz < 1 || ndiag < 0)
    return gw_fail(RGF_E_ARG, "invalid GW dimensions (nx >= 3 for the edge-block copies)");
  if (nm * (2 * ndiag + 1) > 65535) return gw_fail(RGF_E_UNSUPPORTED, "nm*(2*ndiag+1) > 65535");
  if (nx * nky * nkz > 65535) return gw_fail(RGF_E_UNSUPPORTED, "nx*nk > 65535");
  return RGF_OK;
}

}  // namespace

extern "C" const char* rgf_gw_last_error(void) { return g_gw_err; }

extern "C" int rgf_gw_polarization(rgf_ctx* ctx, int64_t nm, int64_t nx, int64_t nen, int64_t nky,
                                   int64_t nkz, int64_t ndiag, double dE, double spindeg,
                                   int32_t imag_only, const rgf_c16* G_lesser,
                                   const rgf_c16* G_greater, const rgf_c16* G_r, rgf_c16* P_lesser,
                                   rgf_c16* P_greater, rgf_c16* P_retarded, void* stream) {
  g_gw_err[0] = 0;
  if (!ctx || !G_lesser || !G_greater || !G_r || !P_lesser || !P_greater || !P_retarded)
    return gw_fail(RGF_E_ARG, "NULL argument");
  int rc = check_dims(nm, nx, nen, nky, nkz, ndiag);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nk = nky * nkz;
  const size_t bytes = sizeof(rgf_c16) * (size_t)nm * nm * nx * nen * nk;
  Workspace ws;
  View gl, gg, gr, pl, pg, pr;
  cudaError_t e = gl.open((void*)G_lesser, bytes, true, false, st);
  if (e == cudaSuccess) e = gg.open((void*)G_greater, bytes, true, false, st);
  if (e == cudaSuccess) e = gr.open((void*)G_r, bytes, true, false, st);
  if (e == cudaSuccess) e = pl.open(P_lesser, bytes, false, true, st);
  if (e == cudaSuccess) e = pg.open(P_greater, bytes, false, true, st);
  if (e == cudaSuccess) e = pr.open(P_retarded, bytes, false, true, st);
  if (e != cudaSuccess) return gw_fail(RGF_E_CUDA, cudaGetErrorString(e));
  GWDims d{nm, nx, nen, nky, nkz, ndiag, nen / 2 - 10};
  if (d.nopmax < 0) {
    for (View* v : {&pl, &pg, &pr}) cudaMemsetAsync(v->dev, 0, bytes, st);
  } else {
    const double2 scale = make_double2(0.0, -1.0 * dE / 2.0 / kPiGW * spindeg / (double)nk);
    const Arrays3 G{{(const double2*)gl.dev, (const double2*)gg.dev, (const double2*)gr.dev}};
    const Lines3 out{{pl.dev, pg.dev, pr.dev}};
    const size_t val = imag_only ? sizeof(double) : sizeof(double2);
    const int64_t tile = imag_only ? GwCfg<true>::TILE : GwCfg<false>::TILE;
    ws.open(ctx, d, 0, nx, 3 * val + 3 * sizeof(double2), 1);
    if (!ws.base) {
      for (View* v : {&pl, &pg, &pr}) cudaMemsetAsync(v->dev, 0, bytes, st);
      const dim3 grid((unsigned)((2 * d.nopmax + kDirectThreads) / kDirectThreads), (unsigned)ws.slots,
                      (unsigned)(nx * nk));
      gw_p_direct_kernel<<<grid, kDirectThreads, 0, st>>>(d, Lines{ws.nd, ws.slots, 0}, scale, imag_only, G, out);
    }
    for (int64_t ix0 = 0; ws.base && ix0 < nx; ix0 += ws.nix) {
      const int64_t n = std::min(ws.nix, nx - ix0);
      const Lines L{ws.nd, ws.slots, ix0};
      const Lines3 pp = ws.take(sizeof(double2), n, 0), gp = ws.take(val, n, 3 * sizeof(double2));
      ws.pack(d, L, n, imag_only, G, gp, ws.flags, st);
      const dim3 grid((unsigned)((2 * d.nopmax + tile) / tile), (unsigned)ws.slots, (unsigned)(n * nk));
      if (imag_only) gw_p_kernel<true><<<grid, GwCfg<true>::TP, 0, st>>>(d, L, scale, imag_only, G, gp, pp, ws.flags);
      else gw_p_kernel<false><<<grid, GwCfg<false>::TP, 0, st>>>(d, L, scale, imag_only, G, gp, pp, ws.flags);
      gw_p_scatter_kernel<<<ws.out_grid(d, n), 256, 0, st>>>(d, L, pp, out);
    }
  }
  e = cudaGetLastError();
  for (View* v : {&pl, &pg, &pr})
    if (e == cudaSuccess) e = v->finish(st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? RGF_OK : gw_fail(RGF_E_CUDA, cudaGetErrorString(e));
}

extern "C" int rgf_gw_self_energy(rgf_ctx* ctx, int64_t nm, int64_t nx, int64_t nen, int64_t nky,
                                  int64_t nkz, int64_t ndiag, double dE, double alpha_mix,
                                  int32_t imag_only, const rgf_c16* G_lesser, const rgf_c16* G_greater,
                                  const rgf_c16* G_r, const rgf_c16* W_lesser, const rgf_c16* W_greater,
                                  const rgf_c16* W_retarded, rgf_c16* Sigma_lesser_gw,
                                  rgf_c16* Sigma_greater_gw, rgf_c16* Sigma_r_gw, void* stream) {
  g_gw_err[0] = 0;
  if (!ctx || !G_lesser || !G_greater || !G_r || !W_lesser || !W_greater || !W_retarded ||
      !Sigma_lesser_gw || !Sigma_greater_gw || !Sigma_r_gw)
    return gw_fail(RGF_E_ARG, "NULL argument");
  int rc = check_dims(nm, nx, nen, nky, nkz, ndiag);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nk = nky * nkz;
  const size_t bytes = sizeof(rgf_c16) * (size_t)nm * nm * nx * nen * nk;
  Workspace ws;
  View gl, gg, gr, wl, wg, wr, sl, sg, sr;
  cudaError_t e = gl.open((void*)G_lesser, bytes, true, false, st);
  if (e == cudaSuccess) e = gg.open((void*)G_greater, bytes, true, false, st);
  if (e == cudaSuccess) e = gr.open((void*)G_r, bytes, true, false, st);
  if (e == cudaSuccess) e = wl.open((void*)W_lesser, bytes, true, false, st);
  if (e == cudaSuccess) e = wg.open((void*)W_greater, bytes, true, false, st);
  if (e == cudaSuccess) e = wr.open((void*)W_retarded, bytes, true, false, st);
  if (e == cudaSuccess) e = sl.open(Sigma_lesser_gw, bytes, true, true, st);
  if (e == cudaSuccess) e = sg.open(Sigma_greater_gw, bytes, true, true, st);
  if (e == cudaSuccess) e = sr.open(Sigma_r_gw, bytes, true, true, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return gw_fail(e == cudaErrorMemoryAllocation ? RGF_E_NOMEM : RGF_E_CUDA, cudaGetErrorString(e));
  }
  GWDims d{nm, nx, nen, nky, nkz, ndiag, nen / 2 - 10};
  const bool have = d.nopmax >= 0;
  const double2 scale = make_double2(0.0, dE / 2.0 / kPiGW / (double)nk);
  const Arrays3 G{{(const double2*)gl.dev, (const double2*)gg.dev, (const double2*)gr.dev}};
  const Arrays3 W{{(const double2*)wl.dev, (const double2*)wg.dev, (const double2*)wr.dev}};
  const Lines3 S{{sl.dev, sg.dev, sr.dev}};
  // the blocks that are summed: the edge copies overwrite the others
  const int64_t first = 2, last = nx < 5 ? 2 : nx - 3;
  const size_t val = imag_only ? sizeof(double) : sizeof(double2);
  const int64_t tile = imag_only ? GwCfg<true>::TILE : GwCfg<false>::TILE;
  ws.open(ctx, d, first, last + 1, 3 * val + 6 * sizeof(double2), 2);
  if (!ws.base) {
    const dim3 grid((unsigned)((nen + kDirectThreads - 1) / kDirectThreads),
                    (unsigned)std::min<int64_t>(nm * nm, 65535), (unsigned)((last + 1 - first) * nk));
    gw_s_direct_kernel<<<grid, kDirectThreads, 0, st>>>(d, Lines{ws.nd, ws.slots, first}, scale, alpha_mix, have,
                                                        imag_only, G, W, S);
  }
  for (int64_t ix0 = first; ws.base && ix0 <= last; ix0 += ws.nix) {
    const int64_t n = std::min(ws.nix, last + 1 - ix0);
    const Lines L{ws.nd, ws.slots, ix0};
    const Lines3 wp = ws.take(sizeof(double2), n, 0), np = ws.take(sizeof(double2), n, 3 * sizeof(double2)),
                 gp = ws.take(val, n, 6 * sizeof(double2));
    if (have) {
      int* wflags = ws.flags + ws.nix * ws.slots;
      ws.pack(d, L, n, imag_only, G, gp, ws.flags, st);
      ws.pack(d, L, n, false, W, wp, wflags, st);
      const dim3 grid((unsigned)((nen + tile - 1) / tile), (unsigned)ws.slots, (unsigned)(n * nk));
      if (imag_only)
        gw_s_kernel<true><<<grid, GwCfg<true>::TS, 0, st>>>(d, L, scale, imag_only, G, W, gp, wp, np, ws.flags, wflags);
      else
        gw_s_kernel<false><<<grid, GwCfg<false>::TS, 0, st>>>(d, L, scale, imag_only, G, W, gp, wp, np, ws.flags, wflags);
    }
    gw_s_scatter_kernel<<<ws.out_grid(d, n), 256, 0, st>>>(d, L, alpha_mix, have, np, S);
  }
  e = cudaGetLastError();
  for (View* v : {&sl, &sg, &sr})
    if (e == cudaSuccess) e = v->finish(st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? RGF_OK : gw_fail(RGF_E_CUDA, cudaGetErrorString(e));
}
