// rgf_staged.cuh -- shared-memory-staged complex DMMA GEMM and blocked
// Gauss-Jordan inverse for the block sizes the benchmarks use
// (nb = 32, 64, 128, 256).
//
// GEMM: C(M x N) = op(A)(M x K) * op(B)(K x N), complex FP64, operands in
// global memory (column-major with leading dimensions lda / ldb), op = N or
// C (conjugate transpose).  The CTA walks output tiles of PM x PN; for each
// it streams K in chunks of KC through two shared-memory stages filled with
// cp.async (16-byte copies, one complex value each), while the 8 warps run
// mma.sync.m8n8k4.f64 on the other stage.  Shared tiles are k-major with a
// row pitch of PM + 2 complex values, which makes the fragment reads of a
// quarter warp (rows g = 0,1 x k = 0..3) hit 8 distinct 16-byte bank groups.
//
// Inverse (nb >= 128): Gauss-Jordan with partial row pivoting, blocked by
// panels of PW columns.  Each panel is eliminated unblocked in shared memory
// (pivot rule: largest |re|+|im|, first index on ties, as zgetrf), its row
// interchanges are applied to the other columns, and the other columns get
// the panel's transformation as one rank-PW GEMM update:
//     rows of the panel:  X[P, j] = U[P, :] R[:, j]
//     other rows:         X[i, j] = X[i, j] + U[i, :] R[:, j]
// with U the eliminated panel and R = X[P, :] before the update.  The pivot
// sequence and the arithmetic per element are those of the unblocked
// elimination; only the order of the sums changes.
#pragma once
#include <type_traits>

#include "rgf_device.cuh"

namespace rgf {
// Internal linkage: every translation unit compiles its own copies, under its
// own register budget (the FP64 kernel's units cap at 128 registers, the
// mixed form's unit does not), so no out-of-line instance is shared.
namespace {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// dynamic shared memory of a CTA with two CTAs on an SM
constexpr size_t kBlockSmem = 108 * 1024 + 512;

template <int NB>
struct StagedCfg {
  static constexpr int PM = NB < 64 ? NB : 64;   // output tile
  static constexpr int PN = PM;
  static constexpr int KC = 16;                  // K chunk
  static constexpr int LDS = PM + 2;             // shared pitch (complex values)
  static constexpr int WARPS_M = 4, WARPS_N = 2;
  static constexpr int WM = PM / WARPS_M, WN = PN / WARPS_N;   // warp tile
  static constexpr int TM = WM / 8, TN = WN / 8;               // 8x8 subtiles per warp
  static constexpr int STAGE = 2 * KC * LDS;                   // complex values per stage (A + B)
  static constexpr int NSTAGE = 3;                             // cp.async pipeline depth (>= 2)
  // the nb = 128 inverse's panel: width and column pitch (complex values; NB + 2
  // makes the rank-8 updates' fragment reads of 4 columns x 2 rows hit 8
  // distinct 16-byte bank groups)
  static constexpr int PW = 48, LDP = NB + 2;
  static_assert(NB != 128 || (size_t(LDP) * PW + PW + NB + 8 * PW) * sizeof(double2) <= kBlockSmem, "panel");
  static constexpr size_t GEMM_SMEM = size_t(NSTAGE) * STAGE * sizeof(double2);
  // inverse: nb = 32: the matrix as assembled, then the exchanged columns;
  // nb = 64: the matrix, then the elimination's scratch; larger: a panel and
  // the scratch (rgf_tiled.cuh's panel_width fills kBlockSmem)
  static constexpr size_t INV_SMEM =
      NB >= 128 ? kBlockSmem
                : (size_t(NB) * NB + (NB == 32 ? 2 * 33 + 1 : 8 * (size_t(NB) - 8))) * sizeof(double2);
  static constexpr size_t SMEM = GEMM_SMEM > INV_SMEM ? GEMM_SMEM : INV_SMEM;
  // two CTAs per SM: 2 x (dynamic + static shared memory + 1 KB reserved)
  // within the SM's 228 KB
  static_assert(SMEM <= kBlockSmem, "shared memory for two CTAs per SM");
  static_assert(TM >= 1 && TN >= 1, "tile");
  static_assert(PM % (8 * WARPS_M) == 0 && PN % (8 * WARPS_N) == 0, "tile");
};

struct NoInit {};

// C = C0 + op(A) op(B); epi(i, j, v) once per element by its owner thread.
// C0 = init(i, j) when an init functor is given (read before the K loop, so
// its loads overlap the first chunks' copies), else 0.  M, N multiples of PM;
// K multiple of KC.  Caller synchronises afterwards.
template <int NB, class Init, class Epi>
__device__ __forceinline__ void gemm_staged_init(int M, int N, int K, const double2* A, int lda, bool cA,
                                                 const double2* B, int ldb, bool cB, double2* stage,
                                                 Init&& init, Epi&& epi, const int16_t* brow) {
  using C = StagedCfg<NB>;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp % C::WARPS_M) * C::WM, wn = (warp / C::WARPS_M) * C::WN;
  const double a_sg = cA ? -1.0 : 1.0, b_sg = cB ? -1.0 : 1.0;
  const int nchunks = K / C::KC;
  for (int tm0 = 0; tm0 < M; tm0 += C::PM) {
    for (int tn0 = 0; tn0 < N; tn0 += C::PN) {
      auto load_chunk = [&](int kc, int s) {
        double2* As = stage + s * C::STAGE;
        double2* Bs = As + C::KC * C::LDS;
        const int k0 = kc * C::KC;
        // op(A)[m][k] -> As[k*LDS + m]
        for (int e = tid; e < C::PM * C::KC; e += kThreads) {
          int m, k;
          if (!cA) { m = e % C::PM; k = e / C::PM; } else { k = e % C::KC; m = e / C::KC; }
          const double2* src = cA ? A + (size_t)(k0 + k) + (size_t)(tm0 + m) * lda
                                  : A + (size_t)(tm0 + m) + (size_t)(k0 + k) * lda;
          cp_async16(As + k * C::LDS + m, src);
        }
        // op(B)[k][n] -> Bs[k*LDS + n]
        for (int e = tid; e < C::PN * C::KC; e += kThreads) {
          int n, k;
          if (cB) { n = e % C::PN; k = e / C::PN; } else { k = e % C::KC; n = e / C::KC; }
          // brow: op(B) row k is row brow[k] of B (op N only)
          const int kr = brow ? (int)brow[k0 + k] : k0 + k;
          const double2* src = cB ? B + (size_t)(tn0 + n) + (size_t)(k0 + k) * ldb
                                  : B + (size_t)kr + (size_t)(tn0 + n) * ldb;
          cp_async16(Bs + k * C::LDS + n, src);
        }
      };
      double cr[C::TM][C::TN][2], ci[C::TM][C::TN][2];
#pragma unroll
      for (int a = 0; a < C::TM; a++)
#pragma unroll
        for (int b = 0; b < C::TN; b++) cr[a][b][0] = cr[a][b][1] = ci[a][b][0] = ci[a][b][1] = 0.0;
      if constexpr (!std::is_same_v<std::decay_t<Init>, NoInit>) {
#pragma unroll
        for (int a = 0; a < C::TM; a++)
#pragma unroll
          for (int b = 0; b < C::TN; b++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
              const double2 v = init(tm0 + wm + 8 * a + g, tn0 + wn + 8 * b + 2 * t + c);
              cr[a][b][c] = v.x;
              ci[a][b][c] = v.y;
            }
      }
      // prologue: chunks 0 .. NSTAGE-2 in flight; one commit group per chunk
      // (possibly empty), so at iteration kc "all but the newest NSTAGE-2
      // groups done" means chunk kc has landed.  One barrier per chunk: it
      // makes chunk kc visible and proves every warp done with chunk kc-1,
      // whose stage the refill after it reuses; the barrier before the
      // prologue frees the stages of the previous tile (or the caller's use
      // of the same shared memory).
      __syncthreads();
#pragma unroll
      for (int c = 0; c < C::NSTAGE - 1; c++) {
        if (c < nchunks) load_chunk(c, c);
        cp_async_commit();
      }
      for (int kc = 0; kc < nchunks; kc++) {
        cp_async_wait<C::NSTAGE - 2>();
        __syncthreads();
        if (kc + C::NSTAGE - 1 < nchunks) load_chunk(kc + C::NSTAGE - 1, (kc + C::NSTAGE - 1) % C::NSTAGE);
        cp_async_commit();
        const double2* As = stage + (kc % C::NSTAGE) * C::STAGE;
        const double2* Bs = As + C::KC * C::LDS;
#pragma unroll
        for (int k4 = 0; k4 < C::KC; k4 += 4) {
          double2 av[C::TM], bv[C::TN];
#pragma unroll
          for (int a = 0; a < C::TM; a++) av[a] = As[(k4 + t) * C::LDS + wm + 8 * a + g];
#pragma unroll
          for (int b = 0; b < C::TN; b++) bv[b] = Bs[(k4 + t) * C::LDS + wn + 8 * b + g];
          cmma_step<C::TM, C::TN>(cr, ci, av, bv, a_sg, b_sg);
        }
      }
      // every warp is done with the stages before any epilogue runs: an
      // epilogue may write shared memory the stages alias (the nb <= 64
      // inverse assembles its matrix there)
      __syncthreads();
#pragma unroll
      for (int a = 0; a < C::TM; a++)
#pragma unroll
        for (int b = 0; b < C::TN; b++)
#pragma unroll
          for (int c = 0; c < 2; c++)
            epi(tm0 + wm + 8 * a + g, tn0 + wn + 8 * b + 2 * t + c,
                make_double2(cr[a][b][c], ci[a][b][c]));
    }
  }
}

template <int NB, class Epi>
__device__ __forceinline__ void gemm_staged(int M, int N, int K, const double2* A, int lda, bool cA,
                                            const double2* B, int ldb, bool cB, double2* stage,
                                            Epi&& epi, const int16_t* brow = nullptr) {
  gemm_staged_init<NB>(M, N, K, A, lda, cA, B, ldb, cB, stage, NoInit{}, epi, brow);
}

// Gauss-Jordan inverse (partial pivoting) of the n x n block X, n <= 32, with
// the matrix in registers: lane i of every warp owns row i, warp h the columns
// 4 h .. 4 h + 3.  Rows are not interchanged (a used pivot row is marked), so
// a warp gets the pivot row of its columns by shuffles and the CTA needs one
// barrier a column: the warp that owns column k + 1 updates it, finds its
// pivot (redux.sync) and publishes column, pivot row and reciprocal in the
// buffer of the other parity before the barrier.  Bound by that chain: with
// interchanges through shared memory and two barriers a column it took 61 k
// cycles at nb = 32.
//   pivot row q:  x_qj <- x_qj / x_qk (j = k: 1 / x_qk)
//   other rows:   x_ij <- x_ij - x_ik x_qj / x_qk (j = k: - x_ik / x_qk)
// With q_k the pivot row of step k, element (k, q_m) of the inverse is
// x[q_k][m].  Pivot key, tie and zero-pivot rules as gj_subblock, ties broken
// by the lower row.  scr: 2 x 33 complex values of shared scratch and two
// words.  Every CTA of a group has the whole inverse and writes its share.
// Returns 1 (and zeros dst) on a zero pivot.
template <class G>
__device__ __noinline__ int gj_invert_reg(G grp, int n, const double2* X, double2* dst, double2* dst2, SmemInv& s,
                                          double2* scr) {
  constexpr int N = 32, CPT = N * N / kThreads;
  const int lane = threadIdx.x & 31, h = threadIdx.x >> 5, j0 = h * CPT;
  double2* col = scr;                          // [2][N] the published column
  double2* piv = col + 2 * N;                  // [2] reciprocal of the pivot
  int* prow = reinterpret_cast<int*>(piv + 2); // [2] pivot row, -1: zero pivot
  double2 x[CPT];
#pragma unroll
  for (int m = 0; m < CPT; m++) x[m] = lane < n && j0 + m < n ? X[lane + (j0 + m) * n] : czero();
  bool used = lane >= n;
  int step = 0;                                // the step this row was the pivot of
  auto publish = [&](double2 v, int k) {
    const int par = k & 1;
    col[par * N + lane] = v;
    const double av = cabs1(v);
    const unsigned hi = (unsigned)((unsigned long long)__double_as_longlong(av) >> 32);
    const unsigned key = used ? 0u : (!(av == av) ? 1u : (av == 0.0 ? 2u : (hi > 1u ? hi : 1u) + 2u));
    const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
    const unsigned q = __reduce_min_sync(0xffffffffu, key == kmax ? (unsigned)lane : 0xffffffffu);
    const double2 r = crecip(v);
    if ((unsigned)lane == q) {
      piv[par] = r;
      prow[par] = kmax == 2u ? -1 : lane;
      s.perm[k] = (int16_t)lane;
    }
  };
  if (h == 0) publish(x[0], 0);
  bool sing = false;
  for (int k0 = 0; k0 < n; k0 += CPT) {
#pragma unroll
    for (int c = 0; c < CPT; c++) {
      const int k = k0 + c, par = c & 1;       // CPT is even: parity of k
      if (k >= n) break;
      __syncthreads();
      const int q = prow[par];
      if (q < 0) { sing = true; break; }       // uniform
      const double2 pinv = piv[par], f = col[par * N + lane];
      const bool own = h * CPT == k0;          // this warp's columns include k
#pragma unroll
      for (int m = 0; m < CPT; m++) {
        const double2 xq = make_double2(__shfl_sync(0xffffffffu, x[m].x, q), __shfl_sync(0xffffffffu, x[m].y, q));
        const bool kc = own && m == c;
        const double2 r = kc ? pinv : cmul(xq, pinv);
        const double2 b = kc ? czero() : x[m];
        x[m] = lane == q ? r : make_double2(b.x - (f.x * r.x - f.y * r.y), b.y - (f.x * r.y + f.y * r.x));
      }
      if (lane == q) {
        used = true;
        step = k;
      }
      if (k + 1 < n && h == (k + 1) / CPT) publish(x[(c + 1) % CPT], k + 1);
    }
    if (sing) break;
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < CPT; m++) {
    const int j = j0 + m;
    if (lane >= n || j >= n || j % grp.size != grp.rank) continue;
    const int o = sing ? lane + j * n : step + s.perm[j] * n;
    const double2 v = sing ? czero() : x[m];
    dst[o] = v;
    if (dst2) dst2[o] = v;
  }
  grp.sync();
  return sing ? 1 : 0;
}

// Gauss-Jordan elimination of the KB = 8 panel columns sb0.. (pivot rows
// p0+sb0..) with the sub-block held in registers: thread tid owns row tid % NB
// and CPT consecutive columns of the sub-block.  Per column:
//   (1) the owners of the pivot column publish it and reduce the pivot key
//       per warp (redux.sync; partials to shared memory), each lane forming
//       the reciprocal of its own entry meanwhile so the winner's is ready;
//       barrier;
//   (2) every thread combines the partials (largest key, first row on ties);
//       the two owners of row q form the scaled pivot row r_j = x_qj / x_qc,
//       the owners of row k publish it, the panel's other columns get the
//       interchange; barrier;
//   (3) every thread updates its own elements, x_ij - f_i r_j.
// The pivot key is the high word of the bit pattern of |re|+|im| (monotonic
// for non-negative doubles), so entries within 2^-20 of each other count as
// equal and the first row among them is taken; EXACT: ties of the high word
// go by the low word (the block sizes whose unblocked search compared all
// bits).  Rows above k have key 0, NaN entries key 1 (never chosen unless the
// whole column is NaN, then row k as the scalar search), exact zeros key 2
// and every other entry a larger key.
// The per-element arithmetic is that of the unblocked elimination.  scr:
// 2 NB + 6 KB + 2 NB/32 complex values of scratch, double-buffered by column
// parity so one column's readers never race the next column's writers.
// Returns with the sub-block written back to the panel and a barrier passed;
// s.singular is set on a zero pivot.
// n <= NB rows; threads of rows from n on carry zeros that are never pivots.
template <int NB, bool EXACT = false>
__device__ __forceinline__ void gj_subblock(int n, int LD, double2* panel, int PW, int p0, int sb0, double2* scr,
                                            int16_t* rmap, SmemInv& s) {
  constexpr int KB = 8;
  constexpr int CPT = KB * NB / kThreads;  // sub-block columns per thread
  constexpr int WPC = NB / 32;             // warps owning one column
  static_assert(CPT * kThreads == KB * NB && KB % CPT == 0, "sub-block layout");
  const int tid = threadIdx.x, warp = tid >> 5;
  const int i = tid % NB, h = tid / NB;
  double2* fraw = scr;           // [2][NB] the pivot column before the step
  double2* rr = scr + 2 * NB;    // [2][KB] the scaled pivot row r
  double2* rk = rr + 2 * KB;     // [2][KB] row k of the sub-block before the step
  double2* pinvw = rk + 2 * KB;  // [2][WPC] per-warp winner's reciprocal
  unsigned* pk = reinterpret_cast<unsigned*>(pinvw + 2 * WPC);  // [2][WPC] keys
  int* pi = reinterpret_cast<int*>(pk + 2 * WPC);               // [2][WPC] rows
  unsigned* pl = reinterpret_cast<unsigned*>(pi + 2 * WPC);     // [2][WPC] low words (EXACT)
  double2 x[CPT];
#pragma unroll
  for (int m = 0; m < CPT; m++) x[m] = i < n ? panel[i + (sb0 + h * CPT + m) * LD] : czero();
#pragma unroll
  for (int cc = 0; cc < KB; cc++) {
    const int k = p0 + sb0 + cc, par = cc & 1;
    const int hc = cc / CPT, mc = cc % CPT;
    if (h == hc) {
      const double2 v = x[mc];
      fraw[par * NB + i] = v;
      const double av = cabs1(v);
      unsigned key = 0u;
      if (i >= k && i < n) {
        const unsigned hi = (unsigned)((unsigned long long)__double_as_longlong(av) >> 32);
        key = !(av == av) ? 1u : (av == 0.0 ? 2u : EXACT ? hi + 3u : (hi > 1u ? hi : 1u) + 2u);
      }
      const double2 pv = crecip(v);
      const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
      bool top = key == kmax;
      unsigned lmax = 0u;
      if constexpr (EXACT) {
        const unsigned lo = top ? (unsigned)__double_as_longlong(av) : 0u;
        lmax = __reduce_max_sync(0xffffffffu, kmax > 2u ? lo : 0u);
        top = top && (kmax <= 2u || lo == lmax);
      }
      const unsigned imin = __reduce_min_sync(0xffffffffu, top ? (unsigned)i : 0xffffffffu);
      if ((unsigned)i == imin) {
        const int w = warp - hc * WPC;
        if constexpr (EXACT) pl[par * WPC + w] = lmax;
        pk[par * WPC + w] = kmax;
        pi[par * WPC + w] = i;
        pinvw[par * WPC + w] = pv;
      }
    }
    __syncthreads();
    unsigned key = pk[par * WPC];
    unsigned low = EXACT ? pl[par * WPC] : 0u;
    int q = pi[par * WPC], wq = 0;
#pragma unroll
    for (int w = 1; w < WPC; w++) {
      const unsigned ek = pk[par * WPC + w];
      const int ei = pi[par * WPC + w];
      bool more = ek > key || (ek == key && ei < q);
      if constexpr (EXACT) {
        const unsigned el = pl[par * WPC + w];
        more = ek > key || (ek == key && (el > low || (el == low && ei < q)));
        if (more) low = el;
      }
      if (more) { key = ek; q = ei; wq = w; }
    }
    // largest |re|+|im| zero: flagged, and the caller discards the block
    if (key == 2u && tid == 0) s.singular = 1;
    if (tid == 0) {
      s.perm[k] = (int16_t)q;
      if (q != k) { const int16_t t = rmap[k]; rmap[k] = rmap[q]; rmap[q] = t; }
    }
    if (i == q) {
      const double2 pinv = pinvw[par * WPC + wq];
#pragma unroll
      for (int m = 0; m < CPT; m++) {
        const int jj = h * CPT + m;
        rr[par * KB + jj] = (jj == cc) ? pinv : cmul(x[m], pinv);
      }
    }
    if (i == k) {
#pragma unroll
      for (int m = 0; m < CPT; m++) rk[par * KB + h * CPT + m] = x[m];
    }
    if (q != k) {  // the panel's other columns: interchange rows k <-> q
      for (int j = tid; j < PW; j += kThreads) {
        if (j >= sb0 && j < sb0 + KB) continue;
        const double2 a = panel[k + j * LD];
        panel[k + j * LD] = panel[q + j * LD];
        panel[q + j * LD] = a;
      }
    }
    __syncthreads();
    const double2 f = (i == k) ? czero() : (i == q ? rk[par * KB + cc] : fraw[par * NB + i]);
#pragma unroll
    for (int m = 0; m < CPT; m++) {
      const int jj = h * CPT + m;
      const double2 r = rr[par * KB + jj];
      if (i == k) {
        x[m] = r;
      } else {
        const double2 base = (i == q) ? rk[par * KB + jj] : x[m];
        const double2 xx = (jj == cc) ? czero() : base;
        x[m] = make_double2(xx.x - (f.x * r.x - f.y * r.y), xx.y - (f.x * r.y + f.y * r.x));
      }
    }
  }
#pragma unroll
  for (int m = 0; m < CPT; m++)
    if (i < n) panel[i + (sb0 + h * CPT + m) * LD] = x[m];
  __syncthreads();
}

// Rank-8 update of a panel's other columns after its sub-block sb0.. (pivot
// rows R = rows p0+sb0.. of those columns, before the update, gathered into
// rbuf, 8 x (PW - 8)):
//   X[i, j] = (i in sub-block rows ? 0 : X[i, j]) + sum_t U[i, t] R[t, j]
// on the FP64 tensor pipe: warp w owns rows 8 TMU w .. (TMU 8-row subtiles)
// and walks the 8-column subtiles of the other columns; K = 8 is two m8n8k4
// steps, U's fragments loaded once.  Ends with a barrier.
template <int NB>
__device__ __forceinline__ void panel_rank8_update(int n, int LD, double2* panel, int PW, int p0, int sb0,
                                                   double2* rbuf) {
  constexpr int KB = 8;
  const int tid = threadIdx.x;
  const int nrest = PW - KB;
  if (nrest <= 0) return;
  for (int e = tid; e < KB * nrest; e += kThreads) {
    const int t = e % KB, jr = e / KB;
    const int j = jr < sb0 ? jr : jr + KB;
    rbuf[t + jr * KB] = panel[(p0 + sb0 + t) + j * LD];
  }
  __syncthreads();
  constexpr int TMU = NB / (8 * (kThreads / 32));
  static_assert(TMU >= 1 && TMU * 8 * (kThreads / 32) == NB, "rows per warp");
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int wm = warp * 8 * TMU;
  double2 av[2][TMU];
#pragma unroll
  for (int ks = 0; ks < 2; ks++)
#pragma unroll
    for (int a = 0; a < TMU; a++)
      av[ks][a] = wm + 8 * a < n ? panel[(wm + 8 * a + g) + (sb0 + 4 * ks + t4) * LD] : czero();
  for (int b = 0; wm < n && b < nrest / 8; b++) {
    double cr[TMU][1][2], ci[TMU][1][2];
#pragma unroll
    for (int a = 0; a < TMU; a++) cr[a][0][0] = cr[a][0][1] = ci[a][0][0] = ci[a][0][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < 2; ks++) {
      const double2 bv[1] = {rbuf[(4 * ks + t4) + (8 * b + g) * KB]};
      cmma_step<TMU, 1>(cr, ci, av[ks], bv, 1.0, 1.0);
    }
#pragma unroll
    for (int a = 0; a < TMU; a++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        if (TMU > 1 && wm + 8 * a >= n) continue;
        const int i = wm + 8 * a + g, jr = 8 * b + 2 * t4 + c;
        const int j = jr < sb0 ? jr : jr + KB;
        const bool prow = i >= p0 + sb0 && i < p0 + sb0 + KB;
        const int o = i + j * LD;
        const double2 x = prow ? czero() : panel[o];
        panel[o] = make_double2(x.x + cr[a][0][c], x.y + ci[a][0][c]);
      }
  }
  __syncthreads();
}

// Blocked Gauss-Jordan inverse of the NB x NB block X0 (global memory, ld
// NB, destroyed), result into dst (and dst2).  X1: a second global block.
// The row interchanges of a panel are never applied in place: the panel's
// update reads the permuted rows of the current matrix (row gather in the
// GEMM loader and in the accumulators' preload) and writes the next matrix,
// the two buffers alternating; the last panel writes dst itself, its columns
// in the inverse's order.  Dynamic shared memory: panel (NB x PW), pivot row
// (PW), multiplier column (NB) -- none of them is live during the update
// GEMM, which reuses the same memory as its staging buffers.  The panel's row
// map is read by that GEMM, so it lives in the static SmemInv.
// Returns 1 (and zeros dst) on a zero pivot.  nb = 128: the update with the
// size at compile time, over all columns, beats the tiled one that leaves the
// panel's own out (the benchmark's 296 energies 331 against 340 ms); the same
// arithmetic.
template <int NB>
__device__ int gj_invert_blocked(double2* X0, double2* X1, double2* dst, double2* dst2,
                                 double2* smem, double2* stage, SmemInv& s) {
  using C = StagedCfg<NB>;
  constexpr int PWM = C::PW;
  double2* panel = smem;
  double2* rowk = panel + (size_t)C::LDP * PWM;
  double2* fcol = rowk + PWM;
  int16_t* rmap = s.rmap;
  const int tid = threadIdx.x;
  double2* cur = X0;
  double2* nxt = X1;
  if (tid == 0) s.singular = 0;
  for (int p0 = 0; p0 < NB; p0 += PWM) {
    const int PW = (NB - p0) < PWM ? (NB - p0) : PWM;
    // (a) panel columns of the current matrix -> shared memory (pitch LDP)
    for (int e = tid; e < NB * PW; e += kThreads) {
      const int jj = e / NB, i = e - jj * NB;
      cp_async16(panel + i + (size_t)jj * C::LDP, cur + (size_t)p0 * NB + e);
    }
    cp_async_commit();
    for (int i = tid; i < NB; i += kThreads) rmap[i] = (int16_t)i;
    cp_async_wait<0>();
    __syncthreads();
    // (b) elimination of the panel in sub-blocks of KB columns: each sub-block
    //     is eliminated unblocked with its columns in registers (gj_subblock;
    //     its row interchanges applied to the whole panel), then the panel's
    //     other columns get the sub-block's
    //     transformation as one rank-KB update (the same U R form as the
    //     panel's own update below), so the panel is read and written once per
    //     sub-block instead of once per column.
    constexpr int KB = 8;
    static_assert(PWM % KB == 0 && (NB % PWM) % KB == 0, "panels of whole sub-blocks");
    double2* rbuf = fcol + NB;  // KB x PWM pivot rows of the other columns
    for (int sb0 = 0; sb0 < PW && !s.singular; sb0 += KB) {
      gj_subblock<NB>(NB, C::LDP, panel, PW, p0, sb0, rowk, rmap, s);
      if (s.singular) break;
      panel_rank8_update<NB>(NB, C::LDP, panel, PW, p0, sb0, rbuf);
    }
    if (s.singular) break;
    // the last panel writes the inverse itself: its column j is column
    // colsrc[j] of the eliminated matrix (the interchanges undone), i.e.
    // column c goes to coldst[c]
    const bool last = p0 + PW >= NB;
    if (last) {
      if (tid == 0) {
        for (int j = 0; j < NB; j++) s.colsrc[j] = (int16_t)j;
        for (int k = NB - 1; k >= 0; k--) {
          const int q = s.perm[k];
          if (q != k) { const int16_t tmp = s.colsrc[k]; s.colsrc[k] = s.colsrc[q]; s.colsrc[q] = tmp; }
        }
      }
      __syncthreads();
      for (int j = tid; j < NB; j += kThreads) s.coldst[s.colsrc[j]] = (int16_t)j;
      __syncthreads();
    }
    // (c) eliminated panel -> next matrix (its rows are already in the new order)
    for (int e = tid; e < NB * PW; e += kThreads) {
      const int jj = e / NB, i = e - jj * NB;
      const double2 v = panel[i + (size_t)jj * C::LDP];
      nxt[(size_t)p0 * NB + e] = v;
      if (last) {
        const size_t o = i + (size_t)s.coldst[p0 + jj] * NB;
        dst[o] = v;
        if (dst2) dst2[o] = v;
      }
    }
    __syncthreads();
    // (d) other columns: with R = rows rmap[P] of cur and U the panel,
    //     nxt[P, j] = U[P, :] R[:, j],   nxt[i, j] = cur[rmap[i], j] + U[i, :] R[:, j]
    gemm_staged_init<NB>(NB, NB, PW, nxt + (size_t)p0 * NB, NB, false, cur, NB, false, stage,
                         [&](int i, int j) {
                           const bool keep = (i < p0 || i >= p0 + PW) && (j < p0 || j >= p0 + PW);
                           return keep ? cur[(size_t)rmap[i] + (size_t)j * NB] : czero();
                         },
                         [&](int i, int j, double2 v) {
                           if (j >= p0 && j < p0 + PW) return;
                           if (last) {
                             const size_t o = i + (size_t)s.coldst[j] * NB;
                             dst[o] = v;
                             if (dst2) dst2[o] = v;
                           } else {
                             nxt[i + (size_t)j * NB] = v;
                           }
                         },
                         rmap + p0);
    __syncthreads();
    double2* t = cur;
    cur = nxt;
    nxt = t;
  }
  const int sing = s.singular;
  if (sing) {
    for (int e = tid; e < NB * NB; e += kThreads) {
      dst[e] = czero();
      if (dst2) dst2[e] = czero();
    }
    __syncthreads();
    return 1;
  }
  return 0;
}

}  // namespace

}  // namespace rgf
