// rgf_tiled.cuh -- block operations for any block size that is a multiple of 8,
// the size known at run time, by one CTA or by the CTAs of a thread-block
// cluster together (Group).
//
// Used for the block sizes from 80 on without a staged form (size at run time)
// and, with the size at compile time, for nb = 32, 64, 128 and 256 where a
// cluster shares a task.
//
// GEMM: as rgf_staged.cuh's (K in chunks of 16 through three cp.async stages,
// 8 warps of DMMA), but the output is cut into tiles of at most 64 x 64 that
// follow the block size, dealt to the CTAs of the group.  Shared tiles are
// k-major with a row pitch of 66 complex values (conflict-free fragments).
//
// Inverse: for nb = 64, 128, 256 as rgf_staged.cuh's, in panels, the panel's
// own columns left out of the update.  For the other sizes, whose unblocked
// elimination had a smaller error than panels have, 8 columns at a time
// (gj_invert_rank8).
#pragma once
#include "rgf_staged.cuh"

namespace rgf {
namespace {

constexpr int kTileDim = 64;               // largest output tile
constexpr int kChunk = 16;                 // K chunk
constexpr int kLds = kTileDim + 2;         // shared pitch (complex values)
constexpr int kStage = 2 * kChunk * kLds;  // complex values per stage (A + B)
constexpr int kStages = 3;                 // cp.async pipeline depth (>= 2)
constexpr int kSmemValues = (int)(kBlockSmem / sizeof(double2));
static_assert(size_t(kStages) * kStage * sizeof(double2) <= kBlockSmem, "GEMM stages");

// Rows covered by the sub-block elimination's threads: 256 threads own NBP
// rows x 8 columns.
__host__ __device__ constexpr int padded_rows(int n) { return n <= 64 ? 64 : (n <= 128 ? 128 : 256); }
// Shared scratch of the elimination (complex values): pivot column twice,
// pivot rows and candidates; the rank-8 update's 8 x PW pivot rows share it.
__host__ __device__ constexpr int sub_scratch(int nbp) { return 2 * nbp + 48 + nbp / 16; }
// Panel width of the blocked inverse: nb = 64 whole; 48 columns at nb = 128;
// 16 at nb = 256 (24 fit, 1 % faster, but with an error against 64 bits 1.04
// to 1.17 times that of 16).  Pitch n + 2, which makes the rank-8 updates'
// fragment reads of 4 columns x 2 rows hit 8 distinct 16-byte bank groups.
__host__ __device__ constexpr int panel_width(int n) { return n <= 64 ? n : (n <= 128 ? 48 : 16); }
constexpr bool panel_fits(int n) {
  return (n + 2) * panel_width(n) + (n <= 64 ? 8 * (n - 8) : 320) <= kSmemValues &&
         (n + 2) * panel_width(n) + sub_scratch(padded_rows(n)) <= kSmemValues;
}
static_assert(panel_fits(64) && panel_fits(128) && panel_fits(256), "panel");

struct AllCols {
  __device__ __forceinline__ int operator()(int j) const { return j; }
};

// Chunk of K on a warp's P pairs of row subtiles (the 16 rows of one m16n8k4)
// x C column subtiles.  The shape is compile-time code chosen per warp and
// chunk: straight-line steps let the next step's fragments load under the
// MMAs (conditional MMAs in one sequence: nb = 128 on 8 CTAs 44 instead of 35
// ms for 12 energies), and single row subtiles are not worth their own shapes
// (with eight shapes the accumulators moved through local memory at every
// chunk).  Rows of an odd subtile beyond the tile are computed from whatever
// the stage holds there and never read.
template <int P, int C>
__device__ __forceinline__ void mma_chunk(double (&cr)[4][2][2], double (&ci)[4][2][2], const double2* As,
                                          const double2* Bs, int kl, double a_sg, double b_sg) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  As += t * kLds + g;
  Bs += t * kLds + g;
  auto step = [&](int k4) {
    double2 av[2 * P], bv[C];
#pragma unroll
    for (int a = 0; a < 2 * P; a++) av[a] = As[k4 * kLds + 8 * a];
#pragma unroll
    for (int b = 0; b < C; b++) bv[b] = Bs[k4 * kLds + 8 * b];
    // four rounds of real products, each over all subtiles, so that
    // consecutive MMAs on one accumulator are 2 P C apart
    auto round = [&](double (&acc)[4][2][2], auto&& fa, auto&& fb) {
#pragma unroll
      for (int p = 0; p < P; p++)
#pragma unroll
        for (int b = 0; b < C; b++)
          dmma1684(acc[2 * p][b][0], acc[2 * p][b][1], acc[2 * p + 1][b][0], acc[2 * p + 1][b][1], fa(av[2 * p]),
                   fa(av[2 * p + 1]), fb(bv[b]));
    };
    auto re = [](double2 v) { return v.x; };
    round(cr, re, re);
    round(ci, re, [&](double2 v) { return v.y * b_sg; });
    round(cr, [&](double2 v) { return -v.y * a_sg; }, [&](double2 v) { return v.y * b_sg; });
    round(ci, [&](double2 v) { return v.y * a_sg; }, re);
  };
  // two steps a trip (kl is 8 or 16): with all four unrolled the fragments of
  // the later ones push accumulators out of the registers (40 against 35 ms)
#pragma unroll 1
  for (int k4 = 0; k4 < kl; k4 += 8) {
    step(k4);
    step(k4 + 4);
  }
}

// C = C0 + op(A) op(B); epi(i, j, v) once per element by its owner thread.
// C0 = init(i, j) when an init functor is given (read before the K loop, so
// its loads overlap the first chunks' copies), else 0.  M, N, K multiples of
// 8.  cols maps an output column to its column of B and of C (the inverse's
// update leaves the panel's own columns out).  brow: row k of B is row
// brow[k] (op N only).  Caller synchronises the group afterwards.
//
// A warp owns up to 4 x 2 subtiles of 8 x 8, rows in pairs: the 8 warps split
// a tile in 2 row halves x 4 column parts.  Warps w and w + 4 share a
// scheduler and its FP64 pipe: they have the same row half and the column
// parts c and c + 2, so a tile of r pairs x c subtiles costs ceil(r / 2) x
// ceil(c / 2) on the busiest pipe; what lies outside the block is not
// computed.
template <class Init, class Epi, class Cols>
__device__ __forceinline__ void gemm_tiles(const Group& grp, int M, int N, int K, const double2* A, int lda, bool cA,
                                           const double2* B, int ldb, bool cB, double2* stage, Init&& init, Epi&& epi,
                                           const int16_t* brow, Cols&& cols) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const double a_sg = cA ? -1.0 : 1.0, b_sg = cB ? -1.0 : 1.0;
  const int nchunks = (K + kChunk - 1) / kChunk;
  // tiles: equal parts in steps of 16, at least one a CTA where the block
  // allows it (columns split first: the row halves then stay full)
  int pr = (M + kTileDim - 1) / kTileDim, pc = (N + kTileDim - 1) / kTileDim;
  while (pr * pc < grp.size) {
    if (N / pc >= 32 && N / pc >= M / pr) pc *= 2;
    else if (M / pr >= 32) pr *= 2;
    else if (N / pc >= 32) pc *= 2;
    else break;
  }
  const int tm = ((M + pr - 1) / pr + 15) & ~15, tn = ((N + pc - 1) / pc + 15) & ~15;
  pr = (M + tm - 1) / tm;
  pc = (N + tn - 1) / tn;
  constexpr bool kPlain = std::is_same_v<std::decay_t<Cols>, AllCols>;   // no column map, no row gather
  // A thread's share of a chunk: four values of A and of B, four steps apart
  // along the dimension that is not contiguous in memory.
  const int am = cA ? tid >> 4 : tid & 63, ak = cA ? tid & 15 : tid >> 6;
  const int bn = cB ? tid & 63 : tid >> 4, bk = cB ? tid >> 6 : tid & 15;
  const unsigned as0 = ak * kLds + am, asd = cA ? 16 : 4 * kLds;
  const unsigned bs0 = kChunk * kLds + bk * kLds + bn, bsd = cB ? 4 * kLds : 16;
  const size_t ad = (size_t)(cA ? 16 : 4) * lda, bd = (size_t)(cB ? 4 : 16) * ldb;
  const size_t astep = cA ? kChunk : (size_t)kChunk * lda, bstep = cB ? (size_t)kChunk * ldb : kChunk;
  const int klast = K - (nchunks - 1) * kChunk;
  for (int tile = grp.rank; tile < pr * pc; tile += grp.size) {
    const int tm0 = (tile % pr) * tm, tn0 = (tile / pr) * tn;
    const int rows = min(tm, M - tm0), ncol = min(tn, N - tn0);
    const int r8 = rows >> 3, c8 = ncol >> 3;
    const int half = ((r8 + 3) >> 2) << 1, wr = warp & 1, wc = (warp & 4) ? 2 + ((warp >> 1) & 1) : (warp >> 1) & 1;
    const int wm = wr ? 8 * half : 0, ra = wr ? max(r8 - half, 0) : min(half, r8);
    const int cq = c8 >> 2, cx = c8 & 3;
    const int wn = 8 * (wc * cq + min(wc, cx)), ca = cq + (wc < cx ? 1 : 0);
    // which of the four lie inside the tile (bits 0-3) and also inside the
    // last chunk (bits 4-7)
    unsigned amask = 0, bmask = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const bool ar = cA ? am + 16 * i < rows : am < rows, br = cB ? bn < ncol : bn + 16 * i < ncol;
      const bool al = cA ? ak < klast : ak + 4 * i < klast, bl = cB ? bk + 4 * i < klast : bk < klast;
      amask |= (ar ? 1u << i : 0u) | (ar && al ? 16u << i : 0u);
      bmask |= (br ? 1u << i : 0u) | (br && bl ? 16u << i : 0u);
    }
    const double2* pa = A + (cA ? ak + (size_t)(tm0 + am) * lda : (tm0 + am) + (size_t)ak * lda);
    const double2* pb = B + (cB ? (tn0 + bn) + (size_t)bk * ldb : bk + (size_t)(tn0 + bn) * ldb);
    int kload = 0;   // next chunk to load
    auto load_next = [&](double2* st) {
      if (kload < nchunks) {
        const unsigned ma = kload == nchunks - 1 ? amask >> 4 : amask, mb = kload == nchunks - 1 ? bmask >> 4 : bmask;
        double2* As = st + as0;
        double2* Bs = st + bs0;
#pragma unroll
        for (int i = 0; i < 4; i++)
          if ((ma >> i) & 1) cp_async16(As + i * asd, pa + i * ad);
        if constexpr (kPlain) {
#pragma unroll
          for (int i = 0; i < 4; i++)
            if ((mb >> i) & 1) cp_async16(Bs + i * bsd, pb + i * bd);
          pb += bstep;
        } else {           // op N: rows brow[k] of the mapped columns
          const int kr = (mb & 15) ? (int)brow[kload * kChunk + bk] : 0;
#pragma unroll
          for (int i = 0; i < 4; i++)
            if ((mb >> i) & 1) cp_async16(Bs + i * bsd, B + kr + (size_t)cols(tn0 + bn + 16 * i) * ldb);
        }
        pa += astep;
        kload++;
      }
      cp_async_commit();   // one group per chunk, possibly empty
    };
    double cr[4][2][2], ci[4][2][2];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 2; b++) cr[a][b][0] = cr[a][b][1] = ci[a][b][0] = ci[a][b][1] = 0.0;
    if constexpr (!std::is_same_v<std::decay_t<Init>, NoInit>) {
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 2; b++)
          if (a < ra && b < ca)
#pragma unroll
            for (int c = 0; c < 2; c++) {
              const double2 v = init(tm0 + wm + 8 * a + g, cols(tn0 + wn + 8 * b + 2 * t + c));
              cr[a][b][c] = v.x;
              ci[a][b][c] = v.y;
            }
    }
    // Chunks 0 .. kStages-2 in flight before the loop, so at each chunk "all
    // but the newest kStages-2 groups done" means it has landed.  One barrier
    // per chunk: it makes the chunk visible and proves every warp done with
    // the one before, whose stage the refill after it reuses; the barrier
    // before the first loads frees the stages of the previous tile (or the
    // caller's use of the same shared memory).
    __syncthreads();
    load_next(stage);
    load_next(stage + kStage);
    double2* cur = stage;                            // this chunk's stage and
    double2* ahead = stage + (kStages - 1) * kStage; // the one to refill
#pragma unroll 1
    for (int kc = 0; kc < nchunks; kc++) {
      cp_async_wait<kStages - 2>();
      __syncthreads();
      load_next(ahead);
      const double2* As = cur + wm;
      const double2* Bs = cur + kChunk * kLds + wn;
      const int kl = kc == nchunks - 1 ? klast : kChunk;
      if (ra > 0 && ca > 0) {
        if (ra > 2) {
          if (ca > 1) mma_chunk<2, 2>(cr, ci, As, Bs, kl, a_sg, b_sg);
          else mma_chunk<2, 1>(cr, ci, As, Bs, kl, a_sg, b_sg);
        } else {
          if (ca > 1) mma_chunk<1, 2>(cr, ci, As, Bs, kl, a_sg, b_sg);
          else mma_chunk<1, 1>(cr, ci, As, Bs, kl, a_sg, b_sg);
        }
      }
      ahead = cur;
      cur = cur == stage + (kStages - 1) * kStage ? stage : cur + kStage;
    }
    // every warp is done with the stages before any epilogue runs: an
    // epilogue may write shared memory they alias (blocks of one tile assemble
    // the matrix to invert there)
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 2; b++)
        if (a < ra && b < ca)
#pragma unroll
          for (int c = 0; c < 2; c++)
            epi(tm0 + wm + 8 * a + g, cols(tn0 + wn + 8 * b + 2 * t + c), make_double2(cr[a][b][c], ci[a][b][c]));
  }
}

// colsrc (and coldst, its inverse) of the interchanges: column j of the
// inverse is column colsrc[j] of the eliminated matrix.
__device__ __forceinline__ void undo_interchanges(int n, SmemInv& s) {
  if (threadIdx.x == 0) {
    for (int j = 0; j < n; j++) s.colsrc[j] = (int16_t)j;
    for (int k = n - 1; k >= 0; k--) {
      const int q = s.perm[k];
      if (q != k) { const int16_t tmp = s.colsrc[k]; s.colsrc[k] = s.colsrc[q]; s.colsrc[q] = tmp; }
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < n; j += kThreads) s.coldst[s.colsrc[j]] = (int16_t)j;
  __syncthreads();
}

__device__ __forceinline__ int zero_inverse(const Group& grp, int n, double2* dst, double2* dst2) {
  for (int e = threadIdx.x + kThreads * grp.rank; e < n * n; e += kThreads * grp.size) {
    dst[e] = czero();
    if (dst2) dst2[e] = czero();
  }
  grp.sync();
  return 1;
}

// Gauss-Jordan inverse (partial pivoting) of the block of n = NB that `panel`
// (shared memory, pitch n + PAD) holds whole: 8-column sub-blocks eliminated with
// their elements in registers (gj_subblock) and the other columns updated by
// rank-8 DMMA products (panel_rank8_update).  Then dst[:, j] =
// panel[:, colsrc[j]] undoes the interchanges (and dst2 the same); every CTA
// of a group eliminates its own copy and writes its share.  scr: shared
// scratch of max(8 (n - 8), sub_scratch(NB)) complex values.  Returns 1 (and
// zeros dst) on a zero pivot.
template <int NB, int PAD>
__device__ __noinline__ int gj_invert_panel(const Group& grp, double2* panel, double2* dst, double2* dst2, SmemInv& s,
                                            double2* scr) {
  constexpr int n = NB, LD = n + PAD;
  if (threadIdx.x == 0) s.singular = 0;
  for (int i = threadIdx.x; i < n; i += kThreads) s.rmap[i] = (int16_t)i;
  __syncthreads();
  for (int sb0 = 0; sb0 < n; sb0 += 8) {
    gj_subblock<NB>(n, LD, panel, n, 0, sb0, scr, s.rmap, s);
    if (s.singular) break;
    panel_rank8_update<NB>(n, LD, panel, n, 0, sb0, scr);
  }
  const int sing = s.singular;
  __syncthreads();
  if (sing) return zero_inverse(grp, n, dst, dst2);
  undo_interchanges(n, s);
  for (int idx = threadIdx.x + kThreads * grp.rank; idx < n * n; idx += kThreads * grp.size) {
    const int j = idx / n, i = idx - j * n;
    const double2 v = panel[i + s.colsrc[j] * LD];
    dst[idx] = v;
    if (dst2) dst2[idx] = v;
  }
  grp.sync();
  return 0;
}

// Blocked Gauss-Jordan inverse of the block X0 of n = NB (global memory, ld n,
// destroyed), result into dst (and dst2).  X1: a second global block.
// The row interchanges of a panel are never applied in place: the panel's
// update reads the permuted rows of the current matrix (row gather in the
// GEMM loader and in the accumulators' preload) and writes the next matrix,
// the two buffers alternating; the last panel writes dst itself, its columns
// in the inverse's order.  Dynamic shared memory: the panel and the
// elimination's scratch, neither live during the update GEMM, which reuses
// the same memory as its staging buffers.  The panel's row map is read by
// that GEMM, so it lives in the static SmemInv.  In a group every CTA
// eliminates its own copy of the panel (the elimination is a serial chain,
// which a broadcast would only lengthen) and the update's tiles are shared.
// Returns 1 (and zeros dst) on a zero pivot.
template <int NB>
__device__ __noinline__ int gj_invert_tiled(const Group& grp, double2* X0, double2* X1, double2* dst, double2* dst2,
                                            double2* smem, SmemInv& s) {
  constexpr int n = NB, PWM = panel_width(n), LD = n + 2;
  double2* panel = smem;
  double2* scr = panel + LD * PWM;
  int16_t* rmap = s.rmap;
  const int tid = threadIdx.x;
  auto load_panel = [&](const double2* src, int PW) {   // columns -> shared memory (pitch LD)
    for (int e = tid; e < n * PW; e += kThreads) {
      const int jj = e / n, i = e - jj * n;
      cp_async16(panel + i + jj * LD, src + e);
    }
    cp_async_commit();
    for (int i = tid; i < n; i += kThreads) rmap[i] = (int16_t)i;
    cp_async_wait<0>();
    __syncthreads();
  };
  if constexpr (PWM >= n) {
    load_panel(X0, n);
    return gj_invert_panel<NB, 2>(grp, panel, dst, dst2, s, scr);
  }
  double2* cur = X0;
  double2* nxt = X1;
  if (tid == 0) s.singular = 0;
  for (int p0 = 0; p0 < n; p0 += PWM) {
    const int PW = (n - p0) < PWM ? (n - p0) : PWM;
    // (a) panel columns of the current matrix
    load_panel(cur + (size_t)p0 * n, PW);
    // (b) elimination of the panel in sub-blocks of 8 columns: each sub-block
    //     is eliminated unblocked with its columns in registers (gj_subblock;
    //     its row interchanges applied to the whole panel), then the panel's
    //     other columns get the sub-block's transformation as one rank-8
    //     update (the same U R form as the panel's own update below), so the
    //     panel is read and written once per sub-block instead of once per
    //     column.
    for (int sb0 = 0; sb0 < PW; sb0 += 8) {
      gj_subblock<NB>(n, LD, panel, PW, p0, sb0, scr, rmap, s);
      if (s.singular) break;
      panel_rank8_update<NB>(n, LD, panel, PW, p0, sb0, scr);
    }
    if (s.singular) break;
    // the last panel writes the inverse itself: its column j is column
    // colsrc[j] of the eliminated matrix (the interchanges undone), i.e.
    // column c goes to coldst[c]
    const bool last = p0 + PW >= n;
    if (last) undo_interchanges(n, s);
    // (c) eliminated panel -> next matrix (its rows are already in the new order)
    for (int e = tid + kThreads * grp.rank; e < n * PW; e += kThreads * grp.size) {
      const int jj = e / n, i = e - jj * n;
      const double2 v = panel[i + jj * LD];
      nxt[(size_t)p0 * n + e] = v;
      if (last) {
        const size_t o = i + (size_t)s.coldst[p0 + jj] * n;
        dst[o] = v;
        if (dst2) dst2[o] = v;
      }
    }
    grp.sync();
    // (d) other columns: with R = rows rmap[P] of cur and U the panel,
    //     nxt[P, j] = U[P, :] R[:, j],   nxt[i, j] = cur[rmap[i], j] + U[i, :] R[:, j]
    gemm_tiles(
        grp, n, n - PW, PW, nxt + (size_t)p0 * n, n, false, cur, n, false, smem,
        [&](int i, int j) {
          return i < p0 || i >= p0 + PW ? cur[(size_t)rmap[i] + (size_t)j * n] : czero();
        },
        [&](int i, int j, double2 v) {
          if (last) {
            const size_t o = i + (size_t)s.coldst[j] * n;
            dst[o] = v;
            if (dst2) dst2[o] = v;
          } else {
            nxt[i + (size_t)j * n] = v;
          }
        },
        rmap + p0, [&](int j) { return j < p0 ? j : j + PW; });
    grp.sync();
    double2* t = cur;
    cur = nxt;
    nxt = t;
  }
  const int sing = s.singular;
  __syncthreads();
  return sing ? zero_inverse(grp, n, dst, dst2) : 0;
}

// Gauss-Jordan inverse of the n x n block X0 (global memory, ld n, destroyed)
// for the block sizes without a panel form, result into dst (and dst2); X1: a
// second global block.  Eight columns at a time: eliminated in registers
// (gj_subblock), then all other columns get them as one rank-8 update, its
// four real products per half summed apart and added to the element once.
// Longer sums round more often: at nb = 80 .. 248 the inverse's error against
// 64 bits is 1.2 to 1.6 times the unblocked elimination's with panels of 48,
// 0.7 to 1.0 times with this form (solves at nb = 80 .. 200: 1.2 to 1.7 and
// 1.00 to 1.08 times).  Rows are gathered through the map of the eight
// columns' interchanges while the two blocks alternate, as in
// gj_invert_tiled.  Bound by the elimination's column chain and by the round
// trips of n / 8 passes over the block through L2, so a warp has four output
// subtiles' loads in flight (200 energies at nb = 104, nx = 30: 152 ms; panels
// through the tiled product 151 ms at 48 columns, 195 ms at 8; unblocked, with
// the register-direct product, 217 ms).  In a group every CTA eliminates its
// own copy of the eight columns; the subtiles are shared.
// Returns 1 (and zeros dst) on a zero pivot.
template <int NB>
__device__ __noinline__ int gj_invert_rank8(const Group& grp, int n, double2* X0, double2* X1, double2* dst,
                                            double2* dst2, double2* smem, SmemInv& s) {
  constexpr int KB = 8, kRow = 12;                   // pivot rows' pitch: 4 x 2 fragments on distinct banks
  static_assert(KB * (NB + 2) + kRow * NB + sub_scratch(NB) <= kSmemValues, "shared memory");
  const int LD = n + 2, r8 = n >> 3, tiles = r8 * (r8 - 1);
  double2* panel = smem;                             // [8][LD]
  double2* rows = panel + KB * LD;                   // [n][kRow] pivot rows of the other columns
  double2* scr = rows + kRow * n;
  int16_t* rmap = s.rmap;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int step = kWarps * grp.size;
  double2* cur = X0;
  double2* nxt = X1;
  if (tid == 0) s.singular = 0;
  for (int p0 = 0; p0 < n; p0 += KB) {
    for (int e = tid; e < KB * n; e += kThreads) {
      const int jj = e / n, i = e - jj * n;
      cp_async16(panel + i + jj * LD, cur + (size_t)p0 * n + e);
    }
    cp_async_commit();
    for (int i = tid; i < n; i += kThreads) rmap[i] = (int16_t)i;
    cp_async_wait<0>();
    __syncthreads();
    gj_subblock<NB, true>(n, LD, panel, KB, p0, 0, scr, rmap, s);
    if (s.singular) break;
    // the last step writes the inverse itself: column c goes to coldst[c]
    const bool last = p0 + KB >= n;
    if (last) undo_interchanges(n, s);
    auto put = [&](int i, int j, double2 v) {
      if (last) {
        const size_t o = i + (size_t)s.coldst[j] * n;
        dst[o] = v;
        if (dst2) dst2[o] = v;
      } else {
        nxt[i + (size_t)j * n] = v;
      }
    };
    for (int e = tid; e < KB * n; e += kThreads) {
      const int t = e & (KB - 1), j = e >> 3;
      if (j < p0 || j >= p0 + KB) cp_async16(rows + t + j * kRow, cur + rmap[p0 + t] + (size_t)j * n);
    }
    cp_async_commit();
    for (int e = tid + kThreads * grp.rank; e < KB * n; e += kThreads * grp.size) {
      const int jj = e / n, i = e - jj * n;
      put(i, p0 + jj, panel[i + jj * LD]);
    }
    cp_async_wait<0>();
    __syncthreads();
    constexpr int U = 4;
    for (int t0 = warp + kWarps * grp.rank; t0 < tiles; t0 += U * step) {
      double2 x[U][2];
      int row[U], col[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int q = t0 + u * step, b = q / r8;
        row[u] = 8 * (q - b * r8);
        col[u] = 8 * (8 * b < p0 ? b : b + 1);
        x[u][0] = x[u][1] = czero();
        if (q < tiles && row[u] != p0) {
          const double2* at = cur + rmap[row[u] + g] + (size_t)(col[u] + 2 * t4) * n;
          x[u][0] = at[0];
          x[u][1] = at[n];
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (t0 + u * step >= tiles) break;
        double rr[2][2] = {}, ii[2][2] = {}, ri[2][2] = {}, ir[2][2] = {};   // [4 columns of the panel][output]
#pragma unroll
        for (int ks = 0; ks < 2; ks++) {
          const double2 a = panel[row[u] + g + (4 * ks + t4) * LD];
          const double2 b = rows[4 * ks + t4 + (col[u] + g) * kRow];
          dmma884(rr[ks][0], rr[ks][1], a.x, b.x);
          dmma884(ri[ks][0], ri[ks][1], a.x, b.y);
          dmma884(ii[ks][0], ii[ks][1], a.y, b.y);
          dmma884(ir[ks][0], ir[ks][1], a.y, b.x);
        }
#pragma unroll
        for (int c = 0; c < 2; c++)
          put(row[u] + g, col[u] + 2 * t4 + c,
              make_double2(x[u][c].x + ((rr[0][c] - ii[0][c]) + (rr[1][c] - ii[1][c])),
                           x[u][c].y + ((ri[0][c] + ir[0][c]) + (ri[1][c] + ir[1][c]))));
      }
    }
    grp.sync();
    double2* t = cur;
    cur = nxt;
    nxt = t;
  }
  const int sing = s.singular;
  __syncthreads();
  return sing ? zero_inverse(grp, n, dst, dst2) : 0;
}

}  // namespace
}  // namespace rgf
