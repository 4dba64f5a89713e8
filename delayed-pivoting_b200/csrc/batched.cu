// Batched delayed-pivoting LU: thousands of independent square matrices of
// uneven sizes (n <= 512) in one persistent launch.
//
// Semantics per matrix are those of delayed_lu/delayed_dgetrf.cpp:129-251
// (column partial pivoting, acceptance |alpha| > threshold, full-pivot
// fallback on a column without an acceptable pivot after bringing the far
// columns up to date, delay when the whole active block has none, swap
// histories, compact L\U in place).  Blocking only changes rounding, so the
// records equal the single-matrix path's and the reference's.
//
// One CTA factors one matrix at a time; CTAs pull matrix indices from a device
// work queue ordered largest first, so the tail is short.  The orders fall into
// four size classes with a CTA shape each (Geo), launched one behind the other
// so that a class's CTAs take the SMs the class before leaves free
// (programmatic dependent launch).  Per panel of nb columns (at most the
// class's window of 16):
//   panel      the n - b panel rows live in REGISTERS, a row per thread for the
//              whole panel, factored in sub-panels of 8 columns with a rank-8 update of
//              the rest of the register window after each.  A row swap only
//              exchanges the logical positions the owners keep (no data
//              moves); the candidate for column s + 1 is taken while column
//              s + 1 is updated, each warp's winning lane pushes its row into
//              shared memory, and ONE barrier per column publishes the warp
//              winners - every thread then knows the pivot row and reads it
//              from shared memory.  Ties go to the smaller logical row, NaN
//              never wins (delayed_dgetrf_cuda.cu:13-20, :46).
//   write-back the panel, in logical row order, to the matrix and to shared
//              memory (L11 and L21 for the update)
//   update     per STAGE trailing columns: the panel's composite row
//              permutation (at most 2 nb rows move) and U12 = L11^{-1} A12,
//              through a shared tile, then A22 -= L21 U12 on the FP64 tensor
//              path (mma.sync m16n8k4, warp tiles 32 x 32)
//   left       the permutations owed to the finished columns, once per matrix
//   fallback   materialize the far columns with the executed prefix, 2-D
//              argmax (smaller column, then smaller row on ties), full-row and
//              full-column swaps, restart the panel at k with the pivot placed
// The panel width is chosen per size bucket (dp_batch_options.nb_bucket);
// dp_batch_autotune fills that table by timing the candidates.  One above the
// window runs as the window.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include <cuda_bf16.h>

#include "delayed_pivoting_b200.h"
#include "dp_device.cuh"
#include "dp_kernels.h"
#include "serve_kernels.h"

namespace dp {
namespace batch {

constexpr int kMaxN = DP_BATCH_MAX_N;
constexpr int kMaxNb = DP_BATCH_MAX_NB;   // panel width limit
constexpr int kWindow = 16;               // panel columns a matrix's CTA holds; wider panels run as this
constexpr int kSb = 8;                    // sub-panel width inside the window
constexpr int kMaxWarps = 16;
constexpr int kLeftMoves = 2 * kMaxN;     // row moves kept for the columns on the left,
constexpr int kLeftSegs = 64;             // in at most this many segments
constexpr int kNone = INT_MAX;            // logical position of a thread's missing row

// One CTA shape: T threads with RPT panel rows each and a register window of
// NB panel columns; trailing updates in rounds of STAGE columns, the warps
// WM x WN over tiles of 32 x 32; MINB CTAs per SM.
template <int T_, int RPT_, int NB_, int STAGE_, int WM_, int MINB_>
struct Geo {
  static constexpr int T = T_, RPT = RPT_, NB = NB_, STAGE = STAGE_, WM = WM_, MINB = MINB_;
  static constexpr int kWarps = T / 32, WN = kWarps / WM;
  static constexpr int kRows = T * RPT;            // largest order
  static constexpr int kTileM = 32 * WM, kTileN = 32 * WN;
  static constexpr int kLdb = NB + 4;              // shared U12 tile stride (== 4 mod 16)
  static_assert(kWarps % WM == 0 && kWarps <= kMaxWarps && STAGE % kTileN == 0 && STAGE <= T && NB % 16 == 0 && NB <= kMaxNb && kWarps * kRows <= kRows * NB + STAGE * kLdb,
                "geometry");
};

struct Params {
  double* base;
  const long long* offsets;      // first element of matrix i (lda = n_i)
  const int* ns;                 // order of matrix i
  const long long* rec_offsets;  // first record of matrix i
  const int* order;              // processing order (largest first)
  int count;
  int* queue;                    // work counter, zeroed before the launch
  int* ipiv;
  int* jpiv;
  int* info;
  unsigned long long* ties;      // near-tie detector: decisions checked, order-sensitive
                                 // ones, bits of the largest runner-up / winner ratio
  double threshold;
  int nb_bucket[DP_BATCH_BUCKETS];
  int pr;                        // column stride of the shared panel
};

__host__ __device__ constexpr int panel_ld(int rows) {
  // >= rows and == 4 (mod 16) doubles: the DMMA A fragments read from the
  // panel are conflict-free
  return ((rows + 11) / 16) * 16 + 4;
}

__host__ __device__ inline int bucket_of(int n) {
  return n < 64 ? 0 : n < 128 ? 1 : n < 256 ? 2 : 3;
}

struct Smem {
  // dynamic part: P [pr * NB], then Bs [STAGE * kLdb]
  double crow[2][kMaxWarps][kSb + 1]; // each warp's candidate row (sub-panel part) and the
                                   // reciprocal of its pivot entry, by step parity
  double rval[2][kMaxWarps];          // each warp's best magnitude (>= 0) and logical row
  int rkey[2][kMaxWarps];
  double rsec[2][kMaxWarps];          // each warp's runner-up magnitude (near-tie detector)
  double psave[kSb][kMaxNb + 2];      // the current sub-panel's pivot rows, whole window
  // The panel's composite row permutation: block row i takes the content of
  // panel row src_blk[i], panel row ext_dst[j] below the block that of ext_src[j]
  short src_blk[kMaxNb], ext_dst[kMaxNb], ext_src[kMaxNb];
  int ext_count;
  // Row moves still owed to the finished columns on the left (settle_left):
  // segment t covers the columns [seg_col[t], seg_end[t]); its moves (matrix
  // row lm_src -> lm_dst, entries [seg_at[t], seg_at[t + 1])) belong to the
  // columns before seg_col[t].
  short lm_dst[kLeftMoves], lm_src[kLeftMoves];
  short seg_col[kLeftSegs], seg_end[kLeftSegs], seg_at[kLeftSegs + 1];
  int segs;
  short cur[kMaxN];
  double fval[kMaxWarps];             // fallback search
  double fsec[kMaxWarps];
  int frow[kMaxWarps];
  int fcol[kMaxWarps];
  int slot;
};

__device__ __forceinline__ void mma_f64(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// Mixed form of the trailing update: BF16 pieces x = x1 + x2 [+ x3] (each the
// BF16 rounding of what the earlier ones left, as in the single-matrix
// tensor-core update), products of pieces (i, j) with i + j <= TERMS - 1 on
// mma.sync.m16n8k16 with FP32 accumulation.
template <int TERMS>
__device__ __forceinline__ void split_pieces(double x, __nv_bfloat16 (&piece)[TERMS]) {
#pragma unroll
  for (int t = 0; t < TERMS; ++t) {
    piece[t] = __double2bfloat16(x);
    x -= (double)__bfloat162float(piece[t]);
  }
}

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4],
                                         const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Candidate (magnitude v, logical row key) beats (cv, ck)?
__device__ __forceinline__ bool beats(double v, int key, double cv, int ck) {
  return v > cv || (v == cv && key < ck);
}

// Best (largest magnitude, then smallest key) of the warp's candidates.  A
// magnitude is >= 0 (a lane without a candidate offers 0 with key kNone), so
// its bit pattern orders like its value: max of the high word, then of the
// low word among the lanes holding that high word, then min key among the
// lanes holding the maximum - three dependent warp reductions.
__device__ __forceinline__ void warp_best(double v, int key, double& bv, int& bk) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  bk = __reduce_min_sync(0xffffffffu, (hi == mhi && lo == mlo) ? key : kNone);
  bv = __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
}

// The same, and the largest of the lanes' non-negative magnitudes `w`, whose
// reductions go between the dependent ones.
__device__ __forceinline__ void warp_best_and_max(double v, int key, double w, double& bv, int& bk,
                                                  double& mw) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned long long x = (unsigned long long)__double_as_longlong(w);
  const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  const unsigned xhi = (unsigned)(x >> 32), xlo = (unsigned)x;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned whi = __reduce_max_sync(0xffffffffu, xhi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  const unsigned wlo = __reduce_max_sync(0xffffffffu, xhi == whi ? xlo : 0u);
  bk = __reduce_min_sync(0xffffffffu, (hi == mhi && lo == mlo) ? key : kNone);
  bv = __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
  mw = __longlong_as_double((long long)(((unsigned long long)whi << 32) | wlo));
}

// Largest of the lanes' non-negative magnitudes (bit-pattern order).
__device__ __forceinline__ double warp_max_pos(double v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  return __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
}

// Offers candidate (v, key) to a running best (cv, ck) with runner-up cs:
// the magnitude that does not win becomes a runner-up candidate.
__device__ __forceinline__ bool offer(double v, int key, double& cv, int& ck, double& cs) {
  if (beats(v, key, cv, ck)) {
    cs = fmax(cs, cv);
    cv = v;
    ck = key;
    return true;
  }
  cs = fmax(cs, v);
  return false;
}

// Factor panel columns [b, b + w) of the n x n matrix A (rows b..n-1).
// Returns the first step without an acceptable pivot (-1: all w steps done).
// Writes the panel back in logical row order to A and to P (column stride
// pr), the step pivots to ipiv, and the rows that moved to s.src_blk / s.ext_*.
//
// Thread t owns the panel rows t + i T (physical rows) and keeps a window of
// NB of their columns in registers, x[i][c] = panel column base + c.  The
// window is factored in sub-panels of kSb columns: kSb unrolled steps of
// rank-1 updates confined to the sub-panel (one barrier each), then the
// sub-panel's pivot rows are solved for the rest of the window (U12 =
// L11^{-1} A12, in shared memory) and the remaining rows take one rank-kSb
// update; finished columns go to P in physical row order and the window
// shifts by kSb.  The compiled step body is one sub-panel long.
template <class G>
__device__ __forceinline__ int panel_regs(double* A, int n, int lda, int b, int w,
                                          bool positioned, double thr, double* P, int pr,
                                          Smem& s, int* ipiv, DecisionTally& tally) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rows = n - b;
  double x[G::RPT][G::NB];
  int lp[G::RPT];
#pragma unroll
  for (int i = 0; i < G::RPT; ++i) {
    const int r = tid + i * G::T;
    lp[i] = r < rows ? r : kNone;
#pragma unroll
    for (int c = 0; c < G::NB; ++c)
      x[i][c] = (r < rows && c < w) ? A[idx(b + r, b + c, lda)] : 0.0;
  }

  // warp best of the lane candidates (cv >= 0, ck from the lane's row ci);
  // the winning lane pushes its sub-panel columns j.., the reciprocal of its
  // entry in column j (computed by every lane ahead of the reductions, off
  // the path after the barrier) and the warp's result
  // The last decision's runner-up: t_lane holds this lane's share of it until the
  // next push, whose reductions hide it (warp 0 records, from its lane 0).
  int t_k = -1;
  double t_best = 0.0, t_lane = 0.0;
  auto push = [&](int j, int par, double cv, int ck, int ci, double cs) {
    double pv = 0.0;
#pragma unroll
    for (int c = 0; c < kSb; ++c)
      if (c == j) pv = ci ? x[G::RPT - 1][c] : x[0][c];
    const double rinv = 1.0 / pv;
    double wv, second;
    int wk;
    warp_best_and_max(cv, ck, t_lane, wv, wk, second);
    if (warp == 0 && t_k >= 0) {
      tally.note(t_k, t_best, second);  // (alike in every lane; one is flushed)
      t_k = -1;
    }
    // the warp's runner-up: the winner lane's runner-up, every other lane's best
    const double ws = warp_max_pos((wk != kNone && ck == wk) ? cs : (ck != kNone ? cv : cs));
    if (wk != kNone ? ck == wk : lane == 0) {
      if (wk != kNone) {
#pragma unroll
        for (int c = 0; c < kSb; ++c)
          if (c >= j) s.crow[par][warp][c] = ci ? x[G::RPT - 1][c] : x[0][c];
        s.crow[par][warp][kSb] = rinv;
      }
      s.rval[par][warp] = wv;
      s.rkey[par][warp] = wk;
      s.rsec[par][warp] = ws;
    }
  };
  // candidate of window column 0 among the rows at logical positions >= first
  auto first_candidate = [&](int first, bool placed) {
    double cv = 0.0, cs = 0.0;
    int ck = kNone, ci = 0;
#pragma unroll
    for (int i = 0; i < G::RPT; ++i) {
      if (lp[i] == kNone || lp[i] < first) continue;
      // a placed pivot (after a fallback) is the only candidate of its step
      if (placed && lp[i] != first) continue;
      const double v = placed ? INFINITY : fabs(x[i][0]);
      if (offer(v, lp[i], cv, ck, cs)) ci = i;
    }
    push(0, first & 1, cv, ck, ci, cs);
  };

  first_candidate(0, positioned);
  if (tid == 0) s.ext_count = 0;
  __syncthreads();

  int stop = -1;
  int base = 0;  // panel column of window column 0
  while (base < w) {
    const int sw = min(kSb, w - base);
    int kd = sw;  // steps executed in this sub-panel
#pragma unroll
    for (int j = 0; j < kSb; ++j) {
      if (j >= sw) break;
      const int st = base + j, par = st & 1;
      const int q = lane & (G::kWarps - 1);  // (lanes >= kWarps repeat the others)
      const double rv = s.rval[par][q], rs = s.rsec[par][q];
      const int rk = s.rkey[par][q];
      double bv;
      int key;  // logical row and warp of the winner: rows below 2^26
      warp_best(rv, rk == kNone ? kNone : rk * kMaxWarps + q, bv, key);
      const int bk = key == kNone ? kNone : key / kMaxWarps;
      const int bw = key == kNone ? 0 : key % kMaxWarps;
      const bool placed = positioned && st == 0;
      if (!placed) {
        t_k = b + st;
        t_best = bk != kNone ? bv : 0.0;
        t_lane = bk != kNone && q == bw ? rs : (rk != kNone ? rv : rs);
      }
      if (!placed && !(bv > thr)) {
        stop = st;
        kd = j;
        break;
      }
      const double* prow = s.crow[par][bw];
      const int p = bk;  // logical position of the pivot row before the swap
      if (tid == 0 && !placed) ipiv[b + st] = b + p;
      const double inv = prow[kSb];
      double cv = 0.0, cs = 0.0;
      int ck = kNone, ci = 0;
#pragma unroll
      for (int i = 0; i < G::RPT; ++i) {
        if (lp[i] == p) {
          lp[i] = st;  // the pivot row: keep its window for the U12 solve
#pragma unroll
          for (int g = 0; g < G::NB / kSb; ++g)
            if (base + g * kSb < w) {
#pragma unroll
              for (int c = g * kSb; c < (g + 1) * kSb; ++c) s.psave[j][c] = x[i][c];
            }
        } else if (lp[i] == st) {
          lp[i] = p;
        }
        if (lp[i] == kNone || lp[i] <= st) continue;
        const double l = x[i][j] * inv;
        x[i][j] = l;
#pragma unroll
        for (int c = j + 1; c < kSb; ++c) x[i][c] = fma(-l, prow[c], x[i][c]);
        if (j + 1 < kSb) {
          const double v = fabs(x[i][j + 1 < kSb ? j + 1 : 0]);
          if (offer(v, lp[i], cv, ck, cs)) ci = i;
        }
      }
      if (j + 1 < sw) {
        push(j + 1, par ^ 1, cv, ck, ci, cs);
        __syncthreads();
      }
    }
    // the window columns right of the sub-panel take its kd executed steps
    const int rest = w - base - kSb;
    __syncthreads();  // psave complete
    if (kd > 0 && rest > 0) {
      for (int c = kSb + tid; c < kSb + rest; c += G::T) {
        double u[kSb];  // a step's multiples go to all later rows before the next step
#pragma unroll
        for (int j = 0; j < kSb; ++j) u[j] = j < kd ? s.psave[j][c] : 0.0;
#pragma unroll
        for (int t = 0; t < kSb - 1; ++t)
#pragma unroll
          for (int j = t + 1; j < kSb; ++j)
            if (j < kd) u[j] = fma(-s.psave[j][t], u[t], u[j]);
#pragma unroll
        for (int j = 1; j < kSb; ++j)
          if (j < kd) s.psave[j][c] = u[j];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < G::RPT; ++i) {
        if (lp[i] == kNone || lp[i] < base) continue;
        if (lp[i] < base + kd) {  // a pivot row of this sub-panel takes its U12 row
          const double* u = s.psave[lp[i] - base];
#pragma unroll
          for (int g = 1; g < G::NB / kSb; ++g)
            if (base + g * kSb < w) {
#pragma unroll
              for (int c = g * kSb; c < (g + 1) * kSb; ++c) x[i][c] = u[c];
            }
        } else {
#pragma unroll
          for (int g = 1; g < G::NB / kSb; ++g)
            if (base + g * kSb < w) {
#pragma unroll
              for (int t = 0; t < kSb; ++t)
                if (t < kd) {
                  const double l = x[i][t];
#pragma unroll
                  for (int c = g * kSb; c < (g + 1) * kSb; ++c)
                    x[i][c] = fma(-l, s.psave[t][c], x[i][c]);
                }
            }
        }
      }
    }
    if (stop >= 0) break;
    // finished sub-panel columns to P (physical rows); shift the window
#pragma unroll
    for (int i = 0; i < G::RPT; ++i) {
      if (lp[i] == kNone) continue;
      double* pc = P + tid + i * G::T + (size_t)base * pr;
#pragma unroll
      for (int c = 0; c < kSb; ++c)
        if (c < sw) pc[c * pr] = x[i][c];
#pragma unroll
      for (int c = 0; c < G::NB - kSb; ++c) x[i][c] = x[i][c + kSb];
#pragma unroll
      for (int c = G::NB - kSb; c < G::NB; ++c) x[i][c] = 0.0;
    }
    base += kSb;
    if (base < w) {
      first_candidate(base, false);
      __syncthreads();
    }
  }
  if (warp == 0 && t_k >= 0) {  // the panel's last decision
    const double second = warp_max_pos(t_lane);
    tally.note(t_k, t_best, second);  // (alike in every lane; one is flushed)
  }
  // the window's remaining columns to P (physical rows)
#pragma unroll
  for (int i = 0; i < G::RPT; ++i) {
    if (lp[i] == kNone) continue;
    double* pc = P + tid + i * G::T;
#pragma unroll
    for (int c = 0; c < G::NB; ++c)
      if (base + c < w) pc[(size_t)(base + c) * pr] = x[i][c];
  }
  __syncthreads();
  // rows to their logical positions, in P and in the matrix
#pragma unroll
  for (int i = 0; i < G::RPT; ++i) {
    if (lp[i] == kNone) continue;
    const double* pc = P + tid + i * G::T;
#pragma unroll
    for (int c = 0; c < G::NB; ++c)
      if (c < w) x[i][c] = pc[c * pr];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < G::RPT; ++i) {
    if (lp[i] == kNone) continue;
    const int r = lp[i], phys = tid + i * G::T;
#pragma unroll
    for (int c = 0; c < G::NB; ++c)
      if (c < w) {
        A[idx(b + r, b + c, lda)] = x[i][c];
        if (r != phys) P[r + c * pr] = x[i][c];
      }
    if (r < w) {
      s.src_blk[r] = (short)phys;
    } else if (r != phys) {  // at most one row per executed step
      const int j = atomicAdd(&s.ext_count, 1);
      s.ext_dst[j] = (short)r;
      s.ext_src[j] = (short)phys;
    }
  }
  return stop;
}

// The row moves kept for the finished columns, applied: each column is read
// and written once, coalesced, through a buffer of its warp in shared memory
// (`buf`, n doubles a warp: P and the U12 tile behind it), instead of 2 nb
// scattered elements per panel and column (n = 512: 0.5 of 3.0 ms).  From the
// last segment back, s.cur holds the composite of the moves after the segment:
// position r of its columns takes row cur[r].
template <class G>
__device__ __forceinline__ void settle_left(double* A, int lda, int n, double* buf, Smem& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* const mine = buf + warp * n;
  __syncthreads();  // the moves are listed, buf is free
  const int segs = s.segs;
  for (int r = tid; r < n; r += G::T) s.cur[r] = (short)r;
  __syncthreads();
  for (int t = segs - 1; t >= 0; --t) {
    const int c0 = s.seg_col[t], c1 = s.seg_end[t];
    if (t + 1 < segs)
      for (int c = c0 + warp; c < c1; c += G::kWarps) {
        double* const col = A + idx(0, c, lda);
        for (int r = c1 + lane; r < n; r += 32) mine[r] = col[r];
        __syncwarp();
        for (int r = c1 + lane; r < n; r += 32) {
          const int from = s.cur[r];
          if (from != r) col[r] = mine[from];
        }
        __syncwarp();
      }
    // cur <- (this segment's moves) o cur; a moved row is looked up in the
    // list through `back`, the moves' sources by position
    const int m0 = s.seg_at[t], m1 = s.seg_at[t + 1];
    if (t == 0 || m0 == m1) continue;
    __syncthreads();  // the columns have read cur, and buf is free
    short* const back = reinterpret_cast<short*>(buf);
    for (int r = tid; r < n; r += G::T) back[r] = (short)r;
    __syncthreads();
    for (int m = m0 + tid; m < m1; m += G::T) back[s.lm_dst[m]] = s.lm_src[m];
    __syncthreads();
    for (int r = tid; r < n; r += G::T) s.cur[r] = back[s.cur[r]];
    __syncthreads();
  }
  __syncthreads();
  if (tid == 0 && segs > 0) {  // the columns settled so far are owed what comes after
    s.seg_end[0] = s.seg_end[segs - 1];
    s.seg_col[0] = 0;
    s.seg_at[0] = s.seg_at[1] = 0;
    s.segs = 1;
  }
  __syncthreads();
}

// Adds the segment of columns [c0, c1) whose `ext` and block moves (a panel's,
// rows from b) the columns before c0 are still owed; every thread calls it.
template <class G>
__device__ __forceinline__ void keep_panel_moves(int b, int w, int c1, Smem& s) {
  // one warp, in list order (the entries' order within a segment is free)
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int at = s.seg_at[s.segs];
    const bool blk = lane < w && s.src_blk[lane] != lane;
    const unsigned mb = __ballot_sync(~0u, blk);
    if (blk) {
      const int m = at + __popc(mb & ((1u << lane) - 1u));
      s.lm_dst[m] = (short)(b + lane);
      s.lm_src[m] = (short)(b + s.src_blk[lane]);
    }
    at += __popc(mb);
    const int ext = s.ext_count;
    if (lane < ext) {
      s.lm_dst[at + lane] = (short)(b + s.ext_dst[lane]);
      s.lm_src[at + lane] = (short)(b + s.ext_src[lane]);
    }
    __syncwarp();
    if (lane == 0) {
      const int t = s.segs;
      s.seg_col[t] = (short)b;
      s.seg_end[t] = (short)c1;
      s.seg_at[t + 1] = (short)(at + ext);
      s.segs = t + 1;
    }
  }
}

// Right of a panel of w columns that executed `kd` steps at [b, b + kd): for
// the columns [c0, n), the panel's row permutation, U12 = L11^{-1}
// A(b:b+kd, :) (written back) and A(b+kd:n, :) -= L21 U12, with L11 / L21 the
// shared panel P.  The permutation is part of the staging: a group of NB lanes
// gathers a column's new block rows into the shared tile and carries the
// displaced rows below the block to their places, all of a column's loads
// before its stores; the solve then runs from shared memory with a thread per
// column, and the block rows go back coalesced.  (As passes of their own over
// global memory, the permutation four lanes a column and the solve a thread a
// column, they took 0.5 and 0.9 of the 3.0 ms of an n = 512 matrix: every
// element access of a warp was a transaction of its own.)  TERMS = 0: the product in FP64 (DMMA); TERMS = 2 / 3: the
// BF16 split product (3 / 6 products, FP32 accumulation), subtracted in FP64.
template <class G, int TERMS>
__device__ __forceinline__ void trailing_update(double* A, int lda, int n, int b, int w, int kd,
                                                int c0, const double* P, int pr, double* Bs,
                                                const Smem& s) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp / G::WN, wn = warp % G::WN;
  const int row0 = b + kd;
  const int M = n - row0, N = n - c0;
  const int kp = (kd + 3) & ~3;
  const double* L21 = P + kd;  // panel rows kd.. = matrix rows row0..
  for (int n0 = 0; n0 < N; n0 += G::STAGE) {
    const int ns = min(G::STAGE, N - n0);
    __syncthreads();  // Bs is free
    constexpr int kLanes = G::NB;               // lanes per column
    constexpr int kCols = 32 / kLanes;          // columns per warp and pass
    constexpr int kUnroll = 4;
    const int li = lane % kLanes, lc = lane / kLanes;
    const int ext = s.ext_count;
    for (int q0 = warp * kCols * kUnroll; q0 < G::STAGE; q0 += G::kWarps * kCols * kUnroll) {
      double blk[kUnroll], low[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int c = q0 + u * kCols + lc;
        const double* col = A + idx(b, c0 + n0 + c, lda);
        blk[u] = (c < ns && li < w) ? col[s.src_blk[li]] : 0.0;
        low[u] = (c < ns && li < ext) ? col[s.ext_src[li]] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) Bs[(q0 + u * kCols + lc) * G::kLdb + li] = blk[u];
      __syncwarp();  // the pass's columns are read
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int c = q0 + u * kCols + lc;
        if (c < ns && li < ext) A[idx(b + s.ext_dst[li], c0 + n0 + c, lda)] = low[u];
      }
    }
    __syncthreads();
    if (tid < ns) {
      double* bcol = Bs + tid * G::kLdb;
      double u[G::NB];
#pragma unroll
      for (int i = 0; i < G::NB; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(bcol + i);
        u[i] = v.x;
        u[i + 1] = v.y;
      }
#pragma unroll
      for (int j = 0; j < G::NB - 1; ++j) {
        if (j >= kd) break;
        const double uj = u[j];
        const double2* pj = reinterpret_cast<const double2*>(P + j * pr);
#pragma unroll
        for (int i = j & ~1; i < G::NB; i += 2)
          if (i < kd) {  // (uniform; pairs: row i <= j and, at the end, row kd are left alone)
            const double2 l = pj[i / 2];
            if (i > j) u[i] = fma(-l.x, uj, u[i]);
            if (i + 1 > j && i + 1 < kd) u[i + 1] = fma(-l.y, uj, u[i + 1]);
          }
      }
#pragma unroll
      for (int i = 0; i < G::NB; i += 2)
        *reinterpret_cast<double2*>(bcol + i) = make_double2(u[i], u[i + 1]);
    }
    __syncthreads();
    for (int q = warp * kCols; q < ns; q += G::kWarps * kCols) {
      const int c = q + lc;
      double* e = Bs + c * G::kLdb + li;
      if (c < ns && li < w) A[idx(b + li, c0 + n0 + c, lda)] = *e;
      if (li >= kd) *e = 0.0;  // not part of the product
    }
    __syncthreads();
    for (int h = 0; h * G::kTileN < ns; ++h) {
      const int nc = min(G::kTileN, ns - h * G::kTileN);
      const double* Bh = Bs + h * G::kTileN * G::kLdb;
      double* C = A + idx(row0, c0 + n0 + h * G::kTileN, lda);
      for (int m0 = 0; m0 < M; m0 += G::kTileM) {
        const int rb = m0 + wm * 32;
        if (rb >= M) continue;  // warp-uniform; no barrier inside this loop
        double cf[2][4][4];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int r = rb + mi * 16 + g + 8 * (v >> 1);
              const int c = wn * 32 + ni * 8 + 2 * t + (v & 1);
              cf[mi][ni][v] = (r < M && c < nc) ? C[idx(r, c, lda)] : 0.0;
            }
        if constexpr (TERMS == 0) {
          // C itself is the accumulator (and -L21 the operand): half the
          // registers of a separate sum, which two CTAs per SM need
          for (int k0 = 0; k0 < kp; k0 += 4) {
            const int kk = k0 + t;
            const bool kok = kk < kd;
            double a[2][2];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
              const int r = rb + mi * 16 + g;
              a[mi][0] = (kok && r < M) ? -L21[r + kk * pr] : 0.0;
              a[mi][1] = (kok && r + 8 < M) ? -L21[r + 8 + kk * pr] : 0.0;
            }
            double bf[4];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) bf[ni] = Bh[(wn * 32 + ni * 8 + g) * G::kLdb + kk];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
              for (int ni = 0; ni < 4; ++ni) mma_f64(cf[mi][ni], a[mi][0], a[mi][1], bf[ni]);
          }
        } else {
          // m16n8k16 fragments: A (row r, k) at r = g / g + 8 and k = 2t, 2t + 1,
          // 2t + 8, 2t + 9 of the 16-deep step; B (k, column) at the same k
          // for column g; C as the FP64 fragments above
          float facc[2][4][4];
#pragma unroll
          for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
              for (int v = 0; v < 4; ++v) facc[mi][ni][v] = 0.0f;
          for (int k0 = 0; k0 < kd; k0 += 16) {
            uint32_t af[TERMS][2][4], bfr[TERMS][4][2];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
              for (int h = 0; h < 4; ++h) {  // register h: rows g (+8 for odd h), k pair
                const int r = rb + mi * 16 + g + 8 * (h & 1);
                const int kk = k0 + 2 * t + 8 * (h >> 1);
                __nv_bfloat16 lo[TERMS], hi[TERMS];
                split_pieces<TERMS>((r < M && kk < kd) ? L21[r + kk * pr] : 0.0, lo);
                split_pieces<TERMS>((r < M && kk + 1 < kd) ? L21[r + (kk + 1) * pr] : 0.0, hi);
#pragma unroll
                for (int q = 0; q < TERMS; ++q) af[q][mi][h] = pack_bf16(lo[q], hi[q]);
              }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const double* bc = Bh + (wn * 32 + ni * 8 + g) * G::kLdb;
                const int kk = k0 + 2 * t + 8 * h;
                __nv_bfloat16 lo[TERMS], hi[TERMS];
                split_pieces<TERMS>(kk < kd ? bc[kk] : 0.0, lo);
                split_pieces<TERMS>(kk + 1 < kd ? bc[kk + 1] : 0.0, hi);
#pragma unroll
                for (int q = 0; q < TERMS; ++q) bfr[q][ni][h] = pack_bf16(lo[q], hi[q]);
              }
#pragma unroll
            for (int d = 0; d < TERMS; ++d)
#pragma unroll
              for (int i = 0; i <= d; ++i)
#pragma unroll
                for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                  for (int ni = 0; ni < 4; ++ni) mma_bf16(facc[mi][ni], af[i][mi], bfr[d - i][ni]);
          }
#pragma unroll
          for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
              for (int v = 0; v < 4; ++v) cf[mi][ni][v] -= (double)facc[mi][ni][v];
        }
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int r = rb + mi * 16 + g + 8 * (v >> 1);
              const int c = wn * 32 + ni * 8 + 2 * t + (v & 1);
              if (r < M && c < nc) C[idx(r, c, lda)] = cf[mi][ni][v];
            }
      }
    }
  }
}

__device__ __forceinline__ bool better2(double va, int ca, int ra, double vb, int cb, int rb) {
  return va > vb || (va == vb && (ca < cb || (ca == cb && ra < rb)));
}

// 2-D argmax over the active block A(k:n, k:n): larger magnitude, then the
// smaller column, then the smaller row; NaN never wins.
template <class G>
__device__ __forceinline__ void active_argmax(const double* A, int lda, int n, int k, Smem& s,
                                              double& bv, int& br, int& bc, double& bs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double v0 = -1.0, s0 = 0.0;  // best, runner-up (largest of the other magnitudes)
  int r0 = INT_MAX, c0 = INT_MAX;
  const int rows = n - k;
  for (int c = k; c < n; ++c)
    for (int r = tid; r < rows; r += G::T) {
      const double v = fabs(A[idx(k + r, c, lda)]);
      if (v > v0) {  // (column, row) increase along this thread's scan
        s0 = fmax(s0, v0);
        v0 = v;
        r0 = k + r;
        c0 = c;
      } else {
        s0 = fmax(s0, v);
      }
    }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, v0, off);
    const double os = __shfl_xor_sync(0xffffffffu, s0, off);
    const int orr = __shfl_xor_sync(0xffffffffu, r0, off);
    const int oc = __shfl_xor_sync(0xffffffffu, c0, off);
    if (better2(ov, oc, orr, v0, c0, r0)) {
      s0 = fmax(os, v0);
      v0 = ov;
      r0 = orr;
      c0 = oc;
    } else {
      s0 = fmax(s0, ov);
    }
  }
  __syncthreads();
  if (lane == 0) {
    s.fval[warp] = v0;
    s.fsec[warp] = s0;
    s.frow[warp] = r0;
    s.fcol[warp] = c0;
  }
  __syncthreads();
  bv = s.fval[0];
  bs = s.fsec[0];
  br = s.frow[0];
  bc = s.fcol[0];
  for (int q = 1; q < G::kWarps; ++q)
    if (better2(s.fval[q], s.fcol[q], s.frow[q], bv, bc, br)) {
      bs = fmax(s.fsec[q], bv);
      bv = s.fval[q];
      br = s.frow[q];
      bc = s.fcol[q];
    } else {
      bs = fmax(bs, s.fval[q]);
    }
}

template <class G, int TERMS>
__device__ __forceinline__ void getrf_one(double* A, int n, int* ipiv, int* jpiv, int* info,
                                          int nb, double thr, double* P, int pr, double* Bs,
                                          Smem& s, DecisionTally& tally) {
  const int tid = threadIdx.x;
  const int lda = n;
  for (int i = tid; i < n; i += G::T) ipiv[i] = jpiv[i] = i;
  if (tid == 0) {
    *info = n;
    s.segs = 0;
    s.seg_at[0] = 0;
  }
  int b = 0;
  bool positioned = false;
  while (b < n) {
    const int w = min(nb, n - b), e = b + w;
    __syncthreads();  // P, Bs, the move lists and the records are settled
    if (s.segs + 3 > kLeftSegs || s.seg_at[s.segs] + 2 * kMaxNb + 2 > kLeftMoves)
      settle_left<G>(A, lda, n, P, s);
    const int stop = panel_regs<G>(A, n, lda, b, w, positioned, thr, P, pr, s, ipiv, tally);
    positioned = false;
    __syncthreads();  // panel written back, move list complete
    keep_panel_moves<G>(b, w, stop < 0 ? e : b + stop, s);
    if (stop < 0) {
      if (e < n) trailing_update<G, TERMS>(A, lda, n, b, w, w, e, P, pr, Bs, s);
      b = e;
      continue;
    }
    // column k has no acceptable pivot: bring the columns right of the panel
    // up to date for the executed steps, then search the whole active block
    const int k = b + stop;
    if (e < n && stop > 0) trailing_update<G, TERMS>(A, lda, n, b, w, stop, e, P, pr, Bs, s);
    __syncthreads();
    double bv, bs;
    int br, bc;
    active_argmax<G>(A, lda, n, k, s, bv, br, bc, bs);
    tally.note(k, bv > 0.0 ? bv : 0.0, bv > 0.0 ? bs : 0.0);
    if (!(bv > thr)) {
      if (tid == 0) *info = k;
      break;
    }
    if (tid == 0) {
      ipiv[k] = br;
      jpiv[k] = bc;
      if (br != k) {  // the columns before k are owed the row swap
        const int t = s.segs, at = s.seg_at[t];
        s.lm_dst[at] = s.lm_src[at + 1] = (short)k;
        s.lm_src[at] = s.lm_dst[at + 1] = (short)br;
        s.seg_col[t] = s.seg_end[t] = (short)k;
        s.seg_at[t + 1] = (short)(at + 2);
        s.segs = t + 1;
      }
    }
    if (br != k)
      for (int c = k + tid; c < n; c += G::T) {
        const double tmp = A[idx(k, c, lda)];
        A[idx(k, c, lda)] = A[idx(br, c, lda)];
        A[idx(br, c, lda)] = tmp;
      }
    __syncthreads();
    if (bc != k)
      for (int r = tid; r < n; r += G::T) {
        const double tmp = A[idx(r, k, lda)];
        A[idx(r, k, lda)] = A[idx(r, bc, lda)];
        A[idx(r, bc, lda)] = tmp;
      }
    b = k;
    positioned = true;
  }
  settle_left<G>(A, lda, n, P, s);
}

template <class G, int TERMS>
__global__ void __launch_bounds__(G::T, G::MINB) batched_getrf_kernel(Params p) {
  // the next size class's CTAs may take the SMs this one leaves free
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(16) double dsm[];
  __shared__ Smem s;
  double* P = dsm;
  double* Bs = dsm + (size_t)p.pr * G::NB;
  DecisionTally tally;
  while (true) {
    __syncthreads();  // s.slot is free
    if (threadIdx.x == 0) s.slot = atomicAdd(p.queue, 1);
    __syncthreads();
    const int slot = s.slot;
    if (slot >= p.count) break;
    const int i = p.order[slot];
    const int n = p.ns[i];
    const int bk = bucket_of(n);  // selected without indexing the parameter array
    const int nb = min(G::NB, bk == 0   ? p.nb_bucket[0]
                              : bk == 1 ? p.nb_bucket[1]
                              : bk == 2 ? p.nb_bucket[2]
                                        : p.nb_bucket[3]);
    getrf_one<G, TERMS>(p.base + p.offsets[i], n, p.ipiv + p.rec_offsets[i],
                        p.jpiv + p.rec_offsets[i], p.info + i, nb, p.threshold, P, p.pr, Bs, s,
                        tally);
  }
  if (threadIdx.x == 0) tally.flush(p.ties, p.ties + 1, p.ties + 2);
  // the launch ends no earlier than the classes before it: what follows on the
  // stream waits for the last class only
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One panel of the blocked LU (PanelParams, the same contract as
// panel_cluster_kernel) on ONE CTA, for panels of at most kMaxN rows and
// kMaxNb columns: the rows stay in registers and the pivot decisions,
// swaps (as relabelled row positions), scalings and rank-1 updates run with
// one CTA barrier per step and no cluster exchange (panel_regs, the batched
// kernel's panel).  Afterwards the composite row permutation is written as
// the swap lists the laswp kernel applies outside the panel.
template <class G>
__global__ void __launch_bounds__(G::T, 1) panel_small_kernel(PanelParams p) {
  after_previous_kernel();
  // every thread reads the same word before any barrier or state write
  if (p.gated && p.state->stop_k >= 0) return;
  extern __shared__ __align__(16) double dsm[];
  __shared__ Smem s;
  const int tid = threadIdx.x, lane = tid & 31;
  const int b = p.begin, w = p.end - p.begin;
  const int pr = panel_ld(p.m - b);
  DecisionTally tally;
  if (tid == 0) p.state->stop_k = -1;
  const int stop = panel_regs<G>(p.a, p.m, (int)p.lda, b, w, p.positioned != 0, p.threshold, dsm, pr,
                              s, p.ipiv, tally);
  __syncthreads();  // rows written back, move lists complete
  if (tid < 32) {
    const int ext = s.ext_count;
    const bool moved = lane < w && s.src_blk[lane] != lane;
    if (lane < w) p.swap_block[lane] = b + s.src_blk[lane];
    if (lane < ext) {
      p.swap_extra[2 * lane + 0] = b + s.ext_dst[lane];
      p.swap_extra[2 * lane + 1] = b + s.ext_src[lane];
    }
    const int changed = __popc(__ballot_sync(~0u, moved));
    if (lane == 0) {
      p.state->swap_count = ext;
      p.state->block_changed = changed;
      if (stop >= 0) p.state->stop_k = b + stop;
      tally.flush(p.state);
    }
  }
}

template <class G>
size_t dynamic_smem(int max_n) {
  return ((size_t)panel_ld(std::max(max_n, 1)) * G::NB + (size_t)G::STAGE * G::kLdb) *
         sizeof(double);
}

// Size classes, by order.  A matrix keeps one CTA busy with chains (a barrier a
// column, trips to L2 between phases), so the SM has to hold several: the class
// takes the fewest threads that give each row one, a window of 16 columns (a
// row's 32 registers leave room for 128 a thread in all) and U12 tiles sized
// for 2, 4 and 7 CTAs per SM.  2048 matrices of a class, one CTA shape of 256
// threads for all (two rows a thread, 32 columns, one CTA per SM) -> these:
// [32, 64] 2.29 -> 0.47 ms, [65, 128] 4.49 -> 1.22, [129, 256] 8.04 -> 3.52,
// [257, 512] 26.6 -> 17.6.  Measured slower: 32-column windows (up to 512:
// 20.6, up to 256: 5.3, up to 128: 2.0), 256 threads of two rows for the
// largest class (18.9; with two CTAs per SM 21.5), tiles of 16 x 32 with the
// next one's loads in flight (19.1).
using Geo3 = Geo<512, 1, kWindow, 256, 4, 1>;
using Geo2 = Geo<256, 1, kWindow, 128, 2, 2>;
using Geo1 = Geo<128, 1, kWindow, 128, 2, 4>;
using Geo0 = Geo<64, 1, kWindow, 64, 1, 7>;

// Panels of the blocked LU: a row per thread (STAGE and the warp grid unused).
template <int T>
using PanelGeo = Geo<T, 1, kMaxNb, 32 * (T / 64), 2, 1>;

int class_of(int n) { return n <= 64 ? 0 : n <= 128 ? 1 : n <= 256 ? 2 : 3; }

template <class G>
int launch_class(Params p, int max_n, int sms, int terms, bool behind, cudaStream_t st) {
  const void* fn = terms == 3   ? (const void*)batched_getrf_kernel<G, 3>
                   : terms == 2 ? (const void*)batched_getrf_kernel<G, 2>
                                : (const void*)batched_getrf_kernel<G, 0>;
  p.pr = panel_ld(max_n);
  const size_t smem = dynamic_smem<G>(max_n);
  if (!dp::ensure_smem(fn, smem)) return DP_CUDA_FAILURE;
  const int per_sm = dp::occupancy_once(fn, G::T, smem);
  if (per_sm < 1) return DP_CUDA_FAILURE;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(std::max(1, std::min(p.count, sms * per_sm)));
  cfg.blockDim = dim3(G::T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = behind ? 1 : 0;
  dp::note_launch();
  void* args[] = {&p};
  return cudaLaunchKernelExC(&cfg, fn, args) == cudaSuccess ? DP_SUCCESS : DP_CUDA_FAILURE;
}

// N(0,1) by the Box-Muller transform of two hashed uniforms (autotuner inputs).
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__global__ void fill_normal_kernel(double* x, long long len, uint64_t seed) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len;
       i += (long long)gridDim.x * blockDim.x) {
    const uint64_t h1 = mix64(seed ^ mix64((uint64_t)i));
    const uint64_t h2 = mix64(h1);
    const double u1 = ((h1 >> 11) + 1) * (1.0 / 9007199254740992.0);
    const double u2 = (h2 >> 11) * (1.0 / 9007199254740992.0);
    x[i] = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
  }
}

}  // namespace batch
}  // namespace dp

// ---------------------------------------------------------------------------
// Host side: batch plans, launches, CUDA-graph replay, autotuner.

struct dp_batch {
  int device = 0;
  int count = 0;
  dp::batch::Classes classes;
  int sms = 0;
  long long total_elements = 0;
  long long total_records = 0;
  std::vector<int> n;
  std::vector<long long> offsets, rec_offsets;
  int* d_n = nullptr;
  long long* d_offsets = nullptr;
  long long* d_rec = nullptr;
  int* d_order = nullptr;
  int* d_queue = nullptr;
  dp_batch_options opt{};
  // captured graph and the arguments it was captured with
  cudaGraphExec_t exec = nullptr;
  const void* g_args[4] = {nullptr, nullptr, nullptr, nullptr};
};

namespace {

bool valid_batch_options(const dp_batch_options* o) {
  if (!(o->threshold >= 0.0) || std::isinf(o->threshold)) return false;
  if (!dp::valid_precision(o->precision)) return false;
  for (int i = 0; i < DP_BATCH_BUCKETS; ++i)
    if (o->nb_bucket[i] < 1 || o->nb_bucket[i] > DP_BATCH_MAX_NB) return false;
  return true;
}

int launch(dp_batch* bp, double* d_base, int* d_ipiv, int* d_jpiv, int* d_info, cudaStream_t st) {
  return dp::batch::launch_raw(bp->classes, bp->sms, bp->d_n, bp->d_offsets, bp->d_rec,
                               bp->d_order, bp->d_queue, d_base, d_ipiv, d_jpiv, d_info, bp->opt,
                               st);
}

bool aligned8(const void* p) { return ((uintptr_t)p & 7) == 0; }

}  // namespace

namespace dp {
namespace batch {

// The batched launch on caller-managed device arrays (the server's small-
// request path, which allocates from the stream-ordered pool): d_n, d_off,
// d_rec, d_order describe `count` matrices as in a dp_batch plan, d_queue is
// kQueueBytes of 8-byte aligned scratch (the work counter, then the launch's
// near-tie counters), cleared here before the launch.
int launch_raw(const Classes& classes, int sms, const int* d_n, const long long* d_off,
               const long long* d_rec, const int* d_order, int* d_queue, double* base, int* ipiv,
               int* jpiv, int* info, const dp_batch_options& opt, cudaStream_t st) {
  if (!valid_batch_options(&opt)) return DP_INVALID_ARGUMENT;
  Params p;
  p.base = base;
  p.offsets = d_off;
  p.ns = d_n;
  p.rec_offsets = d_rec;
  p.ipiv = ipiv;
  p.jpiv = jpiv;
  p.info = info;
  p.ties = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(d_queue) + kTiesAt);
  p.threshold = opt.threshold;
  for (int i = 0; i < DP_BATCH_BUCKETS; ++i) p.nb_bucket[i] = opt.nb_bucket[i];
  if (cudaMemsetAsync(d_queue, 0, kQueueBytes, st) != cudaSuccess) return DP_CUDA_FAILURE;
  const int terms = dp::mixed_terms(opt.precision);
  int first = 0, launched = 0;
  for (int c = kClasses - 1; c >= 0; --c) {  // largest first, as the order is
    if (classes.count[c] <= 0) continue;
    p.order = d_order + first;
    p.count = classes.count[c];
    p.queue = d_queue + c;
    const int top = classes.max_n[c];
    const bool behind = launched > 0;
    const int rc = c == 3   ? launch_class<Geo3>(p, top, sms, terms, behind, st)
                   : c == 2 ? launch_class<Geo2>(p, top, sms, terms, behind, st)
                   : c == 1 ? launch_class<Geo1>(p, top, sms, terms, behind, st)
                            : launch_class<Geo0>(p, top, sms, terms, behind, st);
    if (rc != DP_SUCCESS) return rc;
    first += classes.count[c];
    ++launched;
  }
  return cudaGetLastError() == cudaSuccess ? DP_SUCCESS : DP_CUDA_FAILURE;
}

Classes classes_of(const int* ns, int count) {
  Classes k;
  for (int i = 0; i < count; ++i) {
    const int c = class_of(ns[i]);
    ++k.count[c];
    k.max_n[c] = std::max(k.max_n[c], ns[i]);
  }
  return k;
}

}  // namespace batch

void launch_fill_normal(double* x, long long len, unsigned long long seed, cudaStream_t st) {
  note_launch();
  batch::fill_normal_kernel<<<1184, 256, 0, st>>>(x, len, seed);
}

int panel_small_max_rows() { return batch::kMaxN; }
int panel_small_max_width() { return batch::kMaxNb; }

int launch_panel_small(const PanelParams& pp, cudaStream_t st) {
  const int rows = pp.m - pp.begin, w = pp.end - pp.begin;
  if (rows < 1 || rows > batch::kMaxN || w < 1 || w > batch::kMaxNb) return kInvalidArgument;
  const size_t smem = (size_t)batch::panel_ld(rows) * batch::kMaxNb * sizeof(double);
  // the fewest warps that hold the rows: a step's barrier and its merge of the
  // warps' candidates get shorter
  auto go = [&](auto geo) -> int {
    using G = decltype(geo);
    if (!ensure_smem((const void*)batch::panel_small_kernel<G>, smem)) return kCudaFailure;
    note_launch();
    launch_behind(batch::panel_small_kernel<G>, dim3(1), G::T, smem, st, pp);
    return kOk;
  };
  const int rc = rows <= 128   ? go(batch::PanelGeo<128>{})
                 : rows <= 256 ? go(batch::PanelGeo<256>{})
                               : go(batch::PanelGeo<512>{});
  if (rc != kOk) return rc;
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

}  // namespace dp

namespace {

const int kBucketLo[DP_BATCH_BUCKETS] = {1, 64, 128, 256};
const int kBucketHi[DP_BATCH_BUCKETS] = {63, 127, 255, 512};

}  // namespace

extern "C" {

void dp_batch_options_init(dp_batch_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->threshold = 0.0;
  o->precision = DP_PRECISION_FP64;
  for (int& nb : o->nb_bucket) nb = dp::batch::kWindow;
}

int dp_batch_create(dp_batch** out, int count, const int* n, const long long* offsets,
                    const dp_batch_options* opt) {
  if (!out) return DP_INVALID_ARGUMENT;
  *out = nullptr;
  if (count < 0 || (count > 0 && !n)) return DP_INVALID_ARGUMENT;
  dp_batch_options o;
  dp_batch_options_init(&o);
  if (opt) o = *opt;
  if (!valid_batch_options(&o)) return DP_INVALID_ARGUMENT;
  for (int i = 0; i < count; ++i)
    if (n[i] < 1 || n[i] > DP_BATCH_MAX_N || (offsets && offsets[i] < 0))
      return DP_INVALID_ARGUMENT;
  auto* bp = new (std::nothrow) dp_batch;
  if (!bp) return DP_ALLOCATION_FAILED;
  bp->opt = o;
  bp->count = count;
  bp->n.assign(n, n + count);
  bp->offsets.resize(count);
  bp->rec_offsets.resize(count);
  long long pos = 0, rec = 0;
  for (int i = 0; i < count; ++i) {
    if (offsets) {
      bp->offsets[i] = offsets[i];
      pos = std::max(pos, offsets[i] + (long long)n[i] * n[i]);
    } else {
      bp->offsets[i] = pos;
      pos += ((long long)n[i] * n[i] + 3) & ~3LL;  // each matrix starts 32-byte aligned
    }
    bp->rec_offsets[i] = rec;
    rec += n[i];
  }
  bp->classes = dp::batch::classes_of(n, count);
  bp->total_elements = pos;
  bp->total_records = rec;
  if (cudaGetDevice(&bp->device) != cudaSuccess ||
      cudaDeviceGetAttribute(&bp->sms, cudaDevAttrMultiProcessorCount, bp->device) !=
          cudaSuccess) {
    delete bp;
    return DP_CUDA_FAILURE;
  }
  std::vector<int> order(count);
  for (int i = 0; i < count; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return bp->n[a] > bp->n[b]; });
  const size_t c = (size_t)std::max(count, 1);
  if (cudaMalloc(&bp->d_n, c * sizeof(int)) != cudaSuccess ||
      cudaMalloc(&bp->d_offsets, c * sizeof(long long)) != cudaSuccess ||
      cudaMalloc(&bp->d_rec, c * sizeof(long long)) != cudaSuccess ||
      cudaMalloc(&bp->d_order, c * sizeof(int)) != cudaSuccess ||
      cudaMalloc(&bp->d_queue, dp::batch::kQueueBytes) != cudaSuccess) {
    dp_batch_destroy(bp);
    return DP_ALLOCATION_FAILED;
  }
  if (count > 0 &&
      (cudaMemcpy(bp->d_n, bp->n.data(), count * sizeof(int), cudaMemcpyHostToDevice) !=
           cudaSuccess ||
       cudaMemcpy(bp->d_offsets, bp->offsets.data(), count * sizeof(long long),
                  cudaMemcpyHostToDevice) != cudaSuccess ||
       cudaMemcpy(bp->d_rec, bp->rec_offsets.data(), count * sizeof(long long),
                  cudaMemcpyHostToDevice) != cudaSuccess ||
       cudaMemcpy(bp->d_order, order.data(), count * sizeof(int), cudaMemcpyHostToDevice) !=
           cudaSuccess)) {
    dp_batch_destroy(bp);
    return DP_CUDA_FAILURE;
  }
  *out = bp;
  return DP_SUCCESS;
}

int dp_batch_layout(const dp_batch* bp, long long* offsets, long long* record_offsets,
                    long long* total_elements, long long* total_records) {
  if (!bp) return DP_INVALID_ARGUMENT;
  if (offsets) std::copy(bp->offsets.begin(), bp->offsets.end(), offsets);
  if (record_offsets) std::copy(bp->rec_offsets.begin(), bp->rec_offsets.end(), record_offsets);
  if (total_elements) *total_elements = bp->total_elements;
  if (total_records) *total_records = bp->total_records;
  return DP_SUCCESS;
}

int dp_batch_set_options(dp_batch* bp, const dp_batch_options* opt) {
  if (!bp || !opt || !valid_batch_options(opt)) return DP_INVALID_ARGUMENT;
  bp->opt = *opt;
  if (bp->exec) {  // the captured launch carries the old options
    cudaGraphExecDestroy(bp->exec);
    bp->exec = nullptr;
  }
  return DP_SUCCESS;
}

int dp_batch_getrf_async(dp_batch* bp, double* d_base, int* d_ipiv, int* d_jpiv, int* d_info,
                         void* stream) {
  if (!bp) return DP_INVALID_ARGUMENT;
  if (bp->count == 0) return DP_SUCCESS;
  if (!d_base || !d_ipiv || !d_jpiv || !d_info || !aligned8(d_base)) return DP_INVALID_ARGUMENT;
  return launch(bp, d_base, d_ipiv, d_jpiv, d_info, (cudaStream_t)stream);
}

int dp_batch_getrf_graph(dp_batch* bp, double* d_base, int* d_ipiv, int* d_jpiv, int* d_info,
                         void* stream) {
  if (!bp) return DP_INVALID_ARGUMENT;
  if (bp->count == 0) return DP_SUCCESS;
  if (!d_base || !d_ipiv || !d_jpiv || !d_info || !aligned8(d_base)) return DP_INVALID_ARGUMENT;
  const void* args[4] = {d_base, d_ipiv, d_jpiv, d_info};
  if (bp->exec && !std::equal(args, args + 4, bp->g_args)) {
    cudaGraphExecDestroy(bp->exec);
    bp->exec = nullptr;
  }
  if (!bp->exec) {
    cudaStream_t cap;
    if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess)
      return DP_CUDA_FAILURE;
    cudaGraph_t graph = nullptr;
    int rc = DP_CUDA_FAILURE;
    if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      const int lrc = launch(bp, d_base, d_ipiv, d_jpiv, d_info, cap);
      const cudaError_t ce = cudaStreamEndCapture(cap, &graph);
      if (lrc == DP_SUCCESS && ce == cudaSuccess &&
          cudaGraphInstantiate(&bp->exec, graph, 0) == cudaSuccess)
        rc = DP_SUCCESS;
      else
        rc = lrc != DP_SUCCESS ? lrc : DP_CUDA_FAILURE;
      if (graph) cudaGraphDestroy(graph);
    }
    cudaStreamDestroy(cap);
    if (rc != DP_SUCCESS) {
      cudaGetLastError();
      bp->exec = nullptr;
      return rc;
    }
    std::copy(args, args + 4, bp->g_args);
  }
  for (int c : bp->classes.count)  // the graph's kernels (after the queue reset)
    if (c > 0) dp::note_launch();
  return cudaGraphLaunch(bp->exec, (cudaStream_t)stream) == cudaSuccess ? DP_SUCCESS
                                                                        : DP_CUDA_FAILURE;
}

int dp_batch_last_report(dp_batch* bp, dp_getrf_report* out) {
  if (!bp || !out) return DP_INVALID_ARGUMENT;
  unsigned long long t[3] = {0, 0, 0};
  if (bp->count > 0 &&
      (cudaDeviceSynchronize() != cudaSuccess ||
       cudaMemcpy(t, reinterpret_cast<char*>(bp->d_queue) + dp::batch::kTiesAt, sizeof(t),
                  cudaMemcpyDeviceToHost) != cudaSuccess))
    return DP_CUDA_FAILURE;
  std::memset(out, 0, sizeof(*out));
  out->decisions = (long long)t[0];
  out->near_ties = (long long)t[1];
  std::memcpy(&out->max_closeness, &t[2], sizeof(double));
  out->info = bp->count;
  return DP_SUCCESS;
}

void dp_batch_destroy(dp_batch* bp) {
  if (!bp) return;
  if (bp->exec) cudaGraphExecDestroy(bp->exec);
  cudaFree(bp->d_n);
  cudaFree(bp->d_offsets);
  cudaFree(bp->d_rec);
  cudaFree(bp->d_order);
  cudaFree(bp->d_queue);
  delete bp;
}

// Autotuner: per size bucket, time every candidate panel width on seeded
// N(0,1) matrices whose orders spread log-uniformly over the bucket and keep
// the fastest.
int dp_batch_autotune(dp_batch_options* opt, int samples, unsigned long long seed,
                      void* stream) {
  if (!opt || samples < 1 || samples > 65536) return DP_INVALID_ARGUMENT;
  dp_batch_options base = *opt;
  if (!valid_batch_options(&base)) return DP_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  static const int kCand[] = {8, dp::batch::kWindow};
  int rc = DP_SUCCESS;
  for (int bk = 0; bk < DP_BATCH_BUCKETS && rc == DP_SUCCESS; ++bk) {
    const int lo = std::max(kBucketLo[bk], 16), hi = kBucketHi[bk];
    std::vector<int> ns(samples);
    for (int i = 0; i < samples; ++i) {
      const double f = samples > 1 ? (double)i / (samples - 1) : 0.5;
      const double v = std::exp(std::log((double)lo) + f * (std::log((double)hi) - std::log((double)lo)));
      ns[i] = std::min(std::max((int)std::lround(v), lo), hi);
    }
    dp_batch* bp = nullptr;
    rc = dp_batch_create(&bp, samples, ns.data(), nullptr, &base);
    if (rc != DP_SUCCESS) break;
    double *d_src = nullptr, *d_work = nullptr;
    int *d_ipiv = nullptr, *d_jpiv = nullptr, *d_info = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    const size_t bytes = (size_t)bp->total_elements * sizeof(double);
    if (cudaMalloc(&d_src, bytes) != cudaSuccess || cudaMalloc(&d_work, bytes) != cudaSuccess ||
        cudaMalloc(&d_ipiv, bp->total_records * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&d_jpiv, bp->total_records * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&d_info, samples * sizeof(int)) != cudaSuccess ||
        cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
      rc = DP_ALLOCATION_FAILED;
    } else {
      dp::note_launch();
      dp::batch::fill_normal_kernel<<<1184, 256, 0, st>>>(d_src, bp->total_elements,
                                                          seed + 0x1000003ull * bk);
      float best_ms = 1e30f;
      int best_nb = base.nb_bucket[bk];
      for (int nb : kCand) {
        dp_batch_options o = base;
        for (int q = 0; q < DP_BATCH_BUCKETS; ++q) o.nb_bucket[q] = nb;
        dp_batch_set_options(bp, &o);
        float ms_min = 1e30f;
        for (int rep = 0; rep < 3 && rc == DP_SUCCESS; ++rep) {
          if (cudaMemcpyAsync(d_work, d_src, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
            rc = DP_CUDA_FAILURE;
            break;
          }
          cudaEventRecord(e0, st);
          rc = launch(bp, d_work, d_ipiv, d_jpiv, d_info, st);
          cudaEventRecord(e1, st);
          if (rc == DP_SUCCESS && cudaEventSynchronize(e1) != cudaSuccess) rc = DP_CUDA_FAILURE;
          float ms = 0.f;
          if (rc == DP_SUCCESS) cudaEventElapsedTime(&ms, e0, e1);
          ms_min = std::min(ms_min, ms);
        }
        if (rc != DP_SUCCESS) break;
        if (ms_min < best_ms) {
          best_ms = ms_min;
          best_nb = nb;
        }
      }
      if (rc == DP_SUCCESS) opt->nb_bucket[bk] = best_nb;
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(d_src);
    cudaFree(d_work);
    cudaFree(d_ipiv);
    cudaFree(d_jpiv);
    cudaFree(d_info);
    dp_batch_destroy(bp);
  }
  return rc;
}

// Table file: one line per bucket, "<smallest n> <largest n> <nb>".
int dp_batch_tune_save(const char* path, const dp_batch_options* opt) {
  if (!path || !opt || !valid_batch_options(opt)) return DP_INVALID_ARGUMENT;
  FILE* f = std::fopen(path, "w");
  if (!f) return DP_INVALID_ARGUMENT;
  for (int i = 0; i < DP_BATCH_BUCKETS; ++i)
    std::fprintf(f, "%d %d %d\n", kBucketLo[i], kBucketHi[i], opt->nb_bucket[i]);
  return std::fclose(f) == 0 ? DP_SUCCESS : DP_INVALID_ARGUMENT;
}

int dp_batch_tune_load(const char* path, dp_batch_options* opt) {
  if (!path || !opt) return DP_INVALID_ARGUMENT;
  FILE* f = std::fopen(path, "r");
  if (!f) return DP_INVALID_ARGUMENT;
  dp_batch_options o = *opt;
  int rc = DP_SUCCESS;
  for (int i = 0; i < DP_BATCH_BUCKETS; ++i) {
    int lo, hi, nb;
    if (std::fscanf(f, "%d %d %d", &lo, &hi, &nb) != 3 || lo != kBucketLo[i] ||
        hi != kBucketHi[i] || nb < 1 || nb > DP_BATCH_MAX_NB) {
      rc = DP_INVALID_ARGUMENT;
      break;
    }
    o.nb_bucket[i] = nb;
  }
  std::fclose(f);
  if (rc == DP_SUCCESS) *opt = o;
  return rc;
}

}  // extern "C"
