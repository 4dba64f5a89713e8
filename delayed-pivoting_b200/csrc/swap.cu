// Row and column permutation kernels of the delayed-pivoting LU.
//
// The reference swaps a full row (n elements, stride lda) and, on a fallback,
// a full column (m elements) at every step (delayed_lu/delayed_dgetrf.cpp:202-209,
// delayed_lu_cuda/delayed_dgetrf_cuda.cu:304-317).  Here the panel kernel
// swaps rows only inside the panel columns and writes the composite
// permutation of the whole panel as a list of (destination, source) rows;
// laswp_kernel then moves, per column outside the panel, only the rows that
// changed, once per panel: each warp owns one column, gathers every source
// row into registers and scatters them to their destinations.  The block
// part of the list (destinations begin..end-1) is contiguous, so those writes
// are coalesced.  The full-row and full-column swap of a fallback step are one
// kernel that takes the pivot from the device's search result.
#include "dp_device.cuh"
#include "dp_kernels.h"

namespace dp {

namespace {

constexpr int kLaswpThreads = 256;
constexpr int kMaxSwapEntries = 512;  // 2 * maximum panel width
constexpr int kPerLane = kMaxSwapEntries / 32;
constexpr int kSolveW = 64;           // widest panel whose block rows laswp_kernel solves

// Also, for the columns [s0, s1) (a subset of [c2, c3)) and a panel of at most
// kSolveW columns that did not stop (state->stop_k < 0): U12 = L11^{-1} of the
// panel's block rows right after they are permuted, L11 the panel's unit
// lower triangle (the in-block TRSM, delayed_lu/delayed_dgetrf.cpp:72-74,
// fused: one warp per column, rows begin + lane and begin + 32 + lane, the
// entries of step k passed by shuffle, the same order of operations per row
// as the TRSM kernel).
__global__ void __launch_bounds__(kLaswpThreads)
laswp_kernel(double* a, long long lda, int begin, int nblock, const int* swap_block,
             const int* swap_extra, const State* state, int c0, int c1, int c2, int c3,
             int gate_begin, int s0, int s1) {
  __shared__ int s_dst[kMaxSwapEntries];
  __shared__ int s_src[kMaxSwapEntries];
  __shared__ int s_count;
  __shared__ double s_l[kSolveW * kSolveW];  // s_l[k * kSolveW + i] = L11(i, k), i > k
  after_previous_kernel();
  const int sk = state->stop_k;
  // an earlier panel stopped, or the fallback search before this one found nothing
  if (gate_begin >= 0 && sk >= 0 && (sk < gate_begin || state->delayed)) return;
  const bool solve = s0 < s1 && sk < 0 && nblock <= kSolveW;
  const int tid = threadIdx.x;
  if (solve) {
    for (int e = tid; e < kSolveW * kSolveW; e += blockDim.x) {
      const int k = e / kSolveW, i = e - k * kSolveW;
      s_l[e] = (i > k && i < nblock) ? a[idx(begin + i, begin + k, lda)] : 0.0;
    }
  }
  const int nextra = min(state->swap_count, kMaxSwapEntries - nblock);
  if (tid == 0) s_count = 0;
  __syncthreads();
  // keep only rows whose content changed (warp-aggregated compaction)
  for (int base = 0; base < nblock + nextra; base += blockDim.x) {
    const int i = base + tid;
    int d = 0, sr = 0;
    bool keep = false;
    if (i < nblock) {
      d = begin + i;
      sr = swap_block[i];
      keep = sr != d;
    } else if (i < nblock + nextra) {
      d = swap_extra[2 * (i - nblock)];
      sr = swap_extra[2 * (i - nblock) + 1];
      keep = sr != d;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    int wbase = 0;
    if ((tid & 31) == 0 && mask) wbase = atomicAdd(&s_count, __popc(mask));
    wbase = __shfl_sync(0xffffffffu, wbase, 0);
    if (keep) {
      const int pos = wbase + __popc(mask & ((1u << (tid & 31)) - 1u));
      s_dst[pos] = d;
      s_src[pos] = sr;
    }
    __syncthreads();
  }
  __syncthreads();
  const int total = s_count;
  if (total == 0 && !solve) return;

  const int lane = tid & 31;
  const int warps = blockDim.x >> 5;
  const long long n1 = c1 - c0, ncols = n1 + (c3 - c2);
  for (long long cid = (long long)blockIdx.x * warps + (tid >> 5); cid < ncols;
       cid += (long long)gridDim.x * warps) {
    const long long col = cid < n1 ? c0 + cid : c2 + (cid - n1);
    double* ac = a + idx(0, col, lda);
    double v[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int i = lane + 32 * j;
      if (i < total) v[j] = ac[s_src[i]];
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int i = lane + 32 * j;
      if (i < total) ac[s_dst[i]] = v[j];
    }
    __syncwarp();
    if (solve && col >= s0 && col < s1) {  // (warp-uniform)
      double* bc = ac + begin;
      double x0 = lane < nblock ? bc[lane] : 0.0;
      double x1 = 32 + lane < nblock ? bc[32 + lane] : 0.0;
      for (int k = 0; k < nblock - 1; ++k) {
        const double xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31);
        // only rows below k (an infinite or NaN x_k must not reach the others)
        if (lane > k) x0 = fma(-s_l[k * kSolveW + lane], xk, x0);
        if (32 + lane > k) x1 = fma(-s_l[k * kSolveW + 32 + lane], xk, x1);
      }
      if (lane < nblock) bc[lane] = x0;
      if (32 + lane < nblock) bc[32 + lane] = x1;
      __syncwarp();
    }
  }
}

// The swap lists of consecutive panels applied in panel order: list p covers
// the panel starting at row begin_p = q.base + width[0] + ... + width[p-1],
// its block part at blk[begin_p - q.base] and up to width[p] extra pairs at
// ext[2 (begin_p - q.base)] (unused pairs have a negative destination: the
// region is filled with -1 before the panel runs, and the panel writes its
// pairs from the front).  Each CTA compacts every list into shared memory
// (list p at [s_lb[p], s_lb[p+1])); each warp then applies the lists to one
// column in turn, gathering a list's sources before scattering it, so the
// result equals launching laswp_kernel once per panel.
__global__ void __launch_bounds__(kLaswpThreads)
laswp_seq_kernel(double* a, long long lda, const int* blk, const int* ext, SwapSeq q, int c0,
                 int c1, int c2, int c3) {
  __shared__ int s_dst[kSwapSeqEntries];
  __shared__ int s_src[kSwapSeqEntries];
  __shared__ int s_lb[kSwapSeqLists + 1];
  __shared__ int s_count;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_count = 0;
    s_lb[0] = 0;
  }
  __syncthreads();
  int off = 0;
  for (int p = 0; p < q.lists; ++p) {
    const int nblock = q.width[p], nextra = q.width[p];
    for (int base = 0; base < nblock + nextra; base += blockDim.x) {
      const int i = base + tid;
      int d = 0, sr = 0;
      bool keep = false;
      if (i < nblock) {
        d = q.base + off + i;
        sr = blk[off + i];
        keep = sr != d;
      } else if (i < nblock + nextra) {
        d = ext[2 * off + 2 * (i - nblock)];
        sr = ext[2 * off + 2 * (i - nblock) + 1];
        keep = d >= 0 && sr != d;
      }
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      int wbase = 0;
      if ((tid & 31) == 0 && mask) wbase = atomicAdd(&s_count, __popc(mask));
      wbase = __shfl_sync(0xffffffffu, wbase, 0);
      if (keep) {
        const int pos = wbase + __popc(mask & ((1u << (tid & 31)) - 1u));
        s_dst[pos] = d;
        s_src[pos] = sr;
      }
      __syncthreads();
    }
    // the list's last append is behind the barrier above; no thread appends
    // to the next list before the boundary is read
    if (tid == 0) s_lb[p + 1] = s_count;
    __syncthreads();
    off += nblock;
  }
  if (s_count == 0) return;

  const int lane = tid & 31;
  const int warps = blockDim.x >> 5;
  const long long n1 = c1 - c0, ncols = n1 + (c3 - c2);
  for (long long cid = (long long)blockIdx.x * warps + (tid >> 5); cid < ncols;
       cid += (long long)gridDim.x * warps) {
    const long long col = cid < n1 ? c0 + cid : c2 + (cid - n1);
    double* ac = a + idx(0, col, lda);
    for (int p = 0; p < q.lists; ++p) {
      const int lo = s_lb[p], cnt = s_lb[p + 1] - lo;
      if (cnt == 0) continue;
      double v[kPerLane];
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const int i = lane + 32 * j;
        if (i < cnt) v[j] = ac[s_src[lo + i]];
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const int i = lane + 32 * j;
        if (i < cnt) ac[s_dst[lo + i]] = v[j];
      }
      __syncwarp();
    }
  }
}

// The end of a fallback search at step k: with no magnitude above the
// threshold the factorisation is over (state->delayed, stop_k stays); else the
// pivot (r, c) of state->fallback moves to (k, k) - rows k <-> r over all
// columns, then columns k <-> c over all rows, in one pass (the four elements
// both swaps touch go to one thread) - the swap is recorded and the stop word
// re-armed, so that the kernels enqueued behind this one run.
__global__ void apply_fallback_kernel(double* a, long long lda, int m, int n, int k,
                                      double threshold, State* state, int* ipiv, int* jpiv,
                                      int* done) {
  const Cand f = state->fallback;
  const bool found = f.val > threshold;
  const int r = f.row, c = f.col;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (found) {
    if (r != k)
      for (int j = t0; j < n; j += step)
        if (j != k && j != c) {
          double *x = a + idx(k, j, lda), *y = a + idx(r, j, lda);
          const double t = *x;
          *x = *y;
          *y = t;
        }
    if (c != k)
      for (int i = t0; i < m; i += step)
        if (i != k && i != r) {
          double *x = a + idx(i, k, lda), *y = a + idx(i, c, lda);
          const double t = *x;
          *x = *y;
          *y = t;
        }
    if (t0 == 0) {  // (r == k or c == k: the same elements under two names)
      const double kk = a[idx(k, k, lda)], kc = a[idx(k, c, lda)];
      const double rk = a[idx(r, k, lda)], rc = a[idx(r, c, lda)];
      a[idx(k, k, lda)] = rc;
      a[idx(k, c, lda)] = rk;
      a[idx(r, k, lda)] = kc;
      a[idx(r, c, lda)] = kk;
      ipiv[k] = r;
      jpiv[k] = c;
    }
  }
  // the last CTA, once every CTA has read the search's result
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (last && threadIdx.x == 0) {
    *done = 0;
    if (found)
      state->stop_k = -1;
    else
      state->delayed = 1;
  }
}

__global__ void identity_records_kernel(int* ipiv, int* jpiv, int count) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    ipiv[i] = i;
    jpiv[i] = i;
  }
}

int grid_for(long long work, int threads, int cap) {
  long long g = (work + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

}  // namespace

void launch_laswp(double* a, long long lda, int begin, int nblock, const int* swap_block,
                  const int* swap_extra, const State* state, int c0, int c1, int c2, int c3,
                  cudaStream_t s, int gate_begin, int s0, int s1) {
  const long long ncols = (long long)(c1 - c0) + (c3 - c2);
  if (ncols <= 0 || nblock <= 0) return;
  const int warps = kLaswpThreads / 32;
  const int grid = grid_for(ncols, warps, 148 * 16);
  dp::note_launch();
  launch_behind(laswp_kernel, dim3(grid), kLaswpThreads, 0, s, a, lda, begin, nblock, swap_block,
                swap_extra, state, c0, c1, c2, c3, gate_begin, s0, s1);
}

int laswp_solve_max_width() { return kSolveW; }

int launch_laswp_seq(double* a, long long lda, const int* blk, const int* ext, int base,
                     const int* widths, int lists, int c0, int c1, int c2, int c3,
                     cudaStream_t s) {
  const long long ncols = (long long)(c1 - c0) + (c3 - c2);
  if (ncols <= 0 || lists <= 0) return 0;
  for (int i = 0; i < lists; ++i)  // a panel list: at most kMaxSwapEntries changed rows
    if (widths[i] < 1 || 2 * widths[i] > kMaxSwapEntries) return -1;
  const int warps = kLaswpThreads / 32;
  const int grid = grid_for(ncols, warps, 148 * 16);
  int launches = 0, p = 0, off = 0;
  while (p < lists) {
    // as many whole lists as fit the kernel's list and entry capacity
    SwapSeq q;
    q.base = base + off;
    q.lists = 0;
    int entries = 0, width = 0;
    while (p < lists && q.lists < kSwapSeqLists && entries + 2 * widths[p] <= kSwapSeqEntries) {
      q.width[q.lists] = widths[p];
      entries += 2 * widths[p];
      width += widths[p];
      ++q.lists;
      ++p;
    }
    if (q.lists == 0) return -1;  // one list beyond the capacity: not a panel's list
    dp::note_launch();
    laswp_seq_kernel<<<grid, kLaswpThreads, 0, s>>>(a, lda, blk + off, ext + 2 * off, q, c0, c1,
                                                    c2, c3);
    ++launches;
    off += width;
  }
  return launches;
}

void launch_apply_fallback(double* a, long long lda, int m, int n, int k, double threshold,
                           State* state, int* ipiv, int* jpiv, cudaStream_t s) {
  dp::note_launch();
  apply_fallback_kernel<<<grid_for(m > n ? m : n, 256, 148), 256, 0, s>>>(
      a, lda, m, n, k, threshold, state, ipiv, jpiv, &state->fallback_done);
}

void launch_identity_records(int* ipiv, int* jpiv, int count, cudaStream_t s) {
  if (count <= 0) return;
  dp::note_launch();
  identity_records_kernel<<<grid_for(count, 256, 148 * 4), 256, 0, s>>>(ipiv, jpiv, count);
}

}  // namespace dp
