// B <- L^{-1} B with a unit lower diagonal block of at most 64 rows: the panel's
// block row, U12 = L11^{-1} A12 (delayed_lu/delayed_dgetrf.cpp:72-74), and the first
// half of materialize_partial_panel (:111-114).  Wider blocks are split by the host
// into 64-wide solves and GEMM updates, or solved by the block's inverse.
//
// A CTA owns 64 columns of B; two threads own each column, one per 32-row
// half, holding their half in 32 registers with the substitution fully
// unrolled.  The triangle sits in shared memory (every load of it is a
// broadcast); the tile is staged through shared memory so the global loads
// and stores stay coalesced.  Rows / columns beyond w are an identity block,
// so narrower blocks run the same code.
#include "dp_device.cuh"
#include "dp_kernels.h"

namespace dp {

namespace {

constexpr int kTrsmW = 64;     // maximum block width
constexpr int kHalf = 32;
constexpr int kTrsmCols = 64;  // columns per CTA
constexpr int kTrsmThreads = 2 * kTrsmCols;
constexpr int kStage = kTrsmW + 1;  // odd stride: conflict-free per-thread column access
constexpr size_t kTrsmSmem =
    (size_t)(kTrsmW * kTrsmW + kTrsmCols * kStage) * sizeof(double);

__device__ __forceinline__ void stage_in(const double* B, long long ldb, int w, int ncols,
                                         double* Bt) {
  for (int e = threadIdx.x; e < w * ncols; e += kTrsmThreads) {
    const int i = e % w, c = e / w;
    Bt[c * kStage + i] = B[idx(i, c, ldb)];
  }
}

__device__ __forceinline__ void stage_out(double* B, long long ldb, int w, int ncols,
                                          const double* Bt) {
  for (int e = threadIdx.x; e < w * ncols; e += kTrsmThreads) {
    const int i = e % w, cc = e / w;
    B[idx(i, cc, ldb)] = Bt[cc * kStage + i];
  }
}

// B (w x nc) <- L^{-1} B, L unit lower (w x w).
__global__ void __launch_bounds__(kTrsmThreads)
trsm_lower_unit_kernel(const double* __restrict__ L, long long ldl, double* B, long long ldb, int w,
                       int nc, const int* gate) {
  after_previous_kernel();
  if (gate && *gate >= 0) return;
  extern __shared__ __align__(16) double tsm[];
  double* Ls = tsm;                    // Ls[p * 64 + i] = L(i, p), zero outside the strict lower part
  double* Bt = tsm + kTrsmW * kTrsmW;  // Bt[c * 65 + i] = B(i, c)
  const int tid = threadIdx.x;
  const int col0 = blockIdx.x * kTrsmCols;
  const int ncols = min(kTrsmCols, nc - col0);
  B += idx(0, col0, ldb);

  for (int e = tid; e < kTrsmW * kTrsmW; e += kTrsmThreads) {
    const int i = e % kTrsmW, pcol = e / kTrsmW;
    Ls[e] = (i > pcol && i < w) ? L[idx(i, pcol, ldl)] : 0.0;
  }
  stage_in(B, ldb, w, ncols, Bt);
  __syncthreads();

  const int c = tid % kTrsmCols;
  const bool upper_half = tid < kTrsmCols;  // warps 0-1: rows 0..31, warps 2-3: rows 32..63
  double* bc = Bt + c * kStage;
  if (upper_half && c < ncols) {
    double x[kHalf];
#pragma unroll
    for (int i = 0; i < kHalf; ++i) x[i] = i < w ? bc[i] : 0.0;
#pragma unroll
    for (int p = 0; p < kHalf - 1; ++p) {
#pragma unroll
      for (int i = p + 1; i < kHalf; ++i) x[i] -= Ls[p * kTrsmW + i] * x[p];
    }
#pragma unroll
    for (int i = 0; i < kHalf; ++i)
      if (i < w) bc[i] = x[i];
  }
  __syncthreads();
  if (!upper_half && c < ncols && w > kHalf) {
    double x[kHalf];
#pragma unroll
    for (int i = 0; i < kHalf; ++i) x[i] = kHalf + i < w ? bc[kHalf + i] : 0.0;
#pragma unroll 4
    for (int p = 0; p < kHalf; ++p) {
      const double xp = bc[p];
#pragma unroll
      for (int i = 0; i < kHalf; ++i) x[i] -= Ls[p * kTrsmW + kHalf + i] * xp;
    }
#pragma unroll
    for (int p = 0; p < kHalf - 1; ++p) {
#pragma unroll
      for (int i = p + 1; i < kHalf; ++i) x[i] -= Ls[(kHalf + p) * kTrsmW + kHalf + i] * x[p];
    }
#pragma unroll
    for (int i = 0; i < kHalf; ++i)
      if (kHalf + i < w) bc[kHalf + i] = x[i];
  }
  __syncthreads();
  stage_out(B, ldb, w, ncols, Bt);
}

void configure() {
  ensure_smem((const void*)trsm_lower_unit_kernel, kTrsmSmem);
}

}  // namespace

// T <- I - L^{-1} for a unit lower w x w block L (w <= 256), so that the
// block solve X = L^{-1} B becomes the FP64 tensor-core update
// X = B - T B (T strictly lower).  Columns of L^{-1} are forward substitutions
// L x = e_j, four to a CTA: warp r holds rows 32 r + lane of them.  Warp c
// takes the steps of its own 32 x 32 diagonal block by shuffles, leaves its
// entries in shared memory, and the warps below apply the 32 steps at once
// from rows of L that they loaded while they waited.  The kernel stands
// between two outer blocks, so its latency counts: 20.6 us at w = 256 (12.4 at
// 128), against 36 with a warp per column and L staged through shared memory.
// What bounds it is the chain of 256 shuffles and FMAs (some 60 cycles a step,
// 6 us) and eight barriers with 32 steps' FMAs and loads behind each.
constexpr int kInvMaxW = 256;
constexpr int kInvCols = 4;  // columns per CTA
static_assert(32 % kInvCols == 0, "a group of steps holds the diagonal");

__global__ void __launch_bounds__(kInvMaxW)
lower_inverse_kernel(const double* __restrict__ L, long long ldl, int w, double* __restrict__ T,
                     long long ldt) {
  __shared__ __align__(16) double xs[2][32][kInvCols];  // the entries of a block, by its parity
  extern __shared__ double ds[];  // [warp][32][32]: a warp's diagonal block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  after_previous_kernel();
  const int i = threadIdx.x;  // the row
  const int j = blockIdx.x * kInvCols;
  const int c0 = j / 32, jj = j % 32;
  const double* Li = L + i;
  double x[kInvCols];
#pragma unroll
  for (int u = 0; u < kInvCols; ++u) x[u] = i == j + u ? 1.0 : 0.0;
  if (warp >= c0) {
#pragma unroll 8
    for (int kk = 0; kk < 32; ++kk)  // strictly lower, zeros elsewhere
      ds[(32 * warp + kk) * 32 + lane] = lane > kk && i < w ? Li[(size_t)(32 * warp + kk) * (size_t)ldl]
                                                             : 0.0;
    __syncwarp();
  }
  for (int c = c0; 32 * c < w; ++c) {  // (CTA-uniform)
    const int lo = c == c0 ? jj : 0;   // the block's first step
    double l[32];
    if (warp > c) {
#pragma unroll
      for (int kk = 0; kk < 32; ++kk)
        l[kk] = i < w ? Li[(size_t)(32 * c + kk) * (size_t)ldl] : 0.0;
    } else if (warp == c) {
      const int hi = min(32, w - 1 - 32 * c);
      const int first = c == c0 ? jj : -kInvCols;
#pragma unroll 4
      for (int kk = lo; kk < hi; ++kk) {
        const double d = ds[(32 * c + kk) * 32 + lane];
#pragma unroll
        for (int u = 0; u < kInvCols; ++u) {
          // Before column u's diagonal x_k is zero; d too, lest an infinity reach the column
          // (selected: a branch around the shuffle makes the step seven times as long).
          const double du = kk >= first + u ? d : 0.0;
          x[u] = fma(-du, __shfl_sync(0xffffffffu, x[u], kk), x[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < kInvCols; ++u) xs[c & 1][lane][u] = x[u];
    }
    __syncthreads();  // (this parity is written again after the next one)
    if (warp > c) {
#pragma unroll
      for (int g = 0; g < 32; g += kInvCols) {
        if (g < lo) continue;  // (uniform)
        const bool past = c != c0 || g > lo;
#pragma unroll
        for (int t = 0; t < kInvCols; ++t) {
          const double before = past ? l[g + t] : 0.0;  // (columns whose diagonal is still to come)
#pragma unroll
          for (int u = 0; u < kInvCols; u += 2) {
            const double2 xk = *(const double2*)&xs[c & 1][g + t][u];
            x[u] = fma(-(u <= t ? l[g + t] : before), xk.x, x[u]);
            x[u + 1] = fma(-(u + 1 <= t ? l[g + t] : before), xk.y, x[u + 1]);
          }
        }
      }
    }
  }
  if (i >= w) return;
#pragma unroll
  for (int u = 0; u < kInvCols; ++u)
    if (j + u < w) T[i + (size_t)(j + u) * (size_t)ldt] = i > j + u ? -x[u] : 0.0;
}

// dst(0:rows, 0:cols) <- src(0:rows, 0:cols), both column-major: a CTA per
// column at a time, consecutive threads on consecutive rows.
__global__ void __launch_bounds__(256)
copy_block_kernel(const double* __restrict__ src, long long lds, double* __restrict__ dst,
                  long long ldd, int rows, int cols) {
  after_previous_kernel();
  for (long long c = blockIdx.x; c < cols; c += gridDim.x) {
    const double* s = src + c * lds;
    double* d = dst + c * ldd;
    for (int r = threadIdx.x; r < rows; r += blockDim.x) d[r] = s[r];
  }
}

int trsm_max_width() { return kTrsmW; }

void launch_copy_block(const double* src, long long lds, double* dst, long long ldd, int rows,
                       int cols, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return;
  dp::note_launch();
  launch_behind(copy_block_kernel, dim3(std::min(cols, 148 * 8)), 256, 0, s, src, lds, dst, ldd, rows,
                cols);
}

int lower_inverse_max_width() { return kInvMaxW; }

void launch_lower_inverse(const double* L, long long ldl, int w, double* T, long long ldt,
                          cudaStream_t s) {
  if (w <= 0) return;
  constexpr size_t kSmem = (size_t)kInvMaxW * 32 * sizeof(double);
  dp::ensure_smem((const void*)lower_inverse_kernel, kSmem);
  dp::note_launch();
  launch_behind(lower_inverse_kernel, dim3((w + kInvCols - 1) / kInvCols), (w + 31) / 32 * 32,
                kSmem, s, L, ldl, w, T, ldt);
}

void launch_trsm_lower_unit(const double* L, long long ldl, double* B, long long ldb, int w, int nc,
                            cudaStream_t s, const int* gate) {
  if (w <= 1 || nc <= 0) return;  // w == 1: unit diagonal, nothing to solve
  configure();
  const int grid = (nc + kTrsmCols - 1) / kTrsmCols;
  dp::note_launch();
  launch_behind(trsm_lower_unit_kernel, dim3(grid), kTrsmThreads, kTrsmSmem, s, L, ldl, B, ldb, w,
                nc, gate);
}

void launch_trsm_unit_lower(double* a, long long lda, int r0, int w, int c0, int nc,
                            cudaStream_t s, const int* gate) {
  launch_trsm_lower_unit(a + idx(r0, r0, lda), lda, a + idx(r0, c0, lda), lda, w, nc, s, gate);
}

}  // namespace dp
