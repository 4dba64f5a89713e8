// Kernels of the small-request path of the server: solves, residuals and
// backward errors for many small factorisations at once (one CTA per item),
// on factors made by the batched factorisation (batched.cu).
//
// A factorisation P*A*Q = L*U with swap histories ipiv / jpiv (replayed in
// order, delayed_lu_cuda/example.cu:61-68) solves A x = b as
//   y = L^{-1} (P b),  y = U^{-1} y,  x = Q y,
// with (P b)[k] = b[row[k]] and x[col[k]] = y[k], row / col the histories
// replayed on the identity.
#include <algorithm>

#include "dp_device.cuh"
#include "serve_kernels.h"

namespace dp {
namespace serve {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kBlk = 32;       // diagonal block of the triangular sweeps
constexpr int kCols = kWarps;  // right-hand sides of a solving CTA: one per warp
constexpr int kRowTile = 64;   // rows of a residual CTA
constexpr int kGroups = kThreads / kRowTile;
constexpr int kPass = 8 * kGroups;  // its right-hand sides per pass over A

__host__ __device__ __forceinline__ int ld_of(int n) { return n + 1; }

// Largest of a warp's non-negative values (lane 0).
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace

// Composite row / column orders of each matrix's swap histories: one warp per
// matrix, lane 0 replaying in shared memory, the warp writing out.
__global__ void orders_kernel(const int* __restrict__ ns, const long long* __restrict__ rec,
                              const int* __restrict__ ipiv, const int* __restrict__ jpiv,
                              int* row_order, int* col_order, int count) {
  __shared__ int r[kMaxSmallN], c[kMaxSmallN];
  const int i = blockIdx.x;
  if (i >= count) return;
  const int n = ns[i];
  const long long o = rec[i];
  for (int k = threadIdx.x; k < n; k += 32) r[k] = c[k] = k;
  __syncwarp();
  if (threadIdx.x == 0)
    for (int k = 0; k < n; ++k) {
      const int p = ipiv[o + k], q = jpiv[o + k];
      const int t = r[k];
      r[k] = r[p];
      r[p] = t;
      const int u = c[k];
      c[k] = c[q];
      c[q] = u;
    }
  __syncwarp();
  for (int k = threadIdx.x; k < n; k += 32) {
    row_order[o + k] = r[k];
    col_order[o + k] = c[k];
  }
}

// X = A^{-1} B for each item: a CTA takes kCols of its right-hand sides, the
// columns in shared memory, and steps through the diagonal blocks of 32.  A
// warp solves a block for one column by shuffles, then a thread per row applies
// the block's 32 steps to all columns.  Every load of a step - the next
// diagonal block, 32 entries of a row - is issued before the block's solve and
// arrives behind it: waiting for each in turn, one CTA to an item, the
// sweeps of a burst of requests up to order 512 took 2.0 ms, now 0.24.
// What bounds it is the chain of each column's steps.  The sums keep their order.
__global__ void __launch_bounds__(kThreads) solve_kernel(const SolveItem* __restrict__ items) {
  extern __shared__ double Y[];  // [kCols][n + 1]
  __shared__ double Ds[kBlk * kBlk];                    // the diagonal block, column by column
  __shared__ __align__(16) double Xs[kBlk][kCols];      // its solution, zero outside
  const SolveItem it = items[blockIdx.x];
  const int c0 = blockIdx.y * kCols;
  if (c0 >= it.nrhs) return;
  const int n = it.n, ldy = ld_of(n), nc = min(kCols, it.nrhs - c0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* __restrict__ LU = it.lu;
  for (int c = 0; c < kCols; ++c)
    for (int i = tid; i < n; i += kThreads)
      Y[c * ldy + i] = c < nc ? it.B[idx(it.row[i], c0 + c, it.ldb)] : 0.0;
  double d[kBlk * kBlk / kThreads];
  auto fetch = [&](int kb) {  // the block at kb; a unit diagonal and zeros outside the matrix
#pragma unroll
    for (int q = 0; q < kBlk * kBlk / kThreads; ++q) {
      const int i = kb + lane, k = kb + warp + kWarps * q;
      d[q] = i < n && k < n ? LU[idx(i, k, n)] : (i == k ? 1.0 : 0.0);
    }
  };
  auto place = [&] {
#pragma unroll
    for (int q = 0; q < kBlk * kBlk / kThreads; ++q) Ds[(warp + kWarps * q) * kBlk + lane] = d[q];
  };
  double l[kBlk];
  auto fetch_row = [&](int i, int kb) {
#pragma unroll
    for (int k = 0; k < kBlk; ++k) l[k] = kb + k < n ? LU[(unsigned)(i + (kb + k) * n)] : 0.0;
  };
  auto apply = [&](int i) {
    double acc[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) acc[c] = Y[c * ldy + i];
#pragma unroll
    for (int k = 0; k < kBlk; ++k)
#pragma unroll
      for (int c = 0; c < kCols; c += 2) {
        const double2 x = *(const double2*)&Xs[k][c];
        acc[c] = fma(-l[k], x.x, acc[c]);
        acc[c + 1] = fma(-l[k], x.y, acc[c + 1]);
      }
#pragma unroll
    for (int c = 0; c < kCols; ++c) Y[c * ldy + i] = acc[c];
  };
  // forward: unit lower L
  fetch(0);
  for (int kb = 0; kb < n; kb += kBlk) {
    place();
    __syncthreads();
    const int first = kb + kBlk + tid;
    if (first < n) fetch_row(first, kb);
    if (kb + kBlk < n) fetch(kb + kBlk);
    double y = kb + lane < n ? Y[warp * ldy + kb + lane] : 0.0;
#pragma unroll 8
    for (int k = 0; k < kBlk - 1; ++k) {
      const double t = fma(-Ds[k * kBlk + lane], __shfl_sync(0xffffffffu, y, k), y);
      y = lane > k ? t : y;
    }
    if (kb + lane < n) Y[warp * ldy + kb + lane] = y;
    Xs[lane][warp] = y;
    __syncthreads();
#pragma unroll 1
    for (int i = first; i < n; i += kThreads) {
      if (i != first) fetch_row(i, kb);
      apply(i);
    }
    __syncthreads();
  }
  // backward: upper U with its diagonal
  const int last = (n - 1) / kBlk * kBlk;
  fetch(last);
  for (int kb = last; kb >= 0; kb -= kBlk) {
    place();
    __syncthreads();
    if (tid < kb) fetch_row(tid, kb);
    if (kb > 0) fetch(kb - kBlk);
    double y = kb + lane < n ? Y[warp * ldy + kb + lane] : 0.0;
    const double pivot = Ds[lane * kBlk + lane];
#pragma unroll 4
    for (int k = kBlk - 1; k >= 0; --k) {
      const double x = y / pivot;  // (lane k's is the entry)
      const double t = fma(-Ds[k * kBlk + lane], __shfl_sync(0xffffffffu, x, k), y);
      y = lane == k ? x : (lane < k ? t : y);
    }
    if (kb + lane < n) Y[warp * ldy + kb + lane] = y;
    Xs[lane][warp] = y;
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < kb; i += kThreads) {
      if (i != tid) fetch_row(i, kb);
      apply(i);
    }
    __syncthreads();
  }
  for (int c = 0; c < nc; ++c)
    for (int i = tid; i < n; i += kThreads) it.X[idx(it.col[i], c0 + c, it.ldx)] = Y[c * ldy + i];
}

__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  // non-negative doubles order like their bit patterns
  atomicMax(reinterpret_cast<unsigned long long*>(addr),
            (unsigned long long)__double_as_longlong(v));
}

// |v|, a NaN as +inf.
__device__ __forceinline__ double magnitude(double v) {
  const double a = fabs(v);
  return a == a ? a : INFINITY;
}

// R = B - A X and the normwise backward error
//   max_c ||R_c||_inf / (||A||_inf ||X_c||_inf + ||B_c||_inf)
// into err[item] (NaN reported as +inf).  A CTA per 64 rows of an item, a
// thread per row and eight right-hand sides, entries of A loaded eight ahead
// and X staged 64 rows at a time: 0.48 ms for that burst became 0.07 (one
// CTA per item waited for each entry of its row in turn).  The norms meet in `work`
// (kResidualWork doubles per item, zero before the launch and after it); the
// item's last CTA turns them into the error.
__global__ void __launch_bounds__(kThreads) residual_kernel(const ResidualItem* __restrict__ items,
                                                            double* work, double* err) {
  __shared__ __align__(16) double Xs[kRowTile][kPass + 2];
  __shared__ double norms[3 * kMaxRhs + 1];  // |R|, |X|, |B| per column, ||A||
  __shared__ int is_last;
  const ResidualItem it = items[blockIdx.x];
  const int n = it.n, r0 = blockIdx.y * kRowTile;
  if (r0 >= n) return;
  const int tid = threadIdx.x, lane = tid & 31;
  const int group = tid / kRowTile, i = r0 + tid % kRowTile;
  const bool in = i < n;
  const double* __restrict__ Ai = it.A + i;
  for (int c = tid; c < 3 * kMaxRhs + 1; c += kThreads) norms[c] = 0.0;
  __syncthreads();
  double sum = 0.0;
  for (int c0 = 0; c0 < it.nrhs; c0 += kPass) {
    const int cg = c0 + 8 * group;
    double acc[8], b[8], next[8], rows = 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      acc[c] = b[c] = in && cg + c < it.nrhs ? it.B[idx(i, cg + c, it.ldb)] : 0.0;
    auto fetch = [&](int j) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        next[u] = in && j + u < n ? Ai[(size_t)(j + u) * (size_t)it.lda] : 0.0;
    };
    fetch(0);
    for (int j0 = 0; j0 < n; j0 += kRowTile) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kRowTile * kPass / kThreads; ++q) {
        const int jj = tid % kRowTile, c = group + kGroups * q;
        const double x =
            j0 + jj < n && c0 + c < it.nrhs ? it.X[idx(j0 + jj, c0 + c, it.ldx)] : 0.0;
        Xs[jj][c] = x;
        if (j0 == r0) {  // (uniform: this CTA's rows of X)
          const double m = warp_max(magnitude(x));
          if (lane == 0 && c0 + c < it.nrhs) atomic_max_nonneg(&norms[kMaxRhs + c0 + c], m);
        }
      }
      __syncthreads();
      for (int jj = 0; jj < kRowTile; jj += 8) {
        double a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u] = next[u];
        fetch(j0 + jj + 8);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          rows += fabs(a[u]);
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            const double2 x = *(const double2*)&Xs[jj + u][8 * group + c];
            acc[c] = fma(-a[u], x.x, acc[c]);
            acc[c + 1] = fma(-a[u], x.y, acc[c + 1]);
          }
        }
      }
    }
    if (c0 == 0) sum = rows;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const bool live = cg + c < it.nrhs;
      if (in && live) it.R[idx(i, cg + c, it.ldr)] = acc[c];
      const double mr = warp_max(in ? magnitude(acc[c]) : 0.0);
      const double mb = warp_max(in ? magnitude(b[c]) : 0.0);
      if (lane == 0 && live) {
        atomic_max_nonneg(&norms[cg + c], mr);
        atomic_max_nonneg(&norms[2 * kMaxRhs + cg + c], mb);
      }
    }
  }
  sum = warp_max(in ? magnitude(sum) : 0.0);
  if (lane == 0) atomic_max_nonneg(&norms[3 * kMaxRhs], sum);
  __syncthreads();
  double* const all = work + (size_t)blockIdx.x * kResidualWork;
  int* const arrived = reinterpret_cast<int*>(all + 3 * kMaxRhs + 1);
  for (int c = tid; c < 3 * kMaxRhs + 1; c += kThreads)
    if (norms[c] > 0.0) atomic_max_nonneg(&all[c], norms[c]);
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = atomicAdd(arrived, 1) == (n + kRowTile - 1) / kRowTile - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  for (int c = tid; c < 3 * kMaxRhs + 1; c += kThreads) {
    norms[c] = __ldcg(&all[c]);
    all[c] = 0.0;
  }
  if (tid == 0) *arrived = 0;
  __syncthreads();
  if (tid < 32) {
    const double na = norms[3 * kMaxRhs];
    double e = 0.0;
    for (int c = lane; c < it.nrhs; c += 32) {
      const double den = na * norms[kMaxRhs + c] + norms[2 * kMaxRhs + c];
      const double v = den > 0.0 ? norms[c] / den : (norms[c] > 0.0 ? INFINITY : 0.0);
      e = fmax(e, v == v ? v : INFINITY);
    }
    e = warp_max(e);
    if (lane == 0) err[blockIdx.x] = e;
  }
}

// X += D for each item, the CTAs of an item on its columns in turn.
__global__ void axpy_kernel(const AxpyItem* __restrict__ items) {
  const AxpyItem it = items[blockIdx.x];
  for (int c = blockIdx.y; c < it.nrhs; c += gridDim.y)
    for (int i = threadIdx.x; i < it.n; i += blockDim.x)
      it.X[idx(i, c, it.ldx)] += it.D[idx(i, c, it.ldd)];
}

// dst (rows x cols, ldd) = src (rows x cols, lds) for each item, likewise (one
// CTA per item: 0.7 ms for an item of order 512).
__global__ void copy_kernel(const CopyItem* __restrict__ items) {
  const CopyItem it = items[blockIdx.x];
  for (int c = blockIdx.y; c < it.cols; c += gridDim.y)
    for (int i = threadIdx.x; i < it.rows; i += blockDim.x)
      it.dst[idx(i, c, it.ldd)] = it.src[idx(i, c, it.lds)];
}

constexpr int kCopyCtas = 16;  // per item


int launch_orders(const int* ns, const long long* rec, const int* ipiv, const int* jpiv,
                  int* row_order, int* col_order, int count, cudaStream_t st) {
  if (count <= 0) return kOk;
  dp::note_launch();
  orders_kernel<<<count, 32, 0, st>>>(ns, rec, ipiv, jpiv, row_order, col_order, count);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

int launch_solve(const SolveItem* items, int count, int max_n, int max_nrhs, cudaStream_t st) {
  if (count <= 0 || max_nrhs <= 0) return kOk;
  const size_t sm = sizeof(double) * (size_t)kCols * ld_of(max_n);
  if (!ensure_smem((const void*)solve_kernel, sm)) return kCudaFailure;
  dp::note_launch();
  solve_kernel<<<dim3(count, (max_nrhs + kCols - 1) / kCols), kThreads, sm, st>>>(items);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

int launch_residual(const ResidualItem* items, double* work, double* err, int count, int max_n,
                    cudaStream_t st) {
  if (count <= 0) return kOk;
  dp::note_launch();
  residual_kernel<<<dim3(count, (max_n + kRowTile - 1) / kRowTile), kThreads, 0, st>>>(items, work,
                                                                                        err);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

int launch_axpy(const AxpyItem* items, int count, cudaStream_t st) {
  if (count <= 0) return kOk;
  dp::note_launch();
  axpy_kernel<<<dim3(count, kCopyCtas), kThreads, 0, st>>>(items);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

int launch_copy(const CopyItem* items, int count, cudaStream_t st) {
  if (count <= 0) return kOk;
  dp::note_launch();
  copy_kernel<<<dim3(count, kCopyCtas), kThreads, 0, st>>>(items);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

}  // namespace serve
}  // namespace dp
