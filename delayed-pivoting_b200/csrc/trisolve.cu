// X = Q U^{-1} L^{-1} P B with many right-hand sides in ONE launch: the solve of
// getrs and of every refinement step, the row order of the factorisation
// applied while B is read and its column order while X is written.
//
// Work is cut into tasks (row block of 64, group of NC right-hand sides): the
// L tasks top down, then the U tasks bottom up, each level over all groups.
// CTAs take tasks by tickets from an atomic counter, so every block a task
// waits for was claimed earlier by a CTA that is already running: no
// co-residency (no cooperative launch) is needed, and the launch starts on
// whatever SMs are free.  A task
//   1. starts from its rows of P B (L) or of L's result (U),
//   2. for each earlier block j: waits for that block's values, puts them in
//      shared memory and subtracts T(i, j) y_j, T(i, j) held in registers and
//      loaded one block ahead (each T element is read once per group);
//      thread (r, q) takes row r and the 16 columns 16 q .. of every block.
//      The four partial sums of a block are folded into the row's value
//      behind the next block's barrier: kept apart until the end they lose
//      the cancellation that keeps an elimination's intermediate values
//      small, and the solutions were 1.2 - 1.7 times further off,
//   3. multiplies by the inverse of its 64 x 64 diagonal block (made once per
//      factorisation by diag_inverse_kernel, staged in shared memory while the
//      dependencies were awaited) - a product over all threads instead of a
//      64-step serial substitution,
//   4. publishes its values.
// The values are their own flag: the result buffers start as all-ones bit
// patterns (a NaN that no task publishes: a result with that pattern is
// written as the ordinary NaN), and a consumer polls the element it needs.
// The chain of blocks bounds the launch (2 n / 64 links): with a separate flag
// per block - a fence, a release store, an acquire poll and then a second
// round trip to L2 for the values - and one CTA for all right-hand sides a
// link took 2.9 us with one right-hand side (n = 4096: 186 us a triangle) and
// 13 us with 32 (n = 2311: 490 us).
// A wait that runs out sets *status = kDeviceTimeout; every CTA then returns.
#include <algorithm>
#include <atomic>

#include "dp_device.cuh"
#include "dp_kernels.h"

namespace dp {
namespace {

constexpr int kTB = 64;        // rows per block
constexpr int kTT = 256;       // threads
constexpr int kTQ = kTT / kTB; // column quarters of a block
constexpr int kTK = kTB / kTQ; // columns per quarter
constexpr int kTRhs = 64;      // right-hand sides per launch
constexpr int kTMaxGrid = 32;  // CTAs of one launch under a block-count policy

constexpr unsigned long long kUnset = ~0ull;  // not yet published

// CTAs of a launch (dp_tri_solve_grid): 0 -> as many as fit; g > 0 -> at most
// g; g < 0 -> one CTA per -g row blocks (at most kTMaxGrid).
std::atomic<int> g_tri_grid{0};

__device__ __forceinline__ unsigned long long ld_relaxed(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void publish(double* p, double v) {
  unsigned long long u = (unsigned long long)__double_as_longlong(v);
  if (u == kUnset) u = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}

__device__ __forceinline__ void cp_async16(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// inv + 2 * kTB * kTB * i holds, column-major, the inverse of the unit-lower
// L(i, i) then the inverse of the upper U(i, i) of diagonal block i (identity
// where the last block is shorter than kTB).  Warp w inverts columns w, w + 8,
// ... by substitution on the unit vectors, two rows per lane.
__global__ void __launch_bounds__(kTT) diag_inverse_kernel(const double* __restrict__ T,
                                                           long long ldt, int n, double* inv) {
  __shared__ double dg[kTB * kTB];
  const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = i * kTB, rows = min(kTB, n - r0);
  for (int e = tid; e < kTB * kTB; e += kTT) {
    const int k = e & (kTB - 1), c = e >> 6;
    dg[e] = (k < rows && c < rows) ? T[(r0 + k) + (long long)(r0 + c) * ldt] : 0.0;
  }
  __syncthreads();
  double* Li = inv + (size_t)2 * kTB * kTB * i;
  double* Ui = Li + kTB * kTB;
  double v0[8], v1[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int c = warp + 8 * m;
    v0[m] = lane == c ? 1.0 : 0.0;
    v1[m] = lane + 32 == c ? 1.0 : 0.0;
  }
  for (int k = 0; k < rows - 1; ++k) {
    const double l0 = lane > k ? dg[k * kTB + lane] : 0.0;
    const double l1 = lane + 32 > k ? dg[k * kTB + lane + 32] : 0.0;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const double yk = __shfl_sync(0xffffffffu, k < 32 ? v0[m] : v1[m], k & 31);
      v0[m] = fma(-l0, yk, v0[m]);
      v1[m] = fma(-l1, yk, v1[m]);
    }
  }
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int c = warp + 8 * m;
    Li[c * kTB + lane] = v0[m];
    Li[c * kTB + lane + 32] = v1[m];
    v0[m] = lane == c ? 1.0 : 0.0;
    v1[m] = lane + 32 == c ? 1.0 : 0.0;
  }
  const double inv0 = lane < rows ? 1.0 / dg[lane * kTB + lane] : 1.0;
  const double inv1 = lane + 32 < rows ? 1.0 / dg[(lane + 32) * kTB + lane + 32] : 1.0;
  for (int k = rows - 1; k >= 0; --k) {
    const double u0 = lane < k ? dg[k * kTB + lane] : 0.0;
    const double u1 = lane + 32 < k ? dg[k * kTB + lane + 32] : 0.0;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      if (k < 32) {
        if (lane == k) v0[m] *= inv0;
      } else {
        if (lane == k - 32) v1[m] *= inv1;
      }
      const double yk = __shfl_sync(0xffffffffu, k < 32 ? v0[m] : v1[m], k & 31);
      v0[m] = fma(-u0, yk, v0[m]);
      v1[m] = fma(-u1, yk, v1[m]);
    }
  }
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int c = warp + 8 * m;
    Ui[c * kTB + lane] = v0[m];
    Ui[c * kTB + lane + 32] = v1[m];
  }
}

struct SolveParams {
  const double* lu;
  long long ldlu;
  int n;
  const double* inv;
  const int *row, *col;  // composite row / column orders
  const double* B;
  long long ldb;
  double* X;
  long long ldx;
  int nrhs;
  double* mid;   // n x nrhs, L's result; all ones on entry
  double* xs;    // n x nrhs, U's result in elimination order; all ones on entry
  int* counter;  // all ones on entry
  int* status;
};

template <int NC>
constexpr size_t solve_smem() {
  return sizeof(double) * (2 * kTB * NC + 2 * kTQ * kTB * NC + kTB * kTB);
}

// The values of rows [r0, r0 + rows) and columns [c0, c0 + nc) of `src` once
// they are published, as dst[k * NC + c] (zeros elsewhere); false when the
// wait runs out or another CTA's did.
template <int NC>
__device__ __forceinline__ bool await_values(double* dst, const double* src, int n, int r0, int rows,
                                             int c0, int nc, const int* status) {
  constexpr int kPer = (kTB * NC + kTT - 1) / kTT;
  unsigned long long v[kPer];
  bool want[kPer], all;
  unsigned long long t0 = 0;
  for (unsigned it = 0;; ++it) {
    all = true;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int e = (int)threadIdx.x + u * kTT, k = e & (kTB - 1), c = e >> 6;
      want[u] = c < nc && k < rows;
      v[u] = want[u] ? ld_relaxed(src + (r0 + k) + (long long)(c0 + c) * n) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) all = all && v[u] != kUnset;
    if (all) break;
    if ((it & 63u) == 63u) {
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > kSpinLimitNs || ld_volatile_i32(status) != kOk) break;
    }
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int e = (int)threadIdx.x + u * kTT, k = e & (kTB - 1), c = e >> 6;
    if (c < NC) dst[k * NC + c] = __longlong_as_double((long long)v[u]);
  }
  return all;
}

template <int NC>
__global__ void __launch_bounds__(kTT, 2) lu_solve_kernel(const __grid_constant__ SolveParams p) {
  extern __shared__ __align__(16) double tsm[];
  double* const ys = tsm;                      // [2][kTB][NC] values of the block in hand
  double* const red = ys + 2 * kTB * NC;       // [2][kTQ][NC][kTB] partial sums
  double* const dg = red + 2 * kTQ * kTB * NC; // inverse of the diagonal block, column-major
  constexpr int kOwn = (NC + kTQ - 1) / kTQ;   // columns q, q + kTQ, .. of row r: this thread's
  __shared__ int ticket;
  const int tid = threadIdx.x, r = tid & (kTB - 1), q = tid >> 6;
  const int n = p.n, nblk = (n + kTB - 1) / kTB;
  const int groups = (p.nrhs + NC - 1) / NC;
  const int tasks = 2 * nblk * groups;
  for (;;) {
    __syncthreads();  // ticket, ys, red and dg are free
    if (tid == 0) ticket = atomicAdd(p.counter, 1) + 1;
    __syncthreads();
    const int task = ticket;
    if (task >= tasks) return;
    const int level = task / groups, c0 = (task - level * groups) * NC;
    const int nc = min(NC, p.nrhs - c0);
    const bool up = level >= nblk;
    const int i = up ? 2 * nblk - 1 - level : level;
    const int r0 = i * kTB, rows = min(kTB, n - r0);
    const int deps = up ? nblk - 1 - i : i;
    {
      const double* src = p.inv + (size_t)2 * kTB * kTB * i + (up ? kTB * kTB : 0);
      for (int e = 2 * tid; e < kTB * kTB; e += 2 * kTT) cp_async16(dg + e, src + e);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // T(i, j)'s part of this thread: row r, columns 16 q + k
    const double* const trow = p.lu + (r0 + r) + (long long)(kTK * q) * p.ldlu;
    auto load_tile = [&](double (&t)[kTK], int d) {
      const int j = up ? nblk - 1 - d : d;
      const double* src = trow + (long long)j * kTB * p.ldlu;
      const int left = n - j * kTB - kTK * q;  // columns of this quarter inside the matrix
#pragma unroll
      for (int k = 0; k < kTK; ++k)
        t[k] = (r < rows && k < left) ? src[(long long)k * p.ldlu] : 0.0;
    };
    double tile[2][kTK];
    if (deps > 0) load_tile(tile[0], 0);
    double acc[NC], own[kOwn];
#pragma unroll
    for (int u = 0; u < kOwn; ++u) own[u] = 0.0;
    bool good = true;
    if (up) {
      // L's result at this block: awaited like any other block's values
      good = await_values<NC>(ys, p.mid, n, r0, rows, c0, nc, p.status);
      if (!__syncthreads_and(good)) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (tid == 0) atomicCAS(p.status, kOk, kDeviceTimeout);
        break;
      }
#pragma unroll
      for (int u = 0; u < kOwn; ++u)
        if (q + u * kTQ < NC) own[u] = ys[r * NC + q + u * kTQ];
      __syncthreads();
    } else if (r < rows && q < nc) {
      const long long src = p.row[r0 + r];
#pragma unroll
      for (int u = 0; u < kOwn; ++u)
        if (q + u * kTQ < nc) own[u] = p.B[src + (long long)(c0 + q + u * kTQ) * p.ldb];
    }
    // the four partial sums of block d, in the order of its columns
    auto folded = [&](int d, int c) {
      const double* s = red + ((d & 1) * kTQ * NC + c) * kTB + r;
      return (s[0] + s[NC * kTB]) + (s[2 * NC * kTB] + s[3 * NC * kTB]);
    };
    auto put = [&](int d) {
#pragma unroll
      for (int c = 0; c < NC; ++c) red[(((d & 1) * kTQ + q) * NC + c) * kTB + r] = acc[c];
    };
    auto fold = [&](int d) {
#pragma unroll
      for (int u = 0; u < kOwn; ++u)
        if (q + u * kTQ < NC) own[u] -= folded(d, q + u * kTQ);
    };
    const double* const from = up ? p.xs : p.mid;
    auto step = [&](const double (&t)[kTK], double (&next)[kTK], int d) -> bool {
      const int j = up ? nblk - 1 - d : d;
      if (d + 1 < deps) load_tile(next, d + 1);
      double* const y = ys + (d & 1) * kTB * NC;
      good = await_values<NC>(y, from, n, j * kTB, min(kTB, n - j * kTB), c0, nc, p.status);
      // (this half of ys and of red was last read before the previous barrier)
      if (!__syncthreads_and(good)) return false;
      const double* yq = y + kTK * q * NC;
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] = 0.0;
#pragma unroll
      for (int k = 0; k < kTK; ++k)
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] = fma(t[k], yq[k * NC + c], acc[c]);
      put(d);
      if (d > 0) fold(d - 1);
      return true;
    };
    bool ok = true;
    for (int d = 0; ok && d < deps; d += 2) {
      ok = step(tile[0], tile[1], d);
      if (ok && d + 1 < deps) ok = step(tile[1], tile[0], d + 1);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!ok) {
      if (tid == 0) atomicCAS(p.status, kOk, kDeviceTimeout);
      break;
    }
    // the last block's partial sums, then the diagonal block's inverse
    __syncthreads();
    if (deps > 0) fold(deps - 1);
    double* const y = ys + (deps & 1) * kTB * NC;
#pragma unroll
    for (int u = 0; u < kOwn; ++u)
      if (q + u * kTQ < NC) y[r * NC + q + u * kTQ] = own[u];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0;
#pragma unroll
    for (int k = 0; k < kTK; ++k) {
      const double a = dg[(kTK * q + k) * kTB + r];
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] = fma(a, y[(kTK * q + k) * NC + c], acc[c]);
    }
    put(deps);
    __syncthreads();
    const long long xrow = up && r < rows ? p.col[r0 + r] : 0;
#pragma unroll
    for (int u = 0; u < kOwn; ++u)
      if (const int c = q + u * kTQ; c < nc && r < rows) {
        const double s = folded(deps, c);
        const size_t at = (size_t)(r0 + r) + (size_t)(c0 + c) * n;
        publish((up ? p.xs : p.mid) + at, s);
        if (up) p.X[xrow + (long long)(c0 + c) * p.ldx] = s;
      }
  }
}

template <int NC>
int launch_solve(const SolveParams& p, cudaStream_t st) {
  const void* fn = (const void*)lu_solve_kernel<NC>;
  const size_t smem = solve_smem<NC>();
  if (!ensure_smem(fn, smem)) return kCudaFailure;
  const int sms = sm_count();
  const int per_sm = occupancy_once(fn, kTT, smem);
  if (sms < 1 || per_sm < 1) return kCudaFailure;
  const int nblk = (p.n + kTB - 1) / kTB;
  const int per_level = (p.nrhs + NC - 1) / NC;
  const int policy = g_tri_grid.load(std::memory_order_relaxed);
  const int most = policy == 0 ? sms * per_sm
                   : policy > 0 ? policy
                                : std::min(kTMaxGrid, (nblk - policy - 1) / -policy);
  const int grid = std::max(1, std::min({nblk * per_level, most, sms * per_sm}));
  note_launch();
  lu_solve_kernel<NC><<<grid, kTT, smem, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

}  // namespace

size_t tri_inverse_doubles(int n) { return (size_t)2 * kTB * kTB * ((n + kTB - 1) / kTB); }

int launch_diag_inverse(const double* lu, long long ldlu, int n, double* inv, cudaStream_t st) {
  if (n <= 0) return kOk;
  note_launch();
  diag_inverse_kernel<<<(n + kTB - 1) / kTB, kTT, 0, st>>>(lu, ldlu, n, inv);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

int lu_solve_pass(int nrhs) { return std::min(nrhs, kTRhs); }

size_t lu_solve_work_bytes(int n, int pass) { return sizeof(double) * 2 * (size_t)n * pass + 16; }

int launch_lu_solve(const double* lu, long long ldlu, int n, const double* inv, const int* row,
                    const int* col, const double* B, long long ldb, double* X, long long ldx,
                    int nrhs, void* work, int pass, int* status, cudaStream_t st) {
  if (n <= 0 || nrhs <= 0) return kOk;
  for (int c0 = 0; c0 < nrhs; c0 += pass) {
    SolveParams p;
    p.lu = lu;
    p.ldlu = ldlu;
    p.n = n;
    p.inv = inv;
    p.row = row;
    p.col = col;
    p.B = B + (size_t)c0 * ldb;
    p.ldb = ldb;
    p.X = X + (size_t)c0 * ldx;
    p.ldx = ldx;
    p.nrhs = std::min(pass, nrhs - c0);
    p.mid = static_cast<double*>(work);
    p.xs = p.mid + (size_t)n * p.nrhs;
    p.counter = reinterpret_cast<int*>(p.xs + (size_t)n * p.nrhs);
    p.status = status;
    if (cudaMemsetAsync(work, 0xFF, lu_solve_work_bytes(n, p.nrhs), st) != cudaSuccess)
      return kCudaFailure;
    // Right-hand sides per task: few columns are computed that are not there,
    // and at most eight, so that a link of the chain stays short (a block's
    // product takes 64 NC cycles of the FP64 pipe) and the groups spread over
    // the SMs.
    const int rc = p.nrhs == 1   ? launch_solve<1>(p, st)
                   : p.nrhs == 2 ? launch_solve<2>(p, st)
                   : p.nrhs <= 4 ? launch_solve<4>(p, st)
                                 : launch_solve<8>(p, st);
    if (rc != kOk) return rc;
  }
  return kOk;
}

}  // namespace dp

extern "C" int dp_tri_solve_grid(int policy) {
  if (policy > 1024 || policy < -1024) return -2000;
  return dp::g_tri_grid.exchange(policy);
}
