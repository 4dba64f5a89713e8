// Kernel parameter blocks and host-side launch wrappers of the
// delayed-pivoting LU.  Internal to the library (not part of the C ABI).
#pragma once
#include <vector>

#include <cuda_runtime.h>

#include "delayed_pivoting_b200.h"
#include "dp_device.cuh"

namespace dp {

struct PanelParams {
  double* a;
  long long lda;
  int m;
  int begin, end;     // panel columns [begin, end), rows [begin, m)
  int rows_per_cta;   // R
  int positioned;     // pivot of the first step already sits at (begin, begin)
  int parity;         // which of the two slot buffers this launch uses
  int max_ctas;       // slot buffer stride
  int w_max;          // row-data buffer stride - 1
  double threshold;
  int* ipiv;          // device swap history (global step index)
  State* state;
  unsigned long long* slots;  // mailboxes [2][4][max_ctas reader][max_ctas writer][2 words]
  double* xdata;              // [4][max_ctas][w_max + 1]
  double* rowk;               // [4][w_max + 1]
  int* swap_block;            // [end - begin]: source row of block row begin + i
  int* swap_extra;            // [2 * (end - begin)]: (dst, src) pairs below `end`
  int gated;                  // cluster kernel: 1 -> do nothing when state->stop_k >= 0 (an
                              // earlier panel of the same enqueued sequence stopped)
};

__global__ void panel_factor_kernel(PanelParams p);
// Cluster variant: one thread-block cluster of C <= 16 CTAs holds the panel
// in distributed shared memory (launched with a cluster dimension).
__global__ void panel_cluster_kernel(PanelParams p);
size_t panel_cluster_smem_bytes(int w, int rows_per_cta);
// Cluster variant with the sub-panel in registers (panel_reg.cu), for up to
// panel_reg_max_rows() rows per CTA: the kernel instance for R rows per CTA
// (nullptr beyond the limit) and its dynamic shared memory.
int panel_reg_max_rows();
const void* panel_reg_kernel_for(int rows_per_cta);
int panel_reg_threads(int rows_per_cta);
size_t panel_reg_smem_bytes(int w, int rows_per_cta);
int panel_cluster_threads();
constexpr int kPanelThreadsHost = 256;
// Single-CTA panel (batched.cu) for panels of at most panel_small_max_rows()
// rows and panel_small_max_width() columns: same contract as the cluster
// panel, rows register-resident, one CTA barrier per step.
int panel_small_max_rows();
int panel_small_max_width();
int launch_panel_small(const PanelParams& pp, cudaStream_t st);
// x[0..len) <- seeded N(0,1) (hashed Box-Muller; tuner inputs).
void launch_fill_normal(double* x, long long len, unsigned long long seed, cudaStream_t st);
size_t panel_smem_bytes(int w, int rows_per_cta);

// Applies the composite row permutation of one panel (swap list written by
// panel_factor_kernel) to columns [c0, c1) and [c2, c3).  gate_begin >= 0:
// do nothing when state->stop_k is in [0, gate_begin) (a panel before this
// one stopped; its own stop, at or after gate_begin, still applies).
// [s0, s1) within [c2, c3): when no panel stopped (state->stop_k < 0) and the
// panel is at most laswp_solve_max_width() wide, also solve the panel's block
// rows of those columns with its unit lower triangle (U12 = L11^{-1} A12).
int laswp_solve_max_width();
void launch_laswp(double* a, long long lda, int begin, int nblock, const int* swap_block,
                  const int* swap_extra, const State* state, int c0, int c1, int c2, int c3,
                  cudaStream_t s, int gate_begin = -1, int s0 = 0, int s1 = 0);

// Swap lists of up to kSwapSeqLists consecutive panels (kSwapSeqEntries
// entries in all) applied in order by one launch of laswp_seq_kernel.
constexpr int kSwapSeqLists = 64;
constexpr int kSwapSeqEntries = 2048;
struct SwapSeq {
  int lists;
  int base;  // first row of the first panel
  int width[kSwapSeqLists];
};

// Applies the swap lists of `lists` consecutive panels starting at row
// `base` (panel p of width widths[p], its block part at blk[begin_p - base],
// up to widths[p] extra pairs at ext[2 (begin_p - base)], the unused ones
// holding a negative destination) to the columns [c0, c1) and [c2, c3), in
// panel order.  Returns the number of launches, or -1 when a panel is wider
// than the kernel's lists.
int launch_laswp_seq(double* a, long long lda, const int* blk, const int* ext, int base,
                     const int* widths, int lists, int c0, int c1, int c2, int c3,
                     cudaStream_t s);

// B(w x nc) <- L^{-1} B, L unit lower (w x w) at a(r0, r0), B at a(r0, c0);
// w <= trsm_max_width().  A non-null `gate`: do nothing when *gate >= 0
// (the stop word of an enqueued panel sequence, read when the kernel starts).
int trsm_max_width();
void launch_trsm_unit_lower(double* a, long long lda, int r0, int w, int c0, int nc,
                            cudaStream_t s, const int* gate = nullptr);
// T (w x w, column stride ldt) <- I - L^{-1} for the unit lower w x w block L,
// w <= lower_inverse_max_width(): the solve L^{-1} B is then B - T B, a GEMM.
int lower_inverse_max_width();
void launch_lower_inverse(const double* L, long long ldl, int w, double* T, long long ldt,
                          cudaStream_t s);
// dst <- src for a rows x cols column-major block (device memory).
void launch_copy_block(const double* src, long long lds, double* dst, long long ldd, int rows,
                       int cols, cudaStream_t s);
// Same with separate operands.
void launch_trsm_lower_unit(const double* L, long long ldl, double* B, long long ldb, int w, int nc,
                            cudaStream_t s, const int* gate = nullptr);

// C(M x N) -= A(M x K) * B(K x N); all three inside the same column-major
// matrix (or any column-major operands).  `gate` as for the TRSM.
void launch_gemm_minus(int M, int N, int K, const double* A, long long lda, const double* B,
                       long long ldb, double* C, long long ldc, cudaStream_t s,
                       const int* gate = nullptr);

// The same when *run < 0 only (read when the kernel starts).
void launch_gemm_minus_if(int M, int N, int K, const double* A, long long lda, const double* B,
                          long long ldb, double* C, long long ldc, cudaStream_t s, const int* run);

// C(M x N) -= A(M x K) * B(K x N) on the integer tensor cores (gemm_i8.cu), K <=
// i8_max_k(), where the operands show that no element is further off than its
// FP64 sum, and else by the FP64 kernel.  launch_i8_split_a takes A's digits (M <=
// m rows) and the balance of the K terms from the first of the `cols` columns of
// B; any number of updates with that A then follow on the same stream, each over
// up to n columns.  Once an update has gone to the FP64 kernel, so do those
// after it.  Return status codes.
int i8_max_k();
size_t i8_bytes(long long m, long long n);  // of the memory behind an I8Update
struct I8Update {
  void *a_digits = nullptr, *b_digits = nullptr;
  int *bad = nullptr, *least = nullptr, *ks = nullptr;
};
I8Update i8_update(void* mem, long long m, long long n);
int launch_i8_split_a(const I8Update& u, int M, int K, const double* A, long long lda,
                      const double* B, long long ldb, int cols, cudaStream_t s);
int launch_gemm_minus_i8(const I8Update& u, int M, int N, int K, const double* A, long long lda,
                         const double* B, long long ldb, double* C, long long ldc, int* status,
                         cudaStream_t s);

// Lower triangle of the symmetric N x N C -= A(N x K) * B(K x N); C's strict
// upper triangle is not written.
void launch_gemm_minus_lower(int N, int K, const double* A, long long lda, const double* B,
                             long long ldb, double* C, long long ldc, cudaStream_t s);

// C(M x N) -= A(M x K) * B(K x N) on the tensor cores (BF16 split into
// `terms` pieces: 2 -> three products, 3 -> six products; FP32 accumulation in
// TMEM); scratch of mixed_scratch_bytes(M, N, K, terms) bytes.  Returns a
// status code.
size_t mixed_scratch_bytes(int max_rows, int max_cols, int max_k, int terms);
int launch_gemm_minus_mixed(int M, int N, int K, const double* A, long long lda, const double* B,
                            long long ldb, double* C, long long ldc, void* scratch, int terms,
                            int* status, cudaStream_t s);
// Split pieces of a mixed precision (0 for DP_PRECISION_FP64).
inline int mixed_terms(int precision) {
  return precision == DP_PRECISION_MIXED_BF16X6 ? 3 : precision == DP_PRECISION_MIXED_BF16X3 ? 2 : 0;
}
inline bool valid_precision(int precision) {
  return precision == DP_PRECISION_FP64 || precision == DP_PRECISION_MIXED_BF16X3 ||
         precision == DP_PRECISION_MIXED_BF16X6;
}

// Stream-ordered device memory from the library's two pools (pool.cu), freed
// with cudaFreeAsync: workspaces of one call, and factors that outlive it.
cudaError_t workspace_alloc(void** out, size_t bytes, cudaStream_t st);
cudaError_t resident_alloc(void** out, size_t bytes, cudaStream_t st);
// Gives the current device's unused pool memory back to the driver.
void memory_trim();
// The calling thread's pinned block for device-to-host copies, nullptr when
// `bytes` exceeds it or it cannot be had; its contents belong to the caller
// until the next copy this thread makes through it.
constexpr size_t kPinnedStageBytes = 512 * 1024;
void* pinned_stage(size_t bytes);

// Full-pivot search over a(k:m, k:n); result in state->fallback.
void launch_search_active(const double* a, long long lda, int m, int n, int k, State* state,
                          Cand* block_cands, int max_blocks, cudaStream_t s);

// Column-fallback search (delayed_dgetrf_column.cpp:30-45): right-most column
// j in (k, n) whose active part has a magnitude > threshold, and its argmax row.
void launch_search_nonzero_column(const double* a, long long lda, int m, int n, int k,
                                  double threshold, State* state, cudaStream_t s);

// Ends a fallback search at step k (state->fallback): moves the pivot found to
// (k, k) by full row and column swaps, records it and re-arms state->stop_k, or
// sets state->delayed when no magnitude exceeds the threshold.
void launch_apply_fallback(double* a, long long lda, int m, int n, int k, double threshold,
                           State* state, int* ipiv, int* jpiv, cudaStream_t s);

void launch_identity_records(int* ipiv, int* jpiv, int count, cudaStream_t s);

// ---- triangular solves with many right-hand sides (trisolve.cu) ----------

// X <- Q U^{-1} L^{-1} P B (n x nrhs) in one launch per `pass` right-hand sides
// (at most lu_solve_pass(nrhs), the fastest; no result bit depends on it):
// row / col are the composite orders (B row row[i] is eliminated i-th, unknown
// col[i] takes the i-th value), X may be B.  `inv` holds the inverses of the
// 64 x 64 diagonal blocks of L and U (launch_diag_inverse,
// tri_inverse_doubles(n) doubles, 16-byte aligned), `work`
// lu_solve_work_bytes(n, pass) bytes; a bounded wait that runs out sets
// *status = kDeviceTimeout.
size_t tri_inverse_doubles(int n);
int launch_diag_inverse(const double* lu, long long ldlu, int n, double* inv, cudaStream_t st);
int lu_solve_pass(int nrhs);
size_t lu_solve_work_bytes(int n, int pass);
int launch_lu_solve(const double* lu, long long ldlu, int n, const double* inv, const int* row,
                    const int* col, const double* B, long long ldb, double* X, long long ldx,
                    int nrhs, void* work, int pass, int* status, cudaStream_t st);

// ---- resident factorisations (solve.cu) ----------------------------------

// A factorisation kept on the device for repeated solves: the compact L\U,
// its swap histories (host) and their composite row / column orders (device).
struct Factor {
  int n = 0;
  int info = -1;
  int precision = 0;                  // DP_PRECISION_* of the factors held now
  int refactored = 0;                 // 1 once a stalled refinement forced FP64
  double normA = 0.0;                 // ||A||_inf
  double factor_ms = 0.0;             // device time of all factorisations
  double* lu = nullptr;
  int* d_perm = nullptr;              // row order [n], column order [n]
  double* d_inv = nullptr;            // inverses of the diagonal blocks of L and U
  int panel_rows = 0;                 // rows per panel CTA of its factorisations (0: default)
  std::vector<int> ipiv, jpiv;
};

// Device bytes a Factor of order n holds.
size_t factor_bytes(int n);
// Factor A (n x n, lda, device, not modified) at `precision`; synchronises st.
int factor_create(Factor** out, int n, const double* A, int lda, int precision, cudaStream_t st,
                  int panel_rows = 0);
// Solve A X = B with FP64 refinement; B (n x nrhs, device) becomes X.  Mixed
// factors whose refinement stalls are replaced by plain FP64 factors of A.
int factor_solve(Factor* f, const double* A, int lda, double* B, int ldb, int nrhs, int max_iter,
                 double tol, dp_ir_result* res, cudaStream_t st);
void factor_destroy(Factor* f, cudaStream_t st);
// Hager-Higham estimate of kappa_1(A) = ||A||_1 ||A^{-1}||_1 through the
// factors held now (inv_norm: the estimate of ||A^{-1}||_1, may be null);
// synchronises st.  A singular factorisation gives infinity.
int factor_condest(Factor* f, const double* A, int lda, double* kappa, double* inv_norm,
                   cudaStream_t st);

// Launches a kernel that begins with after_previous_kernel(): its CTAs are in
// place when the last of the kernel before it on the stream has left, instead of
// being sent then.  The panels' chains of short kernels lose about 1 us at each
// link: LU n = 1024 2.09 -> 1.92 ms, 2048 4.61 -> 4.35, 8192 26.5 -> 25.7.  Plain
// under capture.
template <class... P, class... Q>
void launch_behind(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st,
                   Q... args) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &capture);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace dp
