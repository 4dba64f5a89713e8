// FP64 trailing update C -= A B on the 8-bit integer tensor cores.
//
// The FP64 tensor path (gemm_f64.cu) runs at 28.8 TFLOP/s at K = 256, and the
// large factorisations are bound by it.  Here each row of A and each column of
// B is scaled by a power of two and written as a 64-bit integer in eight
// balanced base-256 digits (the Ozaki scheme: K. Ozaki, T. Ogita, S. Oishi,
// S. M. Rump, "Error-free transformations of matrix multiplication by using
// fast routines of matrix multiplication and its applications", 2012; on
// integer tensor cores: H. Ootomo, K. Ozaki, R. Yokota, 2024): the products of
// digits i and j are formed exactly in 32-bit integers by tcgen05.mma kind::i8,
// those with the same i + j = d share an accumulator (|sum| <= 8 K 2^14 <
// 2^26), and the 36 products with d <= 7 are added in FP64 with their weights
// 2^(-8 d), smallest first.
//
// Error: with alpha_i and beta_j the largest scaled entries of row i of A and
// column j of B, the ends of the digits and the products left out (d >= 8) come
// to about 2^-59 alpha_i beta_j over K = 256 terms, whatever the sizes of the
// terms themselves.  An FP64 sum errs by some 2^-55 of sum_k |a_ik b_kj|.  So the
// scheme is the better one where that sum is not far below alpha_i beta_j, and
// loses every bit where the two maxima stand in different terms: rows of U12 that
// are large in some columns and small, or zero, in others.  Two steps keep it to
// the first kind:
//   balance  the terms are scaled by 2^+-ks[k], the size of row k of U12 in a
//            sample of columns, each column in units of its own size, so that the
//            rows' order of magnitude (the pivots') does not count (row_scale_kernel);
//   proof    the split kernels add up min(1, 16 |a'_ik| / alpha_i) for every row
//            and min(1, 16 |b'_kj| / beta_j) for every column.  xy >= x + y - 1
//            holds in [0, 1], so that two sums that exceed K + 32 together show
//            sum_k |a_ik b_kj| >= 32 / 256 alpha_i beta_j: every element is then
//            at least as close as its FP64 sum.  Dense operands have margin (N(0, 1)
//            from n = 2560 to 16384, rows or columns of scales 1e-20 to 1e20:
//            smallest sums 0.52 K and 0.70 K), and zero rows, columns and terms
//            cost none.  Where the least of the rows' sums and a column's fall short
//            the update is the FP64 kernel's.
//            Balance, splits and proof are bound by the trip to memory of one pass
//            over A and B and take 15.7, 21.2 and 16.4 us a launch in an LU of n =
//            16384, 13.5, 20.4 and 14.8 before the proof (the update: 557 us).
// Measured, random operands with K = 256: 0.42 u of the result's size (root mean
// square) and at most 2.7 u, FP64 path 4.8 and 42; on L21 U12 of an N(0, 1) matrix
// (n = 4096) seven digits (28 products, a quarter faster) 8.6e-15, FP64 path
// 2.4e-15.  Integers up to 2^62 times a row's scale, exact zeros and zero columns
// stay exact.  Each scale puts the largest entry just below 127.5, the whole range
// of the first digit.
//
// Operands outside the scheme - those without the proof, a NaN, an infinity, or a
// row / column whose largest entry is outside 2^+-kMaxExp - set a flag on the
// device: the kernel then does nothing and the FP64 kernel behind it does the
// update (its CTAs return at once otherwise).
//
// Pipeline: split kernels write the digits as the shared-memory images of 128
// (A) or 64 (B) rows x 32 bytes of K, all eight digits of a piece side by side,
// so that a piece is one bulk copy.  The update kernel takes tiles of 128 x 64,
// a weight per 64-column accumulator (all 512 columns of tensor memory), in two
// passes over K: the weights d = 7 .. 4 (26 products of all digits), then d = 3
// .. 0 (10 products of the first four digits).  A copy warp feeds a four-stage
// ring; an MMA warp issues the products, those of one digit of A in a row with
// that digit kept in the tensor path's collector (an MMA of 128 x 64 x 32 is
// bound by its reads of shared memory: 48 cycles, 34 with A kept; on real data
// the power limit holds the clock down, 57 in this kernel); 16 epilogue
// warps read one pass's accumulators while the other's products run, and
// subtract from C behind the next tile's first pass.  Wider tiles (128 x 128,
// four accumulators, each pass waiting for the reads of the one before) took
// 583 us for 8192 x 8192 x 256.
#include <algorithm>
#include <climits>

#include "dp_device.cuh"
#include "dp_kernels.h"
#include "umma.cuh"

namespace dp {
namespace i8 {

constexpr int kDigits = 8, kHead = 4;          // digits; weights of the second pass
constexpr int BM = 128, BN = 64, BK = 32;      // tile; bytes of K per piece
constexpr int kImageA = BM * BK, kImageB = BN * BK;  // one digit of a piece
constexpr int kPieceA = kDigits * kImageA, kPieceB = kDigits * kImageB;
constexpr int kStage = kPieceA + kPieceB, kStages = 4;
constexpr size_t kSmem = (size_t)kStages * kStage + 1024;
constexpr int kMaxExp = 400;  // scales and their products stay normal numbers
constexpr int kEpiWarps = 16;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kEpiCols = BN / (kEpiWarps / 4);  // 16 columns per epilogue thread
constexpr unsigned kTmemCols = 512;
constexpr int kMaxK = 256;
constexpr int kScaleCols = 64;  // columns of U12 that balance the K terms

// Byte of (row, k) inside a piece's image: 8 rows x 16 bytes contiguous, the
// two 16-byte halves of K side by side, then the next 8 rows.
__device__ __forceinline__ int image_at(int row, int k) {
  return (row >> 3) * 256 + (k >> 4) * 128 + (row & 7) * 16 + (k & 15);
}

// ---------------------------------------------------------------- split ----
// The scale of a row or column with largest magnitude mx: mx 2^(7 - e) < 127.5
// and as near as a power of two brings it; false when the scheme does not
// cover it (mx == 0: e = 0, digits are zero).
__device__ __forceinline__ bool scale_exponent(double mx, int& e) {
  const unsigned hi = (unsigned)__double2hiint(mx);
  const int be = (int)(hi >> 20);  // (mx >= 0)
  e = mx == 0.0 ? 0 : be - 1022 + ((hi & 0xfffffu) >= 0xfd000u);
  return mx == 0.0 || (be > 0 && be < 0x7ff && e <= kMaxExp && e >= -kMaxExp);
}

__device__ __forceinline__ double pow2(int e) {  // normal range
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// x * 2^(63 - e) as an integer in digits, most significant first.
__device__ __forceinline__ void digits_of(double x, double up, unsigned char (&d)[kDigits]) {
  long long v = __double2ll_rn(x * up);
#pragma unroll
  for (int q = kDigits - 1; q > 0; --q) {
    const long long low = (long long)(signed char)(v & 0xff);
    d[q] = (unsigned char)low;
    v = (v - low) >> 8;
  }
  d[0] = (unsigned char)v;
}

// Digits of 4 consecutive k as one word per digit.
__device__ __forceinline__ void digit_words(const double (&x)[4], double up,
                                            unsigned (&w)[kDigits]) {
#pragma unroll
  for (int q = 0; q < kDigits; ++q) w[q] = 0u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned char d[kDigits];
    digits_of(x[i], up, d);
#pragma unroll
    for (int q = 0; q < kDigits; ++q) w[q] |= (unsigned)d[q] << (8 * i);
  }
}

// Balance of the K terms: ks[k] = the exponent of the largest of the first `cols`
// (at most kScaleCols) entries of row k of B, each in units of the largest of its
// column.  A's columns are scaled by 2^ks[k] and B's rows by 2^-ks[k] before the
// digits are taken.  Without it, rows of very different size in the matrix being
// factored (row k of U small, its multipliers large) put the terms that matter
// below the digits of the row's largest multiplier.  A row without an entry there
// takes the smallest exponent of the others, which raises no row of A.  Also sets
// the operands' flag and the least sum of A's rows (split_a_kernel) to their start.
__global__ void __launch_bounds__(kMaxK) row_scale_kernel(const double* __restrict__ B,
                                                          long long ldb, int K, int cols, int* ks,
                                                          int* bad, int* least) {
  __shared__ int top[kScaleCols], low;
  const int k = threadIdx.x;
  if (k < kScaleCols) top[k] = 0;
  if (k == 0) {
    low = INT_MAX;
    *bad = 0;
    *least = INT_MAX;
  }
  __syncthreads();
  int mine = INT_MIN;
  for (int pass = 0; pass < 2; ++pass) {  // the columns' sizes, then the rows'
    for (int c0 = 0; c0 < cols; c0 += 16) {
      int e[16];  // biased exponents, 0 for zero
#pragma unroll
      for (int u = 0; u < 16; ++u)
        e[u] = k < K && c0 + u < cols ? (__double2hiint(B[idx(k, c0 + u, ldb)]) >> 20) & 0x7ff : 0;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        if (pass == 0) {
          const int m = __reduce_max_sync(~0u, e[u]);
          if ((k & 31) == 0 && m > 0) atomicMax(&top[c0 + u], m);
        } else if (e[u] > 0) {
          mine = max(mine, e[u] - top[c0 + u]);
        }
      }
    }
    __syncthreads();
  }
  const int least_here = __reduce_min_sync(~0u, mine == INT_MIN ? INT_MAX : mine);
  if ((k & 31) == 0) atomicMin(&low, least_here);
  __syncthreads();
  if (mine == INT_MIN) mine = low == INT_MAX ? 0 : low;
  if (k < K) ks[k] = max(mine, -kMaxExp);
}

// Sums of min(1, 16 |x| / largest) are kept in units of 1 / kShare.
constexpr int kShare = 16, kProof = 32;
__device__ __forceinline__ float share_of(double x, double per_max) {
  return fminf(1.0f, (float)(fabs(x) * per_max));
}

// A (M x K, column-major) -> digit images [row tile][piece][digit], scales ra[m]
// = 2^e, the least of the rows' sums in *least (rows of zeros apart).  32 rows a
// CTA; the columns arrive a warp a column (coalesced), warp w then packs piece w: a
// lane its row's 32 columns.
__global__ void __launch_bounds__(256) split_a_kernel(const double* __restrict__ A, long long lda,
                                                      int M, int K, int pieces,
                                                      const int* __restrict__ ks,
                                                      unsigned char* __restrict__ out,
                                                      double* __restrict__ ra, int* bad,
                                                      int* least) {
  extern __shared__ double tile[];  // [32][kMaxK + 1]
  __shared__ double mx[8][32];
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  double m = 0.0;
  bool nan = false;
  for (int k = warp; k < pieces * BK; k += 8) {
    const double x = (row < M && k < K) ? A[idx(row, k, lda)] * pow2(ks[k]) : 0.0;
    tile[lane * (kMaxK + 1) + k] = x;
    m = fmax(m, fabs(x));
    nan |= x != x;
  }
  mx[warp][lane] = nan ? __longlong_as_double(0x7ff0000000000000ll) : m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) m = fmax(m, mx[w][lane]);
  int e;
  const bool ok = scale_exponent(m, e);
  const bool counts = ok && m > 0.0;
  const double per_max = counts ? 16.0 / m : 0.0;
  float sum = 0.0f;
  for (int k = warp; k < K; k += 8) sum += share_of(tile[lane * (kMaxK + 1) + k], per_max);
  part[warp][lane] = sum;
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) sum += part[w][lane];
    const int own = __reduce_min_sync(~0u, row < M && counts ? (int)(kShare * sum) : INT_MAX);
    if (lane == 0) atomicMin(least, own);
    if (row < M) {
      ra[row] = ok ? pow2(e) : 0.0;
      if (!ok) *bad = -1;
    }
  }
  if (row >= M || warp >= pieces || !ok) return;
  const double up = pow2(63 - e);
  unsigned char* const dst = out + ((size_t)(row / BM) * pieces + warp) * kPieceA;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint4 v[kDigits];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      double x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = tile[lane * (kMaxK + 1) + warp * BK + 16 * h + 4 * u + i];
      unsigned w[kDigits];
      digit_words(x, up, w);
#pragma unroll
      for (int q = 0; q < kDigits; ++q) (&v[q].x)[u] = w[q];
    }
#pragma unroll
    for (int q = 0; q < kDigits; ++q)
      *reinterpret_cast<uint4*>(dst + q * kImageA + image_at(row % BM, 16 * h)) = v[q];
  }
}

// B (K x N, column-major) -> digit images [column tile][piece][digit], scales
// cb[n] = 2^(e - 70), and the proof for each column: its sum beside the least of
// A's rows.  A warp per column, a lane packs 8 consecutive rows.
__global__ void __launch_bounds__(256) split_b_kernel(const double* __restrict__ B, long long ldb,
                                                      int K, int N, int pieces,
                                                      const int* __restrict__ ks,
                                                      unsigned char* __restrict__ out,
                                                      double* __restrict__ cb, int* bad,
                                                      const int* __restrict__ least) {
  __shared__ double buf[8][kMaxK + kMaxK / 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * 8 + warp;
  if (n >= N) return;
  if (__shfl_sync(~0u, *bad, 0) < 0) return;  // (one answer a warp; *bad stays)
  double m = 0.0;
  bool nan = false;
  for (int k = lane; k < kMaxK; k += 32) {
    const double x = k < K ? B[idx(k, n, ldb)] * pow2(-ks[k]) : 0.0;
    buf[warp][k + (k >> 3)] = x;
    m = fmax(m, fabs(x));
    nan |= x != x;
  }
  if (nan) m = __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(~0u, m, off));
  __syncwarp();
  int e;
  const bool ok = scale_exponent(m, e);
  const double per_max = ok && m > 0.0 ? 16.0 / m : 0.0;
  float sum = 0.0f;
#pragma unroll
  for (int k = lane; k < kMaxK; k += 32) sum += share_of(buf[warp][k + (k >> 3)], per_max);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(~0u, sum, off);
  if (lane == 0) {
    cb[n] = ok ? pow2(e - 70) : 0.0;
    // (*least is INT_MAX when every row of A is zero)
    const bool proven = m == 0.0 || (int)(kShare * sum) + min(*least, kShare * K) >=
                                        kShare * (K + kProof);
    if (!ok || !proven) *bad = -1;
  }
  if (!ok || 8 * lane >= pieces * BK) return;
  const double up = pow2(63 - e);
  unsigned w[2][kDigits];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = buf[warp][9 * lane + 4 * h + i];
    digit_words(x, up, w[h]);
  }
  unsigned char* const dst = out + ((size_t)(n / BN) * pieces + 8 * lane / BK) * kPieceB +
                             image_at(n % BN, 8 * lane % BK);
#pragma unroll
  for (int q = 0; q < kDigits; ++q)
    *reinterpret_cast<uint2*>(dst + q * kImageB) = make_uint2(w[0][q], w[1][q]);
}

// -------------------------------------------------------------- GEMM ----
using namespace umma;

// The products of one piece for pass P (0: weights 7 .. 4, 1: weights 3 .. 0);
// `fresh`: the pass's first piece, whose first product of a weight (i = 0)
// starts its accumulator.
template <int P>
__device__ __forceinline__ void issue_piece(uint32_t tmem, const unsigned char* a,
                                            const unsigned char* b, bool fresh) {
  constexpr int lo = P ? 0 : kHead, hi = P ? kHead - 1 : kDigits - 1;
  constexpr uint32_t idesc = idesc_i8_s32(BM, BN);
  const uint64_t ad = desc_k_plain(a, 128, 256), bd = desc_k_plain(b, 128, 256);
#pragma unroll
  for (int i = 0; i <= hi; ++i) {
    constexpr uint64_t sa = kImageA >> 4, sb = kImageB >> 4;
    const int j0 = lo > i ? lo - i : 0, j1 = hi - i;  // this digit's products
#pragma unroll
    for (int j = j0; j <= j1; ++j) {
      const uint32_t acc = tmem + (uint32_t)((i + j) * BN), more = (i == 0 && fresh) ? 0u : 1u;
      if (j0 == j1) umma_i8<kDiscard>(acc, ad + i * sa, bd + j * sb, idesc, more);
      else if (j == j0) umma_i8<kFill>(acc, ad + i * sa, bd + j * sb, idesc, more);
      else if (j < j1) umma_i8<kUse>(acc, ad + i * sa, bd + j * sb, idesc, more);
      else umma_i8<kLastUse>(acc, ad + i * sa, bd + j * sb, idesc, more);
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_i8_kernel(const unsigned char* __restrict__ a_digits, const unsigned char* __restrict__ b_digits,
               int M, int N, int pieces, double* C, long long ldc, const double* __restrict__ ra,
               const double* __restrict__ cb, int per_cta, const int* __restrict__ bad,
               int* status) {
  if (*bad < 0) return;  // (uniform over the grid)
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages];
  __shared__ __align__(8) uint64_t tfull_bar[2], tempty_bar[2], done_bar;  // by pass
  __shared__ uint32_t tmem_base_sh;
  __shared__ int failed;
  unsigned char* smem =
      reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(~0u, tid >> 5, 0);  // (uniform)
  const int tiles_m = (M + BM - 1) / BM;
  const int tiles = tiles_m * ((N + BN - 1) / BN);
  const int first = blockIdx.x * per_cta, last = min(tiles, first + per_cta);

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int d = 0; d < 2; ++d) {
      mbar_init(&tfull_bar[d], 1);
      mbar_init(&tempty_bar[d], kEpiWarps);
    }
    mbar_init(&done_bar, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;
  volatile int* const vfailed = &failed;
  auto fail = [&] {
    *vfailed = 1;
    atomicCAS(status, kOk, kDeviceTimeout);
  };

  if (warp == 0) {
    if (elect_one()) {  // copies: 48 KB a piece in the first pass, 24 KB in the second
      int g = 0;
      bool ok = true;
      for (int t = first; t < last && ok && !*vfailed; ++t) {
        const unsigned char* ap = a_digits + (size_t)(t % tiles_m) * pieces * kPieceA;
        const unsigned char* bp = b_digits + (size_t)(t / tiles_m) * pieces * kPieceB;
        for (int pc = 0; pc < 2 * pieces; ++pc, ++g) {
          const int s = g % kStages, c = pc < pieces ? pc : pc - pieces;
          const unsigned digits = pc < pieces ? kDigits : kHead;
          if (!mbar_wait(&empty_bar[s], (unsigned)((g / kStages) & 1) ^ 1u)) {  // (fresh: passes)
            ok = false;
            fail();
            break;
          }
          unsigned char* st = smem + (size_t)s * kStage;
          mbar_expect_tx(&full_bar[s], digits * (kImageA + kImageB));
          bulk_load(st, ap + (size_t)c * kPieceA, digits * kImageA, &full_bar[s]);
          bulk_load(st + kPieceA, bp + (size_t)c * kPieceB, digits * kImageB, &full_bar[s]);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {  // MMA issuer
      int g = 0, it = 0;
      bool ok = true;
      for (int t = first; t < last && ok; ++t, ++it) {
        for (int pc = 0; pc < 2 * pieces; ++pc, ++g) {
          const int s = g % kStages, pass = pc < pieces ? 0 : 1, c = pass ? pc - pieces : pc;
          // the pass's accumulators are read (c == 0), the piece is there
          if ((c == 0 && !mbar_wait(&tempty_bar[pass], (unsigned)(it & 1) ^ 1u)) ||
              !mbar_wait(&full_bar[s], (unsigned)((g / kStages) & 1))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned char* st = smem + (size_t)s * kStage;
          if (pass == 0)
            issue_piece<0>(tmem, st, st + kPieceA, c == 0);
          else
            issue_piece<1>(tmem, st, st + kPieceA, c == 0);
          umma_commit(&empty_bar[s]);  // the stage is free once these MMAs complete
          if (c == pieces - 1) umma_commit(&tfull_bar[pass]);
        }
      }
      if (!ok) fail();
      umma_commit(&done_bar);  // arrives once every issued MMA has completed
    }
  } else {  // epilogue
    const int q = warp & 3, h = (warp - 2) >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * kEpiCols);
    int it = 0;
    for (int t = first; t < last; ++t, ++it) {
      const int m0 = (t % tiles_m) * BM, n0 = (t / tiles_m) * BN;
      const int row = m0 + q * 32 + lane;
      const int col0 = n0 + h * kEpiCols;
      const bool row_ok = row < M;
      double* const crow = C + idx(row_ok ? row : 0, col0, ldc);
      double p[kEpiCols], old[kEpiCols];
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j) p[j] = 0.0;
      bool got = true;
#pragma unroll
      for (int pass = 0; pass < 2; ++pass) {
        got = got && mbar_wait(&tfull_bar[pass], (unsigned)(it & 1));
        if (!got) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int d = pass ? kHead - 1 : kDigits - 1; d >= (pass ? 0 : kHead); --d) {
          uint32_t r[16];
          tmem_ld16(lane_base + (uint32_t)(d * BN), r);
          if (d == (pass ? 0 : kHead)) {  // the pass is read: its accumulators go back
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty_bar[pass]);
          }
          // p += r 2^(8 (7 - d)): the integer as a double by its bits (2^52 +
          // 2^31 + r, the constant subtracted exactly)
          const double w = (double)(1ull << (8 * (kDigits - 1 - d)));
#pragma unroll
          for (int j = 0; j < kEpiCols; ++j) {
            const double v = __hiloint2double(0x43300000, (int)(r[j] ^ 0x80000000u)) -
                             4503601774854144.0;  // 2^52 + 2^31
            p[j] = fma(v, w, p[j]);
          }
        }
        if (pass == 0) {  // C, in flight while the second pass runs
#pragma unroll
          for (int j = 0; j < kEpiCols; ++j)
            old[j] = (row_ok && col0 + j < N) ? __ldcg(crow + (size_t)j * ldc) : 0.0;
        }
      }
      if (!got || *vfailed) {
        if (lane == 0) fail();
        break;
      }
      const double rs = row_ok ? ra[row] : 0.0;
#pragma unroll
      for (int j = 0; j < kEpiCols; ++j)
        if (row_ok && col0 + j < N) crow[(size_t)j * ldc] = fma(-p[j], rs * cb[col0 + j], old[j]);
    }
  }
  // every issued MMA has completed before the tensor memory is released
  __syncthreads();
  if (warp == 1) {
    const bool ok = mbar_wait(&done_bar, 0);
    if (!ok && lane == 0) fail();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
}

size_t al(size_t b) { return (b + 255) / 256 * 256; }
}  // namespace i8

int i8_max_k() { return i8::kMaxK; }

namespace {
size_t i8_digits_bytes(long long rows) {  // images of whole tiles (of A's size), then the scales
  const size_t tiles = (size_t)((rows + i8::BM - 1) / i8::BM);
  return tiles * i8::BM * i8::kMaxK * i8::kDigits + i8::al(sizeof(double) * rows);
}

double* scales_of(void* digits, long long rows) {
  const size_t tiles = (size_t)((rows + i8::BM - 1) / i8::BM);
  return reinterpret_cast<double*>(static_cast<char*>(digits) +
                                   tiles * i8::BM * i8::kMaxK * i8::kDigits);
}
}  // namespace

size_t i8_bytes(long long m, long long n) {
  return i8_digits_bytes(m) + i8_digits_bytes(n) + i8::al(sizeof(int) * (i8::kMaxK + 2));
}

I8Update i8_update(void* mem, long long m, long long n) {
  I8Update u;
  char* p = static_cast<char*>(mem);
  u.a_digits = p;
  u.b_digits = p + i8_digits_bytes(m);
  u.bad = reinterpret_cast<int*>(p + i8_digits_bytes(m) + i8_digits_bytes(n));
  u.least = u.bad + 1;
  u.ks = u.bad + 2;
  return u;
}

int launch_i8_split_a(const I8Update& u, int M, int K, const double* A, long long lda,
                      const double* B, long long ldb, int cols, cudaStream_t s) {
  const size_t smem = sizeof(double) * 32 * (i8::kMaxK + 1);
  if (M <= 0 || K <= 0 || K > i8::kMaxK || !ensure_smem((const void*)i8::split_a_kernel, smem))
    return kCudaFailure;
  note_launch(2);
  i8::row_scale_kernel<<<1, i8::kMaxK, 0, s>>>(B, ldb, K, std::min(cols, i8::kScaleCols), u.ks,
                                               u.bad, u.least);
  i8::split_a_kernel<<<(M + 31) / 32, 256, smem, s>>>(
      A, lda, M, K, (K + i8::BK - 1) / i8::BK, u.ks, static_cast<unsigned char*>(u.a_digits),
      scales_of(u.a_digits, M), u.bad, u.least);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

int launch_gemm_minus_i8(const I8Update& u, int M, int N, int K, const double* A, long long lda,
                         const double* B, long long ldb, double* C, long long ldc, int* status,
                         cudaStream_t s) {
  using namespace i8;
  if (M <= 0 || N <= 0 || K <= 0) return kOk;
  if (K > kMaxK || !ensure_smem((const void*)gemm_i8_kernel, kSmem)) return kCudaFailure;
  const int pieces = (K + BK - 1) / BK;
  note_launch(2);
  split_b_kernel<<<(N + 7) / 8, 256, 0, s>>>(B, ldb, K, N, pieces, u.ks,
                                             static_cast<unsigned char*>(u.b_digits),
                                             scales_of(u.b_digits, N), u.bad, u.least);
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  // two tiles a CTA: more of them keep the tensor path busier (8192 x 8192 alone:
  // 4 a CTA 666 us, all of an SM's 598), fewer give the SMs back sooner to the
  // panels of the next block, which wait for whole SMs (LU of n = 8192, 2 / 4 / 8
  // a CTA: 29.3 / 30.0 / 30.8 ms; n = 12000: 52.5 / 54.1 / 56.1)
  const int per = std::max(1, std::min(2, tiles / (2 * sm_count())));
  gemm_i8_kernel<<<(tiles + per - 1) / per, kThreads, kSmem, s>>>(
      static_cast<const unsigned char*>(u.a_digits), static_cast<const unsigned char*>(u.b_digits),
      M, N, pieces, C, ldc, scales_of(u.a_digits, M), scales_of(u.b_digits, N), per, u.bad, status);
  // operands outside the scheme: the FP64 kernel, which returns unless *bad < 0
  launch_gemm_minus_if(M, N, K, A, lda, B, ldb, C, ldc, s, u.bad);
  return cudaGetLastError() == cudaSuccess ? kOk : kCudaFailure;
}

}  // namespace dp
