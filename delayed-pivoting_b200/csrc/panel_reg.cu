// Panel factorisation on one thread-block cluster with the sub-panel in
// registers (panels of up to 1024 rows per CTA).
//
// Same contract and semantics as panel_cluster_kernel
// (delayed_lu/delayed_dgetrf.cpp:164-240: column partial-pivot search with
// first-index ties and NaN never winning, acceptance |alpha| > threshold,
// row swap, scaling by the reciprocal pivot, rank-1 update, stop at the first
// column without an acceptable pivot), with less work per column:
//   * every thread holds its rows' 8-column sub-panel slice in registers
//     (RPT rows per thread), so the swap, scaling and rank-1 update of a step
//     touch no shared memory;
//   * a step pushes one ~100-byte slot per CTA to every CTA of the cluster
//     (its candidate: magnitude, row, runner-up, reciprocal, source row and
//     the row's 8 sub-panel values; the owner of row k also pushes row k's
//     slice), then one hardware cluster barrier; every CTA then picks the
//     same winner and updates its own registers;
//   * the rest of each row (the finished L columns left of the sub-panel and
//     the columns right of it) does not change during a sub-panel, so rows
//     are moved there only at the sub-panel's end: every CTA replays the
//     sub-panel's swaps into a composite source map and pulls the content of
//     its moved rows - and the pivot rows for U12 = L11^{-1} A12 - from the
//     owning CTAs' shared memory (phase A), a second cluster barrier, then
//     writes them in place (phase B) and applies the rank-8 update of the
//     columns right of the sub-panel.
// Push buffers are indexed by step parity: a slot is written again at step s +
// 2, which every CTA reaches only through the barrier of step s + 1, passed by
// every reader of step s.  The waits for a step's slots are bounded; a thread
// whose wait runs out records the status and leaves with its whole CTA at the
// next CTA barrier.
#include <cooperative_groups.h>

#include "dp_device.cuh"
#include "dp_kernels.h"
#include "panel_argmax.cuh"

namespace cg = cooperative_groups;

namespace dp {

namespace {

using panel::LocalBest;
using panel::offer;
using panel::warp_best;
using panel::warp_lb;
using panel::warp_max_pos;

constexpr int kMaxW = 16;    // most warps of a CTA
constexpr int kS = 8;        // sub-panel width
constexpr int kMaxC = 16;    // largest cluster

// One CTA's candidate (or row k) as pushed to every CTA.
struct __align__(16) Slot {
  double val;    // magnitude (>= 0)
  double sec;    // runner-up magnitude among the CTA's rows
  double inv;    // reciprocal of the candidate's entry in the current column
  int row;       // global row, -1 when the CTA has no candidate
  int orig;      // source row of its content (for the swap lists)
  double v[kS];  // the row over the sub-panel's columns
};

constexpr int kSlotChunks = (int)(sizeof(Slot) / sizeof(uint4));
static_assert(sizeof(Slot) % sizeof(uint4) == 0, "slots travel in 16-byte stores");

// offer() that also keeps the signed entry of the best row, whose reciprocal
// is then taken before the warp reduction instead of after it.
__device__ __forceinline__ void offer_x(LocalBest& b, double& bx, double x, int r) {
  const double v = fabs(x);
  if (v > b.val) {
    b.sec = b.val;
    b.val = v;
    b.row = r;
    bx = x;
  } else if (v > b.sec) {
    b.sec = v;
  }
}

struct Layout {
  double* sm;     // [w][RP] the panel slice
  Slot* slots;    // [2][kMaxC] candidates, by step parity and CTA rank
  Slot* kslot;    // [2] row k, by step parity
  Slot* stage;    // [kMaxW] per-warp candidates, then [1] row k
  double* psave;  // [kS][W1] the sub-panel's pivot rows
  double* tmp;    // [2 kS][W1] pulled content of moved rows (by map entry)
  int* orig;      // [R] source row of each local row
  int* plist;     // [kS][2] (k, pivot row) of the sub-panel's steps
  int* pivs;      // [w] pivot rows (rank 0)
  int* own;       // [1 + 3 * 2 kS]: count, then (local row, source owner, source
                  // local row) of the moved rows this CTA owns
  int* ksrc;      // [2 kS]: (owner, local row) of the content of each step's row k
  unsigned long long* xbar;  // [2] exchange barriers, by step parity
};

__host__ __device__ inline size_t reg_align16(size_t bytes) { return (bytes + 15) & ~(size_t)15; }

__host__ __device__ inline size_t reg_layout(unsigned char* base, int w, int R, Layout* L) {
  const size_t rp = (size_t)(R | 1), w1 = (size_t)w + 1;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = base ? base + off : nullptr;
    off += reg_align16(bytes);
    return p;
  };
  unsigned char* sm = take(sizeof(double) * (size_t)w * rp);
  unsigned char* slots = take(sizeof(Slot) * 2 * kMaxC);
  unsigned char* kslot = take(sizeof(Slot) * 2);
  unsigned char* stage = take(sizeof(Slot) * (kMaxW + 1));
  unsigned char* psave = take(sizeof(double) * kS * w1);
  unsigned char* tmp = take(sizeof(double) * 2 * kS * w1);  // row q: map entry q
  unsigned char* orig = take(sizeof(int) * (size_t)R);
  unsigned char* plist = take(sizeof(int) * 2 * kS);
  unsigned char* pivs = take(sizeof(int) * (size_t)w);
  unsigned char* own = take(sizeof(int) * (1 + 6 * kS));
  unsigned char* ksrc = take(sizeof(int) * 2 * kS);
  unsigned char* xbar = take(sizeof(unsigned long long) * 2);
  if (L) {
    L->sm = reinterpret_cast<double*>(sm);
    L->slots = reinterpret_cast<Slot*>(slots);
    L->kslot = reinterpret_cast<Slot*>(kslot);
    L->stage = reinterpret_cast<Slot*>(stage);
    L->psave = reinterpret_cast<double*>(psave);
    L->tmp = reinterpret_cast<double*>(tmp);
    L->orig = reinterpret_cast<int*>(orig);
    L->plist = reinterpret_cast<int*>(plist);
    L->pivs = reinterpret_cast<int*>(pivs);
    L->own = reinterpret_cast<int*>(own);
    L->ksrc = reinterpret_cast<int*>(ksrc);
    L->xbar = reinterpret_cast<unsigned long long*>(xbar);
  }
  return off;
}

}  // namespace

template <int kT, int RPT>
__global__ void __launch_bounds__(kT, 1) panel_reg_kernel(PanelParams p) {
  constexpr int kW = kT / 32;
  after_previous_kernel();
  // Every CTA reads the same word before any barrier or state write (a stop
  // is recorded only by an earlier kernel), so all of them leave together.
  if (p.gated && p.state->stop_k >= 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int rank = (int)cluster.block_rank();
  const int w = p.end - p.begin;
  const int W1 = w + 1;
  const int R = p.rows_per_cta;
  const int RP = R | 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long row0 = (long long)p.begin + (long long)rank * R;
  const int rows_here = (int)max(0LL, min((long long)R, (long long)p.m - row0));
  Layout S;
  reg_layout(smem_raw, w, R, &S);
  double* const sm = S.sm;
  int* const orig = S.orig;

  // the slice arrives by asynchronous copies, all in flight at once
  for (int c = 0; c < w; ++c) {
    const double* src = p.a + idx(row0, p.begin + c, p.lda);
    for (int r = tid; r < rows_here; r += kT) panel::cp_async8(sm + c * RP + r, src + r);
  }
  for (int r = tid; r < rows_here; r += kT) orig[r] = (int)(row0 + r);
  panel::cp_async_wait_all();
  if (rank == 0 && tid == 0) {
    p.state->stop_k = -1;
    p.state->swap_count = 0;
    p.state->block_changed = 0;
  }
  const unsigned xbar0 = panel::smem_addr(S.xbar);
  if (tid == 0) {
    panel::xbar_init(xbar0);
    panel::xbar_init(xbar0 + 8);
    panel::xbar_init_fence();
  }
  // every CTA's slice loaded and exchange barriers initialised before any
  // peer reads the one or writes to the other
  cluster.sync();

  LocalBest mine{0.0, -1, 0, 0.0};
  double mine_x = 0.0;  // signed entry of the candidate

  // Near-tie record (rank 0, warp 0, recorded by its lane 0): a decision's
  // runner-up is reduced and tallied while the next exchange is awaited
  DecisionTally tally;
  long long t_k = -1;  // the decision to record, -1 when none
  double t_best = 0.0, t_lane = 0.0;
  auto record = [&] {
    if (rank == 0 && warp == 0 && t_k >= 0) {
      const double second = warp_max_pos(t_lane);
      tally.note(t_k, t_best, second);  // (alike in every lane; one is flushed)
      t_k = -1;
    }
  };
  bool stopped = false, timed_out = false, late = false;
  int done = 0;  // steps executed
  bool pending = false;  // a cluster_arrive() awaits its cluster_wait()
  for (int base = 0; base < w && !stopped; base += kS) {
    const int send = min(base + kS, w);
    double x[RPT][kS];  // this thread's rows over the sub-panel's columns
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + i * kT;
#pragma unroll
      for (int t = 0; t < kS; ++t)
        x[i][t] = (r < rows_here && base + t < w) ? sm[(base + t) * RP + r] : 0.0;
    }
    // the candidate of the sub-panel's first column
    mine = LocalBest{0.0, -1, 0, 0.0};
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + i * kT;
      if (r < rows_here && row0 + r >= (long long)p.begin + base) offer_x(mine, mine_x, x[i][0], r);
    }
    int kd = send - base;  // steps executed in this sub-panel

#pragma unroll
    for (int j = 0; j < kS; ++j) {
      if (base + j >= w) break;
      const int s = base + j;
      const long long k = (long long)p.begin + s;
      const int par = s & 1;
      const bool positioned = (s == 0) && p.positioned;
      const int kl = (int)(k - row0);
      const bool own_k = kl >= 0 && kl < rows_here;

      const unsigned xb = xbar0 + 8u * (unsigned)par;
      if (tid == 0) panel::xbar_expect(xb, (unsigned)((C + 1) * sizeof(Slot)));

      // 1. this CTA's candidate: per-warp winners staged with their slices
      if (positioned) {
        mine = LocalBest{0.0, -1, 0, 0.0};
        if (own_k && tid == kl % kT) {
          mine = LocalBest{__longlong_as_double(0x7ff0000000000000ll), kl, 0, 0.0};
          mine_x = sm[kl];  // step 0: column 0 in shared memory is still current
        }
      }
      const double mine_inv = mine.row >= 0 ? 1.0 / mine_x : 0.0;
      const LocalBest wb = warp_lb(mine);
      if (wb.row >= 0 && tid == wb.row % kT) {
        Slot& st = S.stage[warp];
        const int wi = wb.row / kT;
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i == wi) {
#pragma unroll
            for (int t = 0; t < kS; ++t) st.v[t] = x[i][t];
          }
        st.inv = mine_inv;
        st.val = wb.val;
        st.sec = wb.sec;
        st.row = (int)(row0 + wb.row);
        st.orig = orig[wb.row];
      } else if (wb.row < 0 && lane == 0) {
        Slot& st = S.stage[warp];
        st.val = 0.0;
        st.sec = wb.sec;
        st.inv = 0.0;
        st.row = -1;
        st.orig = -1;
      }
      if (own_k && tid == kl % kT) {
        Slot& st = S.stage[kMaxW];
        const int ki = kl / kT;
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i == ki) {
#pragma unroll
            for (int t = 0; t < kS; ++t) st.v[t] = x[i][t];
          }
        st.orig = orig[kl];
        st.row = (int)k;
      }
      // (a wait of the step before that ran out ends every thread here)
      if (__syncthreads_or(late)) {
        timed_out = stopped = true;
        kd = 0;
        break;
      }
      // 2. the CTA's winner among the warps, pushed to every CTA (warp 0 alone:
      //    the other warps leave the SM's reduction unit to it)
      if (warp == 0) {
        const Slot* cs = S.stage + (lane & (kW - 1));
        const bool have = lane < kW && cs->row >= 0;
        const double v = cs->val, sc = cs->sec;
        double bv;
        int brow;
        warp_best(have ? v : 0.0, have ? cs->row : 0x7fffffff, bv, brow);
        const bool won = have && cs->row == brow;
        const int wsel = max(0, __ffs(__ballot_sync(0xffffffffu, won)) - 1);
        const double bsec = warp_max_pos(lane < kW ? (won || !have ? sc : v) : 0.0);
        if (lane < C) {
          uint4 c[kSlotChunks];
          const uint4* src = reinterpret_cast<const uint4*>(S.stage + wsel);
#pragma unroll
          for (int i = 0; i < kSlotChunks; ++i) c[i] = src[i];
          // (a warp without a candidate staged magnitude 0, row -1, reciprocal 0)
          const unsigned long long sb = (unsigned long long)__double_as_longlong(bsec);
          c[0].z = (unsigned)sb;
          c[0].w = (unsigned)(sb >> 32);
          const unsigned dst = panel::peer_addr(panel::smem_addr(S.slots + par * kMaxC + rank), lane);
          const unsigned bar = panel::peer_addr(xb, lane);
#pragma unroll
          for (int i = 0; i < kSlotChunks; ++i) panel::st_async16(dst + 16u * i, c[i], bar);
        }
      } else if (warp == 1 && own_k && lane < C) {
        const uint4* src = reinterpret_cast<const uint4*>(S.stage + kMaxW);
        const unsigned dst = panel::peer_addr(panel::smem_addr(S.kslot + par), lane);
        const unsigned bar = panel::peer_addr(xb, lane);
#pragma unroll
        for (int i = 0; i < kSlotChunks; ++i) panel::st_async16(dst + 16u * i, src[i], bar);
      }
      record();
      // every CTA's slot and row k's slice have arrived (use s >> 1 of this
      // parity's barrier).  No CTA barrier here: the stage is read before its
      // CTA's slot is pushed, and a slot buffer is written again only after
      // every thread has passed the next step's barrier.  A wait that runs out
      // goes on with stale slots (used for values and in-range compares only)
      // to the next barrier, where all threads leave together
      if (!panel::xbar_wait(xb, (unsigned)(s >> 1) & 1u)) {
        late = true;
        p.state->status = kDeviceTimeout;
      }

      // 3. same decision everywhere (rows carry their slot in the low bits: the
      //    smallest key is the smallest row, and names the winner's slot)
      int wslot = -1;
      double wval = 0.0;
      {
        const Slot* cs = S.slots + par * kMaxC + (lane < C ? lane : 0);
        const bool have = lane < C && cs->row >= 0;
        const double v = lane < C ? cs->val : 0.0;
        const unsigned long long u = (unsigned long long)__double_as_longlong(have ? v : 0.0);
        const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
        const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
        const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
        const bool top = have && hi == mhi && lo == mlo;
        const unsigned key = __reduce_min_sync(
            0xffffffffu, top ? ((unsigned)(cs->row - p.begin) << 4) | (unsigned)lane : 0xffffffffu);
        if (key != 0xffffffffu) {
          wslot = (int)(key & 15u);
          wval = __longlong_as_double((long long)(((unsigned long long)mhi << 32) | mlo));
        }
        if (rank == 0 && warp == 0 && !positioned) {
          t_k = k;
          t_best = wval;
          t_lane = lane < C ? (lane == wslot || !have ? cs->sec : v) : 0.0;
        }
      }
      const bool stop = !positioned && !(wslot >= 0 && wval > p.threshold);
      if (stop) {
        // (stale slots may stop some threads only: they meet the others, who
        // are at the next step's barrier, and all leave)
        stopped = true;
        kd = j;
        if (__syncthreads_or(late)) {
          timed_out = true;
          kd = 0;
        } else if (rank == 0 && tid == 0) {
          p.state->stop_k = (int)k;
        }
        break;
      }
      const Slot& ws = S.slots[par * kMaxC + wslot];
      const long long prow = ws.row;
      if (tid == 0) {
        // (to memory at the end: a store on its way would hold up every release
        // of the cluster barrier, about 1500 cycles a sub-panel)
        S.pivs[s] = (int)prow;
        S.plist[2 * j] = (int)k;
        S.plist[2 * j + 1] = (int)prow;
      }
      if (tid < kS && base + tid < w) S.psave[j * W1 + base + tid] = ws.v[tid];
      double pv[kS];
#pragma unroll
      for (int t = 0; t < kS; ++t) pv[t] = ws.v[t];
      const double inv = ws.inv;

      // 4. swap: row k takes the pivot row, the pivot row's place row k
      const int pl = (int)(prow - row0);
      const bool swap_p = pl >= 0 && pl < rows_here && prow != k;
      if (own_k && tid == kl % kT) {
        const int ki = kl / kT;
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i == ki) {
#pragma unroll
            for (int t = 0; t < kS; ++t) x[i][t] = pv[t];
          }
        orig[kl] = ws.orig;
      }
      if (swap_p && tid == pl % kT) {
        const Slot& kr = S.kslot[par];
        const int pi = pl / kT;
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i == pi) {
#pragma unroll
            for (int t = 0; t < kS; ++t) x[i][t] = kr.v[t];
          }
        orig[pl] = kr.orig;
      }

      // 5. scale and update the rows below k; next column's candidate
      mine = LocalBest{0.0, -1, 0, 0.0};
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + i * kT;
        if (r >= rows_here || row0 + r <= k) continue;
        const double l = x[i][j] * inv;
        x[i][j] = l;
#pragma unroll
        for (int t = j + 1; t < kS; ++t) x[i][t] = fma(-l, pv[t], x[i][t]);
        if (j + 1 < kS && s + 1 < send) offer_x(mine, mine_x, x[i][j + 1 < kS ? j + 1 : 0], r);
      }
    }

    // ---- end of the sub-panel: kd steps executed at [base, base + kd) ----
    done = base + kd;
    if (kd == 0) break;  // stopped at its first step: nothing moved
    // a. the register slices back to shared memory
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + i * kT;
      if (r < rows_here) {
#pragma unroll
        for (int t = 0; t < kS; ++t)
          if (base + t < w) sm[(base + t) * RP + r] = x[i][t];
      }
    }
    // b. composite source map of the sub-panel's swaps (the same everywhere):
    //    lane q of warp 0 takes position k_q (q < kd) or p_{q - kd} and traces
    //    it back through the swaps to the row whose content it holds now.
    //    Kept: where the content of each k_q is (the sub-panel's pivot rows,
    //    for U12) and, compacted by a ballot, the moved positions this CTA
    //    owns (a pivot row that is also a later step's row k once), each with
    //    its source's owner and local row
    if (warp == 0) {
      __syncwarp();  // the steps' list is lane 0's
      const bool on = lane < 2 * kd;
      int2 sw[kS];  // (k, pivot row) of the steps
#pragma unroll
      for (int t = 0; t < kS; ++t)
        sw[t] = t < kd ? *reinterpret_cast<const int2*>(S.plist + 2 * t) : make_int2(-1, -1);
      int x = on ? S.plist[lane < kd ? 2 * lane : 2 * (lane - kd) + 1] : -2 - lane;
      const int pos = x;
#pragma unroll
      for (int t = kS - 1; t >= 0; --t) x = x == sw[t].x ? sw[t].y : (x == sw[t].y ? sw[t].x : x);
      const int so = on ? (int)((x - p.begin) / R) : 0;
      const int sl = on ? (int)(x - p.begin - (long long)so * R) : 0;
      if (lane < kd) {
        S.ksrc[2 * lane] = so;
        S.ksrc[2 * lane + 1] = sl;
      }
      // the first occurrence of each position
      const bool first = __ffs(__match_any_sync(0xffffffffu, pos)) - 1 == lane;
      const bool keep = on && first && x != pos && pos >= row0 && pos < row0 + rows_here;
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int at = __popc(bal & ((1u << lane) - 1u));
        S.own[1 + 3 * at] = (int)(pos - row0);
        S.own[2 + 3 * at] = so;
        S.own[3 + 3 * at] = sl;
      }
      if (lane == 0) S.own[0] = __popc(bal);
    }
    if (__syncthreads_or(late)) {
      timed_out = stopped = true;
      break;
    }
    const int nown = S.own[0];
    // the owners' writes of the previous sub-panel end are visible
    if (pending) {
      panel::cluster_wait();
      pending = false;
    }
    // c. phase A: the moved rows of this CTA (into tmp, row q for own entry
    //    q) and the pivot rows' columns right of the sub-panel (into psave),
    //    read from their owners' shared memory: a thread takes a column and
    //    every (kT / 64)-th row, four independent loads in flight
    constexpr int kGrp = kT / 64;
    const int cl = tid & 63, grp = tid >> 6;
    const int nfetch = nown + (send < w ? kd : 0);
    for (int c = cl; c < w; c += 64) {
      if (c >= base && c < send) continue;
      for (int q0 = grp; q0 < nfetch; q0 += 4 * kGrp) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int q = q0 + u * kGrp;
          if (q >= nfetch || (q >= nown && c < send)) continue;
          const int* at = q < nown ? S.own + 2 + 3 * q : S.ksrc + 2 * (q - nown);
          v[u] = cluster.map_shared_rank(sm, at[0])[c * RP + at[1]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int q = q0 + u * kGrp;
          if (q >= nfetch || (q >= nown && c < send)) continue;
          (q < nown ? S.tmp + q * W1 : S.psave + (q - nown) * W1)[c] = v[u];
        }
      }
    }
    cluster.sync();  // every CTA has read what it needs before anyone overwrites
    // d. phase B: moved rows take their sources' content
    for (int c = cl; c < w; c += 64)
      if (c < base || c >= send)
        for (int q = grp; q < nown; q += kGrp) sm[c * RP + S.own[1 + 3 * q]] = S.tmp[q * W1 + c];
    if (send >= w) break;  // no columns right of the sub-panel
    __syncthreads();       // psave and the moved rows complete
    // e. U12 = L11^{-1} A12 of the sub-panel, one column per thread, a step's
    //    multiples subtracted from all later rows before the next step (the
    //    dependent chain is kd long)
    const long long first = (long long)p.begin + base;  // global row of the first pivot
    for (int c = send + tid; c < w; c += kT) {
      double u[kS];
#pragma unroll
      for (int q = 0; q < kS; ++q) u[q] = q < kd ? S.psave[q * W1 + c] : 0.0;
#pragma unroll
      for (int t = 0; t < kS - 1; ++t)
#pragma unroll
        for (int q = t + 1; q < kS; ++q)
          if (q < kd) u[q] = fma(-S.psave[q * W1 + base + t], u[t], u[q]);
#pragma unroll
      for (int q = 0; q < kS; ++q)
        if (q < kd) {
          if (q > 0) S.psave[q * W1 + c] = u[q];
          // the solved rows to the pivot rows of this CTA
          const long long g = first + q - row0;
          if (g >= 0 && g < rows_here) sm[c * RP + (int)g] = u[q];
        }
    }
    __syncthreads();
    // f. rank-kd update of the rows below the sub-panel's pivots on the FP64
    //    tensor path (mma.sync.m16n8k4, the kd <= 8 steps as two k4 steps):
    //    warp w takes rows [32 w + 256 i, + 32) in 16 x 8 tiles over the
    //    columns [send, w), C read from and written to shared memory; rows
    //    above the sub-panel's last pivot or beyond the CTA's keep their
    //    values.  Then the next sub-panel's first candidate.
    {
      const double* __restrict__ ps = S.psave;
      const int g = lane >> 2, t4 = lane & 3;
      const int lim = (int)max(0LL, min((long long)rows_here, first + kd - row0));
      const int ncol = w - send;
#pragma unroll
      for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          const int rb = warp * 32 + i * kT + mt * 16;
          if (rb >= rows_here || rb + 16 <= lim) continue;  // (warp-uniform)
          const bool ok0 = rb + g < rows_here, ok1 = rb + g + 8 < rows_here;
          double a[2][2];
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            const int k = 4 * ks + t4;
            a[ks][0] = (k < kd && ok0) ? -sm[(base + k) * RP + rb + g] : 0.0;
            a[ks][1] = (k < kd && ok1) ? -sm[(base + k) * RP + rb + g + 8] : 0.0;
          }
          const bool st0 = ok0 && rb + g >= lim, st1 = ok1 && rb + g + 8 >= lim;
          for (int c0 = 0; c0 < ncol; c0 += 8) {
            double b[2];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
              const int k = 4 * ks + t4;
              b[ks] = (k < kd && c0 + g < ncol) ? ps[k * W1 + send + c0 + g] : 0.0;
            }
            const int ca = send + c0 + 2 * t4;  // this lane's columns ca, ca + 1
            double c[4];
            c[0] = (ok0 && ca < w) ? sm[ca * RP + rb + g] : 0.0;
            c[1] = (ok0 && ca + 1 < w) ? sm[(ca + 1) * RP + rb + g] : 0.0;
            c[2] = (ok1 && ca < w) ? sm[ca * RP + rb + g + 8] : 0.0;
            c[3] = (ok1 && ca + 1 < w) ? sm[(ca + 1) * RP + rb + g + 8] : 0.0;
            panel::mma_f64(c, a[0][0], a[0][1], b[0]);
            panel::mma_f64(c, a[1][0], a[1][1], b[1]);
            if (st0 && ca < w) sm[ca * RP + rb + g] = c[0];
            if (st0 && ca + 1 < w) sm[(ca + 1) * RP + rb + g] = c[1];
            if (st1 && ca < w) sm[ca * RP + rb + g + 8] = c[2];
            if (st1 && ca + 1 < w) sm[(ca + 1) * RP + rb + g + 8] = c[3];
          }
        }
    }
    __syncthreads();  // every warp's tiles are stored: the next columns are final
    // released to the readers of the next sub-panel end (phase A); the
    // steps in between exchange through the transaction barriers alone
    panel::cluster_arrive();
    pending = true;
  }
  // No CTA may exit while a peer could still read its shared memory, and
  // rows were written by other threads than those writing them back.
  if (pending)
    panel::cluster_wait();
  else
    cluster.sync();
  if (timed_out) return;
  record();
  if (rank == 0) {
    if (tid == 0) tally.flush(p.state);
    for (int t = tid + (p.positioned ? 1 : 0); t < done; t += kT) p.ipiv[p.begin + t] = S.pivs[t];
  }

#pragma unroll 4
  for (int c = 0; c < w; ++c) {
    double* dst = p.a + idx(row0, p.begin + c, p.lda);
    for (int r = tid; r < rows_here; r += kT) dst[r] = sm[c * RP + r];
  }
  // Swap lists: whole warps walk the rows together, so that the moved rows
  // below the block take their slots with one atomic per warp.
  int changed = 0;
  for (int r0w = warp * 32; r0w < rows_here; r0w += kT) {
    const int r = r0w + lane;
    const long long g = row0 + r;
    const int src = r < rows_here ? orig[r] : (int)g;
    if (r < rows_here && g < p.end) {
      p.swap_block[g - p.begin] = src;
      changed += src != (int)g;
    }
    const bool moved = r < rows_here && g >= p.end && src != (int)g;
    const unsigned bal = __ballot_sync(0xffffffffu, moved);
    if (bal) {
      int slot = 0;
      if (lane == 0) slot = atomicAdd(&p.state->swap_count, __popc(bal));
      slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(bal & ((1u << lane) - 1u));
      if (moved) {
        p.swap_extra[2 * slot + 0] = (int)g;
        p.swap_extra[2 * slot + 1] = src;
      }
    }
  }
  changed = __reduce_add_sync(0xffffffffu, changed);
  if (lane == 0 && changed) atomicAdd(&p.state->block_changed, changed);
}

size_t panel_reg_smem_bytes(int w, int rows_per_cta) {
  return reg_layout(nullptr, w, rows_per_cta, nullptr);
}

// Rows per CTA and threads: a thread a row up to 512 rows, two up to 1024.  LU,
// ms, a thread a row up to 512 / 256 threads of two rows there: n = 8192
// 27.5 / 28.0, n = 16384 94.8 / 95.7.  Above 512 rows the shared-memory panel
// (panel_kernel 3) was as fast (n = 16384 97.1 with it, before the changes
// below).  What a column costs is a chain of about 3600 cycles (C = 16, 256
// rows a CTA): stage the warps' winners 850, CTA winner and push 400, wait 520,
// decide 460, swap and update 230, an eighth of the sub-panel's end 1100.  It
// was 3900 while every warp reduced the CTA's winner and every thread the
// runner-ups, the end's rows were fetched in two rounds with a division per
// element, and each step's pivot was stored to memory.
int panel_reg_max_rows() { return 1024; }
int panel_reg_threads(int rows_per_cta) { return rows_per_cta <= 256 ? 256 : 512; }

const void* panel_reg_kernel_for(int rows_per_cta) {
  if (rows_per_cta <= 256) return (const void*)panel_reg_kernel<256, 1>;
  if (rows_per_cta <= 512) return (const void*)panel_reg_kernel<512, 1>;
  if (rows_per_cta <= 1024) return (const void*)panel_reg_kernel<512, 2>;
  return nullptr;
}

}  // namespace dp
