// CUDA kernels of the gstb engine, sm_100a.
//
// Hot path of one query (the reference's DPBF_GPU, code/GPUGST/src/DPQ.cu:275-624,
// and DPBF_gpu, code/D-GPUGST/src/DPQ.cu:149-269, re-designed).  Every round is
//   k_small    one cluster: the control step (one thread per query slot
//              advances the query's state machine: distance rounds -> tour
//              tables -> DP seed -> DP rounds -> extraction, and the round's
//              work description is written), then, while rounds are small,
//              the rounds themselves;
//   k_light    warp tasks: near-far splits, seeds, tour tables, extraction,
//              distance items (a vertex with its pending groups; the arcs of
//              a task's items are relaxed as one flat list by the whole warp:
//              multi-source relax, replacing dis0_init_1, DPQ.cu:241-271) and
//              DP items, one warp per state: best update from complement /
//              one-label completion, lower-bound prune, grow along the
//              weight-sorted adjacency, merge with every disjoint subset at
//              the vertex (replaces Relax, DPQ.cu:73-172 and
//              D-GPUGST/src/DPQ.cu:62-126);
//   k_heavy    the arc chunks k_light handed over in the same round (hub
//              vertices of distance items, high-degree DP states), then
//              lower-bound table rows;
//   split      near-far bucketing: far items whose cost entered the new
//              window move to the near list
//   tour       group-to-group distances and tour tables (host DP at
//              DPQ.cu:409-483, re-done on device by a warp per starting group)
//   seeds      members at distance 0 (DPQ.cu:359-368); cost-0 states of every
//              subset of a member's group mask (DPQ.cu:341-358)
//   extract    follow parents from the best full state into a tree (the
//              reference's extraction, CPUNONHOP.h:390-432 / CPUHOP.h:234-259,
//              which its GPU path leaves commented out)
#include "gst_device.cuh"

// Round kernels take their tasks by work stealing (1) or by static striding
// (0, the default: on the 170k-vertex power-law workload stealing changed the
// order of the label-correcting distance work enough to add 11% more arc
// relaxations and ran 10% slower).
#ifndef GSTB_STEAL
#define GSTB_STEAL 0
#endif

namespace gstb {

__device__ __forceinline__ uint32_t warp_sum(uint32_t x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
  return x;
}

// Bound-table entries: LB_INF marks a completion that is impossible (a group
// out of reach); finite bounds saturate at LB_INF - 1, which stays a valid
// lower bound.
constexpr uint32_t LB_INF = 0xFFFFu;
__device__ __forceinline__ bool lb_ok(uint32_t cost, uint32_t lb, uint32_t best) {
  return lb != LB_INF && (unsigned long long)cost + lb <= best;
}

// Statistics of the query a warp is working for, kept in shared memory by
// lane 0 and added to the query's counters only when the warp moves to
// another query and at kernel end (one atomic per event would queue on the
// query's control block).
struct WarpStat {
  QCtl* cur;
  uint32_t v[12];
};

__device__ __forceinline__ void ws_init(WarpStat& w) {
  w.cur = nullptr;
#pragma unroll
  for (int i = 0; i < 12; i++) w.v[i] = 0u;
}

__device__ __forceinline__ void ws_flush(WarpStat& w) {
  if (w.cur)
    for (int i = 0; i < 12; i++)
      if (w.v[i]) atomicAdd(&w.cur->stat[i], (unsigned long long)w.v[i]);
#pragma unroll
  for (int i = 0; i < 12; i++) w.v[i] = 0u;
}

// Lane 0 only.
__device__ __forceinline__ void ws_add(WarpStat& w, QCtl* c, int idx, uint32_t val) {
  if (w.cur != c) {
    ws_flush(w);
    w.cur = c;
  }
  w.v[idx] += val;
}

// Warp-local staging of list appends.  The near-out and far entries of one
// query collect in shared memory and reach the global lists in bulk: every
// warp working for a query appends to the same two counters, and one counter
// atomic per flush instead of one per warp step keeps them from queueing.
constexpr uint32_t WBUF = 256;
struct WarpBuf {
  const QDev* q;
  uint32_t nN, nF;
  uint32_t it[2 * WBUF];  // near-out entries, then far ones (tour_warp's scratch between uses)
};

__device__ __forceinline__ void wb_init(WarpBuf& b) {  // lane 0
  b.q = nullptr;
  b.nN = b.nF = 0u;
}

// Every lane of the warp calls it.
__device__ __forceinline__ void wb_flush(WarpBuf& b, uint32_t lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  __syncwarp();
  const QDev* q = b.q;
  const uint32_t nN = b.nN, nF = b.nF;
  if (q != nullptr && (nN | nF) != 0u) {
    uint32_t bN = 0, bF = 0;
    if (lane == 0) {
      if (nN) bN = atomicAdd(&q->ctl->n_near, nN);
      if (nF) bF = atomicAdd(&q->ctl->n_far, nF);
    }
    bN = __shfl_sync(FULL, bN, 0);
    bF = __shfl_sync(FULL, bF, 0);
    uint32_t* outN = q->qbuf[q->out_idx];
    uint32_t* outF = q->qbuf[q->far_idx];
    const uint32_t cap = q->cap;
    bool ovf = false;
    for (uint32_t i = lane; i < nN; i += 32u) {
      if (bN + i < cap)
        outN[bN + i] = b.it[i];
      else
        ovf = true;
    }
    for (uint32_t i = lane; i < nF; i += 32u) {
      if (bF + i < cap)
        outF[bF + i] = b.it[WBUF + i];
      else
        ovf = true;
    }
    if (__any_sync(FULL, ovf) && lane == 0) atomicExch(&q->ctl->overflow, 1u);
  }
  __syncwarp();
  if (lane == 0) b.nN = b.nF = 0u;
  __syncwarp();
}

// Append up to U items per lane to the near-out and far lists of query q
// through the warp's buffer.  Every lane of the warp calls it; returns this
// lane's number of appended items.
template <int U>
__device__ __forceinline__ uint32_t append_lists(const bool (&takeN)[U], const bool (&takeF)[U],
                                                 const uint32_t (&item)[U], const QDev& q, uint32_t lane,
                                                 WarpBuf& b) {
  const unsigned FULL = 0xFFFFFFFFu;
  uint32_t cN = 0, cF = 0;
#pragma unroll
  for (int u = 0; u < U; u++) {
    cN += takeN[u] ? 1u : 0u;
    cF += takeF[u] ? 1u : 0u;
  }
  if (!__any_sync(FULL, (cN | cF) != 0u)) return 0u;
  uint32_t xN = cN, xF = cF;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t yN = __shfl_up_sync(FULL, xN, o), yF = __shfl_up_sync(FULL, xF, o);
    if (lane >= (uint32_t)o) {
      xN += yN;
      xF += yF;
    }
  }
  const uint32_t totN = __shfl_sync(FULL, xN, 31), totF = __shfl_sync(FULL, xF, 31);
  __syncwarp();
  if (b.q != &q || b.nN + totN > WBUF || b.nF + totF > WBUF) {
    wb_flush(b, lane);
    if (lane == 0) b.q = &q;
    __syncwarp();
  }
  const uint32_t oN = b.nN, oF = b.nF;
  uint32_t pN = oN + xN - cN, pF = oF + xF - cF;
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (takeN[u]) b.it[pN++] = item[u];
    if (takeF[u]) b.it[WBUF + pF++] = item[u];
  }
  __syncwarp();
  if (lane == 0) {
    b.nN = oN + totN;
    b.nF = oF + totF;
  }
  __syncwarp();
  return cN + cF;
}

// Enqueue of DP state s at `cost`: the near list when the cost is inside the
// current window, the far list otherwise; a flag bit per state and list
// keeps each list free of duplicates (near entries carry the next round's
// parity).  Every lane calls it (want may be false); returns 1 if this lane
// enqueued.
__device__ __forceinline__ uint32_t enqueue_warp(bool want, uint32_t s, uint32_t cost, const QDev& q, uint32_t lane,
                                                 WarpBuf& b) {
  const bool nearq = cost < q.theta_hi;
  bool take = false;
  if (want) {
    const uint32_t bit = dflag_bit(s, nearq ? (q.par ^ 1u) : 2u);
    take = !(atomicOr(&q.dflag[s >> 3], bit) & bit);
  }
  const bool tN[1] = {take && nearq}, tF[1] = {take && !nearq};
  const uint32_t it[1] = {s};
  return append_lists<1>(tN, tF, it, q, lane, b);
}

// Single-entry push for warps whose lanes may serve different queries
// (split and seed tasks): lanes are aggregated per (query, list) with
// __match_any_sync.  which: 0 = near-out list, 1 = far-out list.
__device__ __forceinline__ void push_multi(bool take, uint32_t item, uint32_t which, const QDev& q, uint32_t slot,
                                           uint32_t lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t key = take ? slot * 2u + which : 0xFFFFFFFFu;
  const unsigned m = __match_any_sync(FULL, key);
  const uint32_t leader = (uint32_t)(__ffs(m) - 1);
  uint32_t base = 0;
  if (take && lane == leader) base = atomicAdd(which == 0u ? &q.ctl->n_near : &q.ctl->n_far2, (uint32_t)__popc(m));
  base = __shfl_sync(FULL, base, leader);
  if (take) {
    const uint32_t pos = base + (uint32_t)__popc(m & ((1u << lane) - 1u));
    uint32_t* buf = which == 0u ? q.qbuf[q.out_idx] : q.qbuf[q.far2_idx];
    if (pos < q.cap)
      buf[pos] = item;
    else
      atomicExch(&q.ctl->overflow, 1u);
  }
}

// Lower bound on the cost of a tree over the groups of S, whatever its vertices:
// u16 [2^k] after the tour tables (64 words are kept there).
__device__ __forceinline__ unsigned short* span_table(const QDev& q) {
  return reinterpret_cast<unsigned short*>(q.tour + (size_t)q.k * q.k * (1u << q.k) + (size_t)q.k * (1u << q.k));
}

// Largest arc weight worth a grow from a state of cost c that misses the groups
// of comp (-1: none): whatever the target, a tree over those groups is still to be
// paid for.  A heavier arc fails the target's own bound, which this spares the
// scattered read of: 76% of the targets of the 3M-vertex mix failed it.
__device__ __forceinline__ int64_t grow_limit(const QDev& q, uint32_t comp, uint32_t c, uint32_t best) {
  const uint32_t s = ld_round(span_table(q) + comp);
  return s == LB_INF ? -1 : (int64_t)best - (int64_t)c - (int64_t)s;
}

// Hop-bounded queries: the largest distance from vertex u to a group of comp
// over paths of at most b hops (INF32 if one is out of reach), computed by
// one lane for its own u; for b = 0 only u itself counts (distance 0: u is a
// member).
__device__ __forceinline__ uint32_t hop_budget_one(const QDev& q, uint32_t u, uint32_t comp, uint32_t b) {
  const uint32_t* row = (b == 0u ? q.dist : q.rows[b]) + (size_t)u * ROW;
  const Row8 rr = ld_row(row);
  const uint32_t(&r)[8] = rr.w;
  uint32_t mx = 0;
#pragma unroll
  for (int j = 0; j < KMAX; j++)
    if (j < q.k && ((comp >> j) & 1u)) {
      const uint32_t d = b == 0u ? (r[j] == 0u ? 0u : INF32) : r[j];
      mx = max(mx, d);
    }
  return mx;
}

// ---------------------------------------------------------------------------
// Grow of one DP state (v, p) -- or (v, p, d) with target hop count d+1 --
// along its arcs [a0, a1): target (u, p[, d+1]) at cost c + w(v, u).  GROW_U
// arcs per lane per step, so every lane keeps GROW_U independent chains
// (arc -> target word and bound -> flag) in flight.  A target is lowered
// with a fire-and-forget 64-bit min after a pre-check against its cost and
// the bound check; its state flag gates the list entry.
// ---------------------------------------------------------------------------
#ifndef GSTB_GROW_U
#define GSTB_GROW_U 4
#endif
constexpr int GROW_U = GSTB_GROW_U;
constexpr uint32_t GROW_LOCAL = 32u * GROW_U;  // arcs a state grows itself; the rest go out in chunks

struct GrowCnt {
  uint32_t arcs = 0, upd = 0, enq = 0;
};

__device__ __forceinline__ void grow_arcs(const QDev& q, const GraphDev& g, uint32_t lane, uint32_t v, uint32_t p,
                                          uint32_t comp, uint32_t c, uint32_t best, uint32_t lim, int dnext,
                                          uint32_t a0, uint32_t a1, GrowCnt& cnt, WarpBuf& wb) {
  const int k = q.k;
  const uint32_t nd = (uint32_t)q.nd, thi = q.theta_hi, par = q.par;
  const unsigned short* __restrict__ lbt = q.lbt;
  for (uint32_t base = a0; base < a1; base += 32u * GROW_U) {
    uint2 arc[GROW_U];
    bool ok[GROW_U];
#pragma unroll
    for (int u = 0; u < GROW_U; u++) {
      const uint32_t a = base + (uint32_t)u * 32u + lane;
      ok[u] = a < a1;
      arc[u] = ok[u] ? __ldg(g.adj + a) : make_uint2(0u, 0u);
    }
    // the target's bound first: it rejects most targets (a neighbour of a
    // hub is rarely close to the missing groups), and only the targets it
    // passes need their 8-byte table word (another random sector)
    uint32_t t[GROW_U], cur[GROW_U], lbu[GROW_U], nc[GROW_U];
    bool want[GROW_U];
#pragma unroll
    for (int u = 0; u < GROW_U; u++) {
      ok[u] = ok[u] && arc[u].y <= lim;
      const uint32_t vp = (arc[u].x << k) | p;
      t[u] = dnext < 0 ? vp : vp * nd + (uint32_t)dnext;
      lbu[u] = ok[u] ? (uint32_t)ld_round(lbt + ((size_t)arc[u].x << k) + comp) : 0u;
    }
    bool any = false;
#pragma unroll
    for (int u = 0; u < GROW_U; u++) {
      nc[u] = c + arc[u].y;
      want[u] = ok[u] && lb_ok(nc[u], lbu[u], best);
      any = any || want[u];
      if (ok[u]) cnt.arcs++;
    }
    if (__any_sync(0xFFFFFFFFu, any)) {
#pragma unroll
      for (int u = 0; u < GROW_U; u++) cur[u] = want[u] ? (uint32_t)(ld_cg(q.table + t[u]) >> 32) : 0u;
#pragma unroll
      for (int u = 0; u < GROW_U; u++) want[u] = want[u] && nc[u] < cur[u];
    }
    if (dnext >= 0) {
      // hop-bounded target (u, p, dnext): its missing groups must stay within
      // the D - dnext hops left from u (the test its expansion would apply);
      // a target that fails is never written, flagged or queued
#pragma unroll
      for (int u = 0; u < GROW_U; u++)
        if (want[u]) {
          const uint32_t h = hop_budget_one(q, arc[u].x, comp, (uint32_t)(q.D - dnext));
          want[u] = h != INF32 && (unsigned long long)nc[u] + h <= best;
        }
    }
#pragma unroll
    for (int u = 0; u < GROW_U; u++) {
      if (want[u]) {
        // the pre-check already saw a higher cost: enqueue on it and let the
        // 64-bit min land without waiting for its result (a concurrent lower
        // write also enqueues; the flag keeps the list free of duplicates)
        red_min(q.table + t[u], pack(nc[u], PAR_GROW | v));
        cnt.upd++;
      }
    }
    // near entries are flagged with the next round's parity, far ones with bit 2
    uint32_t old[GROW_U], bit[GROW_U];
#pragma unroll
    for (int u = 0; u < GROW_U; u++) {
      bit[u] = dflag_bit(t[u], nc[u] < thi ? (par ^ 1u) : 2u);
      old[u] = want[u] ? atomicOr(&q.dflag[t[u] >> 3], bit[u]) : bit[u];
    }
    bool tN[GROW_U], tF[GROW_U];
#pragma unroll
    for (int u = 0; u < GROW_U; u++) {
      const bool take = !(old[u] & bit[u]);
      tN[u] = take && nc[u] < thi;
      tF[u] = take && !(nc[u] < thi);
    }
    cnt.enq += append_lists<GROW_U>(tN, tF, t, q, lane, wb);
  }
}

// A warp hands the arcs [a0, a1) of a state's grow to k_heavy in HUB_CHUNK
// pieces.  Entries below the list's capacity are always written (empty
// ranges when the run does not fit), so k_heavy never reads a stale entry.
// Returns false if the run did not fit: the caller then grows those arcs.  The
// caller keeps the first GROW_LOCAL arcs, so it needs more than that, also where
// the threshold (hub_min_deg, 32 or more) is lower.
constexpr uint32_t CH_GROW = 1u << 31;  // big-list entry is a DP grow chunk
constexpr uint32_t CH_HOP = 1u << 30;   // ... of a hop-bounded state

__device__ __forceinline__ bool push_grow_chunks(const RoundDesc& sd, RoundDesc* rd, uint32_t slot, bool hop, uint32_t s, uint32_t a0,
                                                 uint32_t a1, uint32_t lane) {
  const uint32_t nch = (a1 - a0 + HUB_CHUNK - 1u) / HUB_CHUNK;
  uint32_t cb = 0;
  if (lane == 0) cb = atomicAdd(&rd->n_big, nch);
  cb = __shfl_sync(0xFFFFFFFFu, cb, 0);
  const bool fits = cb + nch <= sd.big_cap;
  const uint32_t x = slot | CH_GROW | (hop ? CH_HOP : 0u);
  for (uint32_t c = lane; c < nch && cb + c < sd.big_cap; c += 32u) {
    const uint32_t s0 = a0 + c * HUB_CHUNK;
    sd.big[cb + c] = fits ? make_uint4(x, s, s0, min(s0 + HUB_CHUNK, a1)) : make_uint4(slot, 0u, 0u, 0u);
  }
  return fits;
}

// Load the capped group distances of vertex v into every lane's registers.
__device__ __forceinline__ void load_dl(const QDev& q, uint32_t v, uint32_t (&dl)[KMAX],
                                        uint32_t& raw_sum_ok, uint32_t comp,
                                        unsigned long long& raw_sum) {
  const Row8 row = ld_row(q.dist + (size_t)v * ROW);
  const uint32_t(&r)[8] = row.w;
  raw_sum = 0;
  raw_sum_ok = 1;
#pragma unroll
  for (int j = 0; j < KMAX; j++) {
    dl[j] = min(r[j], q.cap1);
    if (j < q.k && (comp >> j & 1u)) {
      if (r[j] == INF32) raw_sum_ok = 0;
      raw_sum += r[j];
    }
  }
}

// Slot owning flat item `it` of task type t: largest s with pre[s] <= it.
__device__ __forceinline__ uint32_t find_slot(const uint32_t* __restrict__ pre, int nslots, uint32_t it) {
  int lo = 0, hi = nslots;  // pre[lo] <= it < pre[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (__ldcg(pre + mid) <= it)
      lo = mid;
    else
      hi = mid;
  }
  return (uint32_t)lo;
}

// Same search over a prefix array staged in shared memory.
__device__ __forceinline__ uint32_t find_slot_s(const uint32_t* pre, int nslots, uint32_t it) {
  int lo = 0, hi = nslots;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (pre[mid] <= it)
      lo = mid;
    else
      hi = mid;
  }
  return (uint32_t)lo;
}

// A DP state's vertex row staged for its merges: the costs of its 2^k table
// entries and its 2^k bound-table entries.
struct MergeTile {
  uint32_t cost[1u << KMAX];
  unsigned short lb[1u << KMAX];
};

// ---------------------------------------------------------------------------
// Unbounded DP item (v, p), in two parts.  dp_gate runs on one lane for its
// own item: it takes the item out of the near list, drops it when its cost
// is above the incumbent, updates the incumbent from the complement merge
// and the one-label completion, and applies the bound; dp_expand then grows
// and merges the surviving state with the whole warp.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool dp_gate(const QDev& q, uint32_t s, uint32_t& c_out, uint32_t& best_out,
                                        bool& counted) {
  const int k = q.k;
  const uint32_t K2 = 1u << k, full = (uint32_t)q.full;
  const uint32_t v = s >> k, p = s & (K2 - 1u);
  counted = false;
  atomicAnd(&q.dflag[s >> 3], ~dflag_bit(s, q.par));
  const uint32_t c = (uint32_t)(ld_cg(q.table + s) >> 32);
  uint32_t best = ld_best(q.ctl);
  if (c == INF32 || c > best) return false;
  unsigned long long* row = q.table + (size_t)v * K2;
  if (p == full) {
    if (c < best) atomicMin(&q.ctl->best, c);
    return false;
  }
  const uint32_t comp = full ^ p;
  uint32_t dl[KMAX], sum_ok;
  unsigned long long raw_sum;
  load_dl(q, v, dl, sum_ok, comp, raw_sum);
  // complement merge straight into the full state (DPQ.cu:82-94); a full
  // state of cost equal to best is still recorded: best may come from a
  // bound-only tree (star or one-label) that has no table entry
  const uint32_t cc = (uint32_t)(ld_cg(row + comp) >> 32);
  if (cc != INF32) {
    const unsigned long long m = (unsigned long long)c + cc;
    if (m <= best) {
      atomicMin(row + full, pack((uint32_t)m, PAR_MERGE | p));
      atomicMin(&q.ctl->best_full, (m << 32) | v);
      if (m < best) {
        atomicMin(&q.ctl->best, (uint32_t)m);
        best = (uint32_t)m;
      }
    }
  }
  // one-label completion: T(v,p) plus shortest paths to the missing groups
  // (DPQ.cu:95-107, CPUNONHOP.h:684-699)
  if (sum_ok) {
    const unsigned long long ol = (unsigned long long)c + raw_sum;
    if (ol < best) {
      atomicMin(&q.ctl->best, (uint32_t)ol);
      best = (uint32_t)ol;
    }
  }
  counted = true;
  const uint32_t lbv = ld_round(q.lbt + ((size_t)v << k) + comp);
  c_out = c;
  best_out = best;
  return lb_ok(c, lbv, best);
}

__device__ void dp_expand(const QDev& q, const GraphDev& g, uint32_t s, uint32_t c, uint32_t best, uint32_t lane,
                          const RoundDesc& sd, RoundDesc* rd, uint32_t slot, WarpStat& ws, WarpBuf& wb,
                          MergeTile* mt) {
  const int k = q.k;
  const uint32_t K2 = 1u << k, full = (uint32_t)q.full;
  const uint32_t v = s >> k, p = s & (K2 - 1u), comp = full ^ p;
  unsigned long long* row = q.table + (size_t)v * K2;
  const unsigned short* lbt = q.lbt;
  GrowCnt gc;
  // grow, only from states of cost <= best/2 (optimal-tree decomposition,
  // CPUNONHOP.h:820; exact for the unbounded problem); a high-degree vertex
  // grows its first GROW_LOCAL arcs here and hands the rest to k_heavy
  const int64_t glim = 2ull * c <= best ? grow_limit(q, comp, c, best) : -1;
  if (glim > 0) {
    const uint32_t lim = (uint32_t)glim;
    uint32_t a0, a1;
    arc_range(g, v, lim, a0, a1);
    if (sd.grow_chunks && a1 - a0 >= max(sd.hub_min_deg, GROW_LOCAL + 1u) &&
        push_grow_chunks(sd, rd, slot, false, s, a0 + GROW_LOCAL, a1, lane))
      a1 = a0 + GROW_LOCAL;
    grow_arcs(q, g, lane, v, p, comp, c, best, lim, -1, a0, a1, gc, wb);
  }
  // merge with every proper, non-empty subset p2 of the complement
  // (DPQ.cu:140-170; the complement itself went to the full state above).
  // Lane j takes the subsets idx = j, j+32, .. (p2 = the idx+1-th subset of
  // the complement, by bit deposit); a state with many partners first stages
  // its vertex's costs and bound row in shared memory with coalesced loads,
  // so every partner is read from there.  A staged cost can be higher than
  // the table's by then (another warp lowered it): a partner missed that way
  // merges with this state when it is expanded itself, and a target whose
  // cost only looked higher gets a min that changes nothing.
  uint32_t merges = 0;
  {
    const uint32_t nsub = (1u << __popc(comp)) - 2u;
    const bool staged = mt != nullptr && sd.merge_stage != 0u && nsub >= sd.merge_stage;
    if (staged) {
      for (uint32_t i = lane; i < K2; i += 32u) {
        mt->cost[i] = (uint32_t)(ld_cg(row + i) >> 32);
        mt->lb[i] = ld_round(lbt + ((size_t)v << k) + i);
      }
      __syncwarp();
    }
    for (uint32_t b = 0; b < nsub; b += 32) {
      uint32_t idx = b + lane;
      bool want = false;
      uint32_t t = 0, m32 = 0;
      if (idx < nsub) {
        uint32_t p2 = pdep(idx + 1u, comp);
        uint32_t qset = p | p2;
        uint32_t c2 = staged ? mt->cost[p2] : (uint32_t)(ld_cg(row + p2) >> 32);
        uint32_t cq = staged ? mt->cost[qset] : (uint32_t)(ld_cg(row + qset) >> 32);
        if (c2 != INF32) {
          merges++;
          unsigned long long m = (unsigned long long)c + c2;
          // conditional tree merging: 3m <= 2 best (CPUNONHOP.h:941)
          if (3ull * m <= 2ull * best && m < cq) {
            uint32_t lbq = staged ? (uint32_t)mt->lb[full ^ qset] : ld_round(lbt + ((size_t)v << k) + (full ^ qset));
            if (lb_ok((uint32_t)m, lbq, best)) {
              m32 = (uint32_t)m;
              t = (v << k) | qset;
              red_min(q.table + t, pack(m32, PAR_MERGE | p));
              want = true;
              gc.upd++;
            }
          }
        }
      }
      gc.enq += enqueue_warp(want, t, m32, q, lane, wb);
    }
    if (staged) __syncwarp();  // the tile is free for the next state
  }
  const uint32_t sa = warp_sum(gc.arcs), su = warp_sum(gc.upd), se = warp_sum(gc.enq), sm = warp_sum(merges);
  if (lane == 0) {
    ws_add(ws, q.ctl, ST_ARCS, sa);
    ws_add(ws, q.ctl, ST_UPDATES, su);
    ws_add(ws, q.ctl, ST_ENQ, se);
    ws_add(ws, q.ctl, ST_MERGES, sm);
  }
}

// ---------------------------------------------------------------------------
// Hop-bounded DP item (v, p, d): state id ((v << k) | p) * nd + d; gate on
// one lane, expansion by the warp, as for the unbounded items.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool hop_gate(const QDev& q, uint32_t s, uint32_t& c_out, uint32_t& best_out,
                                         bool& counted) {
  const int k = q.k, nd = q.nd, D = q.D;
  const uint32_t K2 = 1u << k, full = (uint32_t)q.full;
  const uint32_t d = s % (uint32_t)nd, vp = s / (uint32_t)nd;
  const uint32_t v = vp >> k, p = vp & (K2 - 1u);
  counted = false;
  atomicAnd(&q.dflag[s >> 3], ~dflag_bit(s, q.par));
  const uint32_t c = (uint32_t)(ld_cg(q.table + s) >> 32);
  const uint32_t best = ld_best(q.ctl);
  if (c == INF32 || c > best) return false;
  // dominance: the same subset at a smaller hop count and no higher cost
  for (uint32_t e = 0; e < d; e++)
    if ((uint32_t)(ld_cg(q.table + (size_t)vp * nd + e) >> 32) <= c) return false;
  if (p == full) {
    if (c < best) atomicMin(&q.ctl->best, c);
    return false;
  }
  const uint32_t comp = full ^ p;
  // In a derivation of a tree of hop diameter <= D from (v, p, d), a group
  // missing from p is reached from v by a path outside the subtree, and that
  // path plus the subtree's height d is a path of the tree: it has at most
  // D - d hops.  So the missing groups must be within D - d hops of v.
  const uint32_t lbh = hop_budget_one(q, v, comp, (uint32_t)D - d);
  if (lbh == INF32 || (unsigned long long)c + lbh > best) return false;
  counted = true;
  const uint32_t lbv = ld_round(q.lbt + ((size_t)v << k) + comp);
  c_out = c;
  best_out = best;
  return lb_ok(c, lbv, best);
}

__device__ void hop_expand(const QDev& q, const GraphDev& g, uint32_t s, uint32_t c, uint32_t best, uint32_t lane,
                           const RoundDesc& sd, RoundDesc* rd, uint32_t slot, WarpStat& ws, WarpBuf& wb) {
  const int k = q.k, nd = q.nd, D = q.D;
  const uint32_t K2 = 1u << k, full = (uint32_t)q.full;
  const uint32_t d = s % (uint32_t)nd, vp = s / (uint32_t)nd;
  const uint32_t v = vp >> k, p = vp & (K2 - 1u), comp = full ^ p;
  const unsigned short* lbt = q.lbt;
  GrowCnt gc;
  const int64_t glim = d < (uint32_t)D ? grow_limit(q, comp, c, best) : -1;
  if (glim > 0) {  // grow d -> d+1 (CPUHOP.h:192-206)
    const uint32_t lim = (uint32_t)glim;
    uint32_t a0, a1;
    arc_range(g, v, lim, a0, a1);
    if (sd.grow_chunks && a1 - a0 >= max(sd.hub_min_deg, GROW_LOCAL + 1u) &&
        push_grow_chunks(sd, rd, slot, true, s, a0 + GROW_LOCAL, a1, lane))
      a1 = a0 + GROW_LOCAL;
    grow_arcs(q, g, lane, v, p, comp, c, best, lim, (int)d + 1, a0, a1, gc, wb);
  }
  // merge with (v, p2, d2), p2 a non-empty subset of the complement,
  // d2 <= D - d, into (v, p|p2, max(d, d2))  (CPUHOP.h:208-227)
  uint32_t merges = 0;
  {
    const uint32_t nsub = (1u << __popc(comp)) - 1u;
    const uint32_t nd2 = (uint32_t)D - d + 1u;
    const uint32_t npairs = nsub * nd2;
    unsigned long long* rowv = q.table + ((size_t)v << k) * nd;
    for (uint32_t b = 0; b < npairs; b += 32) {
      uint32_t idx = b + lane;
      bool want = false;
      uint32_t t = 0, m32 = 0;
      if (idx < npairs) {
        uint32_t p2 = pdep(idx / nd2 + 1u, comp);
        uint32_t d2 = idx % nd2;
        uint32_t c2 = (uint32_t)(ld_cg(rowv + (size_t)p2 * nd + d2) >> 32);
        if (c2 != INF32) {
          merges++;
          unsigned long long m = (unsigned long long)c + c2;
          uint32_t qset = p | p2;
          uint32_t ndd = max(d, d2);
          uint32_t par = PAR_MERGE | p | (d << 8) | (d2 << 11);
          if (m <= best) {
            m32 = (uint32_t)m;
            t = ((v << k) | qset) * (uint32_t)nd + ndd;
            if (qset == full) {
              // recorded at cost == best too: best may come from a tree
              // that has no table entry
              atomicMin(q.table + t, pack(m32, par));
              atomicMin(&q.ctl->best_full, ((unsigned long long)m32 << 32) | (v * 8u + ndd));
              if (m32 < best) atomicMin(&q.ctl->best, m32);
            } else {
              uint32_t lbq = ld_round(lbt + ((size_t)v << k) + (full ^ qset));
              if (lb_ok(m32, lbq, best) && m32 < (uint32_t)(ld_cg(q.table + t) >> 32)) {
                red_min(q.table + t, pack(m32, par));
                want = true;
                gc.upd++;
              }
            }
          }
        }
      }
      gc.enq += enqueue_warp(want, t, m32, q, lane, wb);
    }
  }
  const uint32_t sa = warp_sum(gc.arcs), su = warp_sum(gc.upd), se = warp_sum(gc.enq), sm = warp_sum(merges);
  if (lane == 0) {
    ws_add(ws, q.ctl, ST_ARCS, sa);
    ws_add(ws, q.ctl, ST_UPDATES, su);
    ws_add(ws, q.ctl, ST_ENQ, se);
    ws_add(ws, q.ctl, ST_MERGES, sm);
  }
}

// A DP task: W items (one per lane) of the round's DP or hop-bounded list.
// Each lane runs its item's gates; then the warp expands the surviving
// states one after another.  W is chosen per round by the control step (1 when the
// round has few items, so that each state gets a warp of its own; up to 32
// when it has many, most of which the gates drop).
__device__ void dp_task(const QDev* qd, const uint32_t* __restrict__ pre, int nslots, uint32_t total,
                        uint32_t task, uint32_t W, bool hop, const GraphDev& g, uint32_t lane,
                        const RoundDesc& sd, RoundDesc* rd, WarpStat& ws, WarpBuf& wb, MergeTile* mt) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t it = task * W + lane;
  const bool valid = lane < W && it < total;
  uint32_t slot = 0xFFFFFFFFu, s = 0, c = 0, best = 0;
  bool live = false, counted = false;
  if (valid) {
    slot = find_slot_s(pre, nslots, it);
    const QDev& q = qd[slot];
    s = q.qbuf[q.in_idx][it - pre[slot]];
    live = hop ? hop_gate(q, s, c, best, counted) : dp_gate(q, s, c, best, counted);
  }
  // expanded-state counts, per query of the task
  unsigned cm = __ballot_sync(FULL, counted);
  while (cm) {
    const uint32_t si = __shfl_sync(FULL, slot, __ffs(cm) - 1);
    const unsigned same = __ballot_sync(FULL, counted && slot == si);
    if (lane == 0) ws_add(ws, qd[si].ctl, ST_EXPANDED, __popc(same));
    cm &= ~same;
  }
  unsigned lm = __ballot_sync(FULL, live);
  while (lm) {
    const uint32_t i = __ffs(lm) - 1;
    lm &= lm - 1u;
    const uint32_t si = __shfl_sync(FULL, slot, i), ss = __shfl_sync(FULL, s, i);
    const uint32_t cc = __shfl_sync(FULL, c, i), bb = __shfl_sync(FULL, best, i);
    const QDev& q = qd[si];
    if (hop)
      hop_expand(q, g, ss, cc, bb, lane, sd, rd, si, ws, wb);
    else
      dp_expand(q, g, ss, cc, bb, lane, sd, rd, si, ws, wb, mt);
  }
}

// Next task of a warp.  Each warp's first task is its own index; after that
// the warps take tasks from a shared counter (work stealing), so a warp that
// met cheap tasks keeps taking new ones while one with a long task (a hub
// vertex, a state with many merge partners) is still busy.
__device__ __forceinline__ uint32_t next_task(uint32_t* counter, uint32_t nwarps, uint32_t lane) {
  uint32_t t = 0;
  if (lane == 0) t = nwarps + atomicAdd(counter, 1u);
  return __shfl_sync(0xFFFFFFFFu, t, 0);
}

// ---------------------------------------------------------------------------
// Distance items.  A warp task holds W items (a vertex with the mask of its
// pending groups); W is chosen per round by the control step: 4 when the round has
// few items (short rounds, low latency), up to 32 when it has many (fewer
// per-task overheads).  Lanes 0..W-1 read the items' headers in parallel;
// then the arcs of all items of one query in the task are relaxed as one flat
// list, 32 x SSSP_U arcs per step.  Each lane keeps SSSP_U independent chains
// (arc -> distance row -> pending flag) in flight, and uneven degrees are
// spread over all 32 lanes.
// ---------------------------------------------------------------------------
constexpr uint32_t SSSP_WMAX = 32;   // most items per warp task
#ifndef GSTB_SSSP_U
#define GSTB_SSSP_U 4
#endif
constexpr int SSSP_U = GSTB_SSSP_U;  // arcs per lane per step
constexpr uint32_t HUB_LOCAL = 32;   // arcs of a hub item its own task relaxes

struct alignas(16) RelaxHdr {
  uint32_t d[KMAX];  // group distances at the item's vertex
  uint32_t rm;       // groups to relax from it
  uint32_t lim;      // largest arc weight that can still lower a distance
  uint32_t a0;       // first arc to relax
  uint32_t pad;
};

struct RelaxCnt {
  uint32_t arcs = 0, upd = 0, enq = 0;
};

// Per-warp shared scratch; a warp uses one member at a time: the headers of
// its distance items (or of a hub chunk), its bound rows' list, or a DP state's
// merge tile.
struct LbScratch {
  uint32_t v[64];         // live vertices still to evaluate, all of query `slot`
  uint32_t n, slot;
};
union WarpScratch {
  RelaxHdr hdr[32];
  LbScratch lb;
  MergeTile mg;
};

// Relax the arcs of the task's items [i0, i1), all of query q.  Lane j holds
// in `x` the inclusive prefix n_0 + ... + n_j of the task's arc counts; item
// i's arcs are [h[i].a0, h[i].a0 + n_i).  Every lane of the warp calls it with
// the same i0, i1.  A lowered distance is written with a fire-and-forget
// atomicMin after a pre-check; the pending-groups flag of the target gates
// its list entry (parity-split flags, so no update is lost); appends are
// aggregated over the whole warp.
__device__ __forceinline__ void relax_flat(const QDev& q, const RelaxHdr* __restrict__ h, uint32_t x, uint32_t i0,
                                           uint32_t i1, uint32_t capb, const GraphDev& g, uint32_t lane,
                                           RelaxCnt& cnt, WarpBuf& wb) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t lo_end = __shfl_sync(FULL, x, i0 == 0u ? 0u : i0 - 1u);
  const uint32_t f0 = i0 == 0u ? 0u : lo_end;
  const uint32_t f1 = __shfl_sync(FULL, x, i1 - 1u);
  const uint32_t thi = q.theta_hi, nsh = near_sh(q.par ^ 1u);
  uint32_t* __restrict__ dist = q.dist_nx;  // targets: the rows this round writes

  for (uint32_t base = f0; base < f1; base += 32u * SSSP_U) {
    uint2 arc[SSSP_U];
    uint32_t itm[SSSP_U], lim[SSSP_U];
    bool ok[SSSP_U];
#pragma unroll
    for (int u = 0; u < SSSP_U; u++) {
      const uint32_t f = base + (uint32_t)u * 32u + lane;
      // item of flat position f: the first i in [i0, i1) with x_i > f
      // (binary lifting over the lanes' prefixes)
      uint32_t pos = i0;
#pragma unroll
      for (uint32_t step = 16; step > 0; step >>= 1) {
        const uint32_t cand = pos + step - 1u;
        const uint32_t xc = __shfl_sync(FULL, x, min(cand, 31u));
        if (cand < i1 && xc <= f) pos += step;
      }
      const uint32_t xs = __shfl_sync(FULL, x, pos == 0u ? 0u : min(pos - 1u, 31u));
      const uint32_t start = pos == 0u ? 0u : xs;
      ok[u] = f < f1;
      itm[u] = ok[u] ? pos : i0;
      // the item's weight limit and first arc in one 8-byte shared load
      const uint2 la = *reinterpret_cast<const uint2*>(&h[itm[u]].lim);
      lim[u] = la.x;
      arc[u] = ok[u] ? __ldg(g.adj + la.y + (f - start)) : make_uint2(0u, 0u);
    }
    Row8 row[SSSP_U];
#pragma unroll
    for (int u = 0; u < SSSP_U; u++) {
      ok[u] = ok[u] && arc[u].y <= lim[u];
      if (ok[u])
        row[u] = ld_row(dist + (size_t)arc[u].x * ROW);
      else
        row[u] = Row8{};
    }
    uint32_t nn[SSSP_U], nf[SSSP_U];
#pragma unroll
    for (int u = 0; u < SSSP_U; u++) {
      nn[u] = nf[u] = 0u;
      if (ok[u]) {
        cnt.arcs++;
        // the item's distances and group mask in two 16-byte shared loads
        const uint4* hv = reinterpret_cast<const uint4*>(&h[itm[u]]);
        const uint4 h0 = hv[0], h1 = hv[1];
        const uint32_t rm = h1.w;
        const uint32_t dv[KMAX] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z};
        const uint32_t(&du)[8] = row[u].w;
#pragma unroll
        for (int t = 0; t < KMAX; t++) {
          if ((rm >> t) & 1u) {
            const uint32_t dt = dv[t];
            const uint32_t nd = dt + arc[u].y;
            if (nd >= dt && nd <= capb && nd < du[t]) {
              red_min(dist + (size_t)arc[u].x * ROW + t, nd);
              if (nd < thi)
                nn[u] |= 1u << t;
              else
                nf[u] |= 1u << t;
              cnt.upd++;
            }
          }
        }
      }
    }
    // flags: one fire-and-forget OR per target for both lists, skipped when
    // the row just read shows the bits set already.  The list entry is taken
    // when that row showed the list's byte empty.  Within a round the
    // next-parity and far bytes only gain bits, so the first OR to reach a
    // byte comes from a lane that read it empty: every newly pending vertex
    // is appended at least once.  Every lane that read it empty appends it;
    // the consumer's atomicAnd hands the groups to one of the entries and the
    // others find none.  No lane waits for an atomic's result.
    uint32_t itv[SSSP_U];
    bool tN[SSSP_U], tF[SSSP_U];
#pragma unroll
    for (int u = 0; u < SSSP_U; u++) {
      const uint32_t bits = (nn[u] << nsh) | (nf[u] << FAR_SH);
      // (exact rounds compare with the written row, the running minimum of
      // the round: it filters repeated relaxations of a target far better
      // than the previous round's row, at the price of a few entries for
      // vertices whose own new value has not been carried across yet)
      const uint32_t fw = row[u].w[FLAGW];
      if (bits & ~fw) red_or(dist + (size_t)arc[u].x * ROW + FLAGW, bits);
      tN[u] = nn[u] && ((fw >> nsh) & 0xFFu) == 0u;
      tF[u] = nf[u] && ((fw >> FAR_SH) & 0xFFu) == 0u;
      itv[u] = arc[u].x;
    }
    cnt.enq += append_lists<SSSP_U>(tN, tF, itv, q, lane, wb);
  }
}

// Warp-reduce a relaxation's counters into the warp's statistics.
__device__ __forceinline__ void relax_cnt_add(WarpStat& ws, QCtl* c, RelaxCnt cnt, uint32_t items, uint32_t lane) {
  const uint32_t a = warp_sum(cnt.arcs), u = warp_sum(cnt.upd), e = warp_sum(cnt.enq);
  if (lane == 0) {
    ws_add(ws, c, ST_SSSP, items);
    ws_add(ws, c, ST_SSSP_ARCS, a);
    ws_add(ws, c, ST_SSSP_UPDATES, u);
    ws_add(ws, c, ST_SSSP_ENQ, e);
  }
}

__device__ void sssp_task(const QDev* qd, const uint32_t* __restrict__ pre, int nslots,
                          uint32_t total, uint32_t task, uint32_t W, const GraphDev& g, uint32_t lane, WarpStat& ws,
                          const RoundDesc& sd, RoundDesc* rd, RelaxHdr* __restrict__ sh, WarpBuf& wb) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t it = task * W + lane;
  const bool valid = lane < W && it < total;
  const uint32_t slot = valid ? find_slot_s(pre, nslots, it) : 0xFFFFFFFFu;
  uint32_t n = 0, capb = INF32;
  bool active = false;
  if (valid) {
    const QDev& q = qd[slot];
    const int k = q.k;
    const uint32_t v = q.qbuf[q.in_idx][it - pre[slot]];
    // the header's loads depend on v only, so they are all in flight at once;
    // take the groups pending at v for this round's parity
    const uint32_t psh = near_sh(q.par);
    const uint32_t m =
        (atomicAnd(q.dist + (size_t)v * ROW + FLAGW, ~(0xFFu << psh)) >> psh) & 0xFFu;
    const Row8 dr = ld_row(q.dist + (size_t)v * ROW);
    uint32_t best = ld_best(q.ctl);
    const Row8 cut = ld_row_nc(g.wcut + (size_t)v * 8);
    const uint32_t b0 = cut.w[7];
    const uint32_t(&d)[8] = dr.w;
    if (q.dist_nx != q.dist) {
      // exact rounds: the distances that changed last round carry over into
      // the rows this round writes (the other rows hold them already)
      uint32_t* nx = q.dist_nx + (size_t)v * ROW;
#pragma unroll
      for (int t = 0; t < KMAX; t++)
        if (t < k && ((m >> t) & 1u)) red_min(nx + t, d[t]);
    }
    // star bound at v (unbounded queries only): v joined to every group by
    // shortest paths is a feasible tree (one-label completion, CPUNONHOP.h:684-699)
    if (q.D < 0) {
      unsigned long long sum = 0;
      bool fin = true;
#pragma unroll
      for (int t = 0; t < KMAX; t++)
        if (t < k) {
          fin = fin && d[t] != INF32;
          sum += d[t];
        }
      if (fin && sum < best) {
        atomicMin(&q.ctl->best, (uint32_t)sum);
        best = (uint32_t)sum;
      }
    }
    // distances beyond cap(best) cannot lower a bound below best: skip them
    capb = (uint32_t)((unsigned long long)best * q.cap_num / q.cap_den);
    // nor, for now, those from the reach on
    const bool beyond = capb >= q.reach;
    capb = min(capb, q.reach - 1u);
    uint32_t rm = 0, dmin = INF32, dmax = 0;
#pragma unroll
    for (int t = 0; t < KMAX; t++)
      if (t < k && ((m >> t) & 1u) && d[t] <= capb) {
        rm |= 1u << t;
        dmin = min(dmin, d[t]);
        dmax = max(dmax, d[t]);
      }
    active = rm != 0;
    uint32_t lim = 0;
    if (active) {
      lim = capb - dmin;
      if (beyond && capb - dmax < g.wmax && __ldca(&q.ctl->deferred) == 0u) q.ctl->deferred = 1u;
      const uint32_t a1 = arcs_end(g, v, cut, lim);
      n = a1 - b0;
      // hub: hand all but the first HUB_LOCAL arcs to k_heavy in chunks of
      // HUB_CHUNK arcs, one warp each
      if (n >= sd.hub_deg && n - HUB_LOCAL >= sd.hub_min_rest) {
        const uint32_t st0 = b0 + HUB_LOCAL;
        const uint32_t nch = (a1 - st0 + HUB_CHUNK - 1u) / HUB_CHUNK;
        const uint32_t cb = atomicAdd(&rd->n_big, nch);
        const bool fits = cb + nch <= sd.big_cap;
        // entries below the cap are always written (empty ranges when the
        // whole run does not fit) so k_heavy never reads a stale entry
        for (uint32_t c = 0; c < nch && cb + c < sd.big_cap; c++) {
          const uint32_t s0 = st0 + c * HUB_CHUNK;
          sd.big[cb + c] = fits ? make_uint4(slot | (rm << 16), v, s0, min(s0 + HUB_CHUNK, a1))
                                 : make_uint4(slot, v, 0u, 0u);
        }
        if (fits) n = HUB_LOCAL;
      }
    }
    RelaxHdr hd;
#pragma unroll
    for (int t = 0; t < KMAX; t++) hd.d[t] = d[t];
    hd.rm = rm;
    hd.lim = lim;
    hd.a0 = b0;
    hd.pad = 0;
    sh[lane] = hd;
  }
  __syncwarp();
  // valid items are lanes [0, nvalid); split them into runs of one query
  const unsigned vmask = __ballot_sync(FULL, valid);
  if (vmask == 0u) return;
  const uint32_t nvalid = 32u - __clz(vmask);
  uint32_t x = n;  // inclusive prefix of the arc counts over the lanes
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  const uint32_t prev_slot = __shfl_up_sync(FULL, slot, 1);
  unsigned runs = __ballot_sync(FULL, valid && (lane == 0u || prev_slot != slot));
  const unsigned amask = __ballot_sync(FULL, active);
  while (runs) {
    const uint32_t i0 = (uint32_t)(__ffs(runs) - 1);
    runs &= runs - 1u;
    const uint32_t i1 = runs ? (uint32_t)(__ffs(runs) - 1) : nvalid;
    const uint32_t si = __shfl_sync(FULL, slot, i0);
    const bool in_run = lane >= i0 && lane < i1;
    uint32_t cb = in_run ? capb : INF32;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cb = min(cb, __shfl_xor_sync(FULL, cb, o));
    const unsigned rmask = (i1 >= 32u ? 0xFFFFFFFFu : ((1u << i1) - 1u)) & ~((1u << i0) - 1u);
    const uint32_t n_items = __popc(amask & rmask);
    const QDev& q = qd[si];
    RelaxCnt cnt;
    relax_flat(q, sh, x, i0, i1, cb, g, lane, cnt, wb);
    relax_cnt_add(ws, q.ctl, cnt, n_items, lane);
  }
}

// One hub chunk (k_heavy, one warp): relax arcs [first, end) of vertex v for
// the pending groups recorded by k_light.  Same relaxation as sssp_task.
__device__ void hub_chunk(const QDev* qd, const uint4 item, const GraphDev& g, uint32_t lane,
                          RelaxHdr* __restrict__ sh, WarpStat& ws, WarpBuf& wb) {
  const unsigned FULL = 0xFFFFFFFFu;
  if (item.z >= item.w) return;  // filler entry of a chunk run that did not fit
  const uint32_t slot = item.x & 0xFFFFu, v = item.y;
  const QDev& q = qd[slot];
  uint32_t capb = 0, n = 0;
  if (lane == 0) {
    const Row8 dr = ld_row(q.dist + (size_t)v * ROW);
    const uint32_t best = ld_best(q.ctl);
    const uint32_t(&d)[8] = dr.w;
    capb = min((uint32_t)((unsigned long long)best * q.cap_num / q.cap_den), q.reach - 1u);
    uint32_t rm = 0, dmin = INF32;
#pragma unroll
    for (int t = 0; t < KMAX; t++)
      if (((item.x >> (16 + t)) & 1u) && d[t] <= capb) {
        rm |= 1u << t;
        dmin = min(dmin, d[t]);
      }
    RelaxHdr hd;
#pragma unroll
    for (int t = 0; t < KMAX; t++) hd.d[t] = d[t];
    hd.rm = rm;
    hd.lim = rm ? capb - dmin : 0u;
    hd.a0 = item.z;
    hd.pad = 0;
    sh[0] = hd;
    n = rm ? item.w - item.z : 0u;
  }
  __syncwarp();
  capb = __shfl_sync(FULL, capb, 0);
  n = __shfl_sync(FULL, n, 0);
  if (n == 0) return;
  RelaxCnt cnt;
  relax_flat(q, sh, n, 0u, 1u, capb, g, lane, cnt, wb);  // one item: every lane holds its prefix n
  relax_cnt_add(ws, q.ctl, cnt, 0u, lane);
}

// One DP grow chunk (k_heavy, one warp): arcs [first, end) of a state that a
// k_light warp handed over.  The state's current cost is read again (it can
// only have dropped, and a lower cost grows validly too) and the gates of the
// state's own expansion are re-checked.
__device__ void grow_chunk(const QDev* qd, const uint4 item, const GraphDev& g, uint32_t lane,
                           WarpStat& ws, WarpBuf& wb) {
  const unsigned FULL = 0xFFFFFFFFu;
  if (item.z >= item.w) return;  // filler entry of a chunk run that did not fit
  const uint32_t slot = item.x & 0xFFFFu;
  const bool hop = (item.x & CH_HOP) != 0u;
  const QDev& q = qd[slot];
  const int k = q.k;
  const uint32_t K2 = 1u << k, full = (uint32_t)q.full, nd = (uint32_t)q.nd, s = item.y;
  const uint32_t vp = hop ? s / nd : s, d = hop ? s % nd : 0u;
  const uint32_t v = vp >> k, p = vp & (K2 - 1u), comp = full ^ p;
  uint32_t c = 0, best = 0, lbv = 0;
  if (lane == 0) {
    c = (uint32_t)(ld_cg(q.table + s) >> 32);
    best = ld_best(q.ctl);
    lbv = ld_round(q.lbt + ((size_t)v << k) + comp);
  }
  c = __shfl_sync(FULL, c, 0);
  best = __shfl_sync(FULL, best, 0);
  lbv = __shfl_sync(FULL, lbv, 0);
  if (c == INF32 || c > best || !lb_ok(c, lbv, best)) return;
  if (!hop && 2ull * c > best) return;
  const int64_t glim = grow_limit(q, comp, c, best);
  if (glim <= 0) return;
  GrowCnt gc;
  grow_arcs(q, g, lane, v, p, comp, c, best, (uint32_t)glim, hop ? (int)d + 1 : -1, item.z, item.w, gc, wb);
  const uint32_t a = warp_sum(gc.arcs), u = warp_sum(gc.upd), e = warp_sum(gc.enq);
  if (lane == 0) {
    ws_add(ws, q.ctl, ST_ARCS, a);
    ws_add(ws, q.ctl, ST_UPDATES, u);
    ws_add(ws, q.ctl, ST_ENQ, e);
  }
}

// ---------------------------------------------------------------------------
// Gathered distance rows of hop-bounded queries.  A state at vertex v with b
// hops left has a subtree of at most D - b hops below it, which holds a member:
// the rows over b hops are only ever read at vertices within D - b hops of a
// member, and so are the rows over b - 1 hops at their neighbours.  The first
// half of the rounds reaches that far anyway and relaxes from the vertices that
// changed; from round floor(D/2) + 1 on the set shrinks back to the members,
// and each of its vertices gathers min over its arcs of the neighbour's row over
// b - 1 hops: plain loads, no atomics, no lists, none of the arcs of the many
// vertices that no tree can use.  On 3M vertices with D = 4, relaxing in rounds
// 3 and 4 scanned 83-99% of all 234M arcs each.  Measured against relaxing in
// all D rounds: 48 queries with D = 2..4 on 2^20 vertices 27.2 -> 4.5 ms, six
// one at a time 4.1 -> 2.2 ms, 48 mixed queries on 3M vertices 202 -> 117 ms.
//
// Four items of the lists 0 .. D - b per warp, 8 lanes each; a vertex with at
// least hub_min_deg arcs hands all but the first 32 to k_heavy in chunks.  With 4
// and 16 lanes (queries one at a time, then 48 in a batch, on 2^20 vertices): 1579
// and 1454 us against 1491, 2.98 and 2.88 ms against 2.94.
// ---------------------------------------------------------------------------
constexpr uint32_t CH_PULL = 1u << 29;  // big-list entry is a chunk of a gathered row
constexpr uint32_t PULL_LANES = 8;
constexpr int PULL_U = 4;  // arcs per lane per step

// Item idx of the lists 0, 1, ..: vertex, and the list it is in.
__device__ __forceinline__ uint32_t list_item(const QDev& q, uint32_t idx, uint32_t& h) {
  h = 0;
  while (h < 3u && idx >= q.n_list[h]) idx -= q.n_list[h++];
  return q.qbuf[h][idx];
}

__device__ __forceinline__ void load_row(const uint32_t* rows, uint32_t v, uint32_t (&r)[KMAX]) {
  const Row8 x = ld_row(rows + (size_t)v * ROW);
#pragma unroll
  for (int t = 0; t < KMAX; t++) r[t] = x.w[t];
}

// Lower m[] over up to PULL_U arcs a0 + i * stride (< a1) of weight <= lim;
// returns the arcs taken.
__device__ __forceinline__ uint32_t pull_arcs(const GraphDev& g, const uint32_t* src, int k, uint32_t a0,
                                              uint32_t stride, uint32_t a1, uint32_t lim, uint32_t capb,
                                              uint32_t (&m)[KMAX]) {
  uint2 arc[PULL_U];
  bool ok[PULL_U];
  uint32_t n = 0;
#pragma unroll
  for (int u = 0; u < PULL_U; u++) {
    const uint32_t a = a0 + (uint32_t)u * stride;
    ok[u] = a < a1;
    arc[u] = ok[u] ? __ldg(g.adj + a) : make_uint2(0u, 0u);
  }
  Row8 x[PULL_U];
#pragma unroll
  for (int u = 0; u < PULL_U; u++) {
    if (ok[u] && arc[u].y <= lim) {
      x[u] = ld_row(src + (size_t)arc[u].x * ROW);
      n++;
    } else {
      x[u] = Row8{{INF32, INF32, INF32, INF32, INF32, INF32, INF32, INF32}};
    }
  }
#pragma unroll
  for (int u = 0; u < PULL_U; u++) {
#pragma unroll
    for (int t = 0; t < KMAX; t++) {
      const uint32_t r = x[u].w[t], d = r + arc[u].y;
      if (t < k && r != INF32 && d <= capb) m[t] = min(m[t], d);
    }
  }
  return n;
}

__device__ void pull_task(const QDev* qd, const uint32_t* __restrict__ pre, int nslots, uint32_t total, uint32_t task,
                          const GraphDev& g, uint32_t lane, WarpStat& ws, const RoundDesc& sd, RoundDesc* rd) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t gl = lane & (PULL_LANES - 1u), g0 = lane - gl;
  const unsigned gm = ((1u << PULL_LANES) - 1u) << g0;
  const uint32_t it = task * (32u / PULL_LANES) + g0 / PULL_LANES;
  uint32_t slot = 0xFFFFFFFFu, arcs = 0;
  if (it < total) {
    slot = find_slot(pre, nslots, it);
    const QDev& q = qd[slot];
    const int k = q.k;
    const uint32_t b = q.hops + 1u;
    const uint32_t* src = q.rows[b - 1u];
    uint32_t h, m[KMAX];
    const uint32_t v = list_item(q, it - __ldcg(pre + slot), h);
    load_row(src, v, m);
    // a vertex of a list may be in a nearer one too: it is done there
    bool seen = false;
    if (h == 1u) {
#pragma unroll
      for (int t = 0; t < KMAX; t++) seen = seen || (t < k && m[t] == 0u);
    } else if (h > 1u) {
      uint32_t r[KMAX];
      load_row(q.rows[h - 1u], v, r);
#pragma unroll
      for (int t = 0; t < KMAX; t++) seen = seen || (t < k && r[t] != INF32);
    }
    if (!seen) {
      const uint32_t capb = ld_best(q.ctl);  // what exceeds the incumbent is as good as out of reach
      uint32_t a0, a1;
      arc_range(g, v, capb, a0, a1);
      const uint32_t n = a1 - a0;
      if (sd.big != nullptr && n >= sd.hub_min_deg && n - HUB_LOCAL >= sd.hub_min_rest) {
        const uint32_t st0 = a0 + HUB_LOCAL, nch = (a1 - st0 + HUB_CHUNK - 1u) / HUB_CHUNK;
        uint32_t cb = 0;
        if (gl == 0u) cb = atomicAdd(&rd->n_big, nch);
        cb = __shfl_sync(gm, cb, g0);
        const bool fits = cb + nch <= sd.big_cap;
        for (uint32_t c = gl; c < nch && cb + c < sd.big_cap; c += PULL_LANES) {
          const uint32_t s0 = st0 + c * HUB_CHUNK;
          sd.big[cb + c] = fits ? make_uint4(slot | CH_PULL, v, s0, min(s0 + HUB_CHUNK, a1)) : make_uint4(slot, v, 0u, 0u);
        }
        if (fits) a1 = a0 + HUB_LOCAL;
      }
      for (uint32_t base = a0; base < a1; base += PULL_LANES * PULL_U)
        arcs += pull_arcs(g, src, k, base + gl, PULL_LANES, a1, capb, capb, m);
#pragma unroll
      for (int t = 0; t < KMAX; t++) m[t] = __reduce_min_sync(gm, m[t]);
      uint4* out = reinterpret_cast<uint4*>(q.rows[b] + (size_t)v * ROW);
      if (gl == 0u) out[0] = make_uint4(m[0], m[1], m[2], m[3]);
      if (gl == 1u) out[1] = make_uint4(m[4], m[5], m[6], 0u);
    }
  }
  __syncwarp();
  // counters: the 8 lanes of an item, then per query
#pragma unroll
  for (uint32_t o = PULL_LANES / 2u; o > 0u; o >>= 1) arcs += __shfl_xor_sync(FULL, arcs, o);
  for (uint32_t i = 0; i < 32u; i += PULL_LANES) {
    const uint32_t si = __shfl_sync(FULL, slot, i), a = __shfl_sync(FULL, arcs, i);
    if (lane == 0 && si != 0xFFFFFFFFu) {
      ws_add(ws, qd[si].ctl, ST_SSSP, 1u);
      ws_add(ws, qd[si].ctl, ST_SSSP_ARCS, a);
    }
  }
}

// One chunk of a gathered row (k_heavy, one warp): lowers the row that the
// vertex's own task wrote.  The arcs ascend in weight, so a chunk whose first
// arc cannot lower any of the row's distances ends at once.
__device__ void pull_chunk(const QDev* qd, const uint4 item, const GraphDev& g, uint32_t lane, WarpStat& ws) {
  const uint32_t slot = item.x & 0xFFFFu, v = item.y;
  const QDev& q = qd[slot];
  const int k = q.k;
  const uint32_t b = q.hops + 1u, capb = ld_best(q.ctl);
  uint32_t* out = q.rows[b] + (size_t)v * ROW;
  uint32_t cur[KMAX], m[KMAX], top = 0;
  load_row(out, 0u, cur);
#pragma unroll
  for (int t = 0; t < KMAX; t++) {
    m[t] = INF32;
    if (t < k) top = max(top, cur[t]);
  }
  const uint32_t lim = min(capb, top == 0u ? 0u : top - 1u);
  if (__ldg(&g.adj[item.z].y) > lim) return;
  uint32_t arcs = 0;
  for (uint32_t base = item.z; base < item.w; base += 32u * PULL_U)
    arcs += pull_arcs(g, q.rows[b - 1u], k, base + lane, 32u, item.w, lim, capb, m);
#pragma unroll
  for (int t = 0; t < KMAX; t++) {
    const uint32_t x = __reduce_min_sync(0xFFFFFFFFu, m[t]);
    if (lane == (uint32_t)t && t < k && x < cur[t]) red_min(out + t, x);
  }
  const uint32_t a = warp_sum(arcs);
  if (lane == 0) ws_add(ws, q.ctl, ST_SSSP_ARCS, a);
}

// Near-far split of one far item: cost in [theta_lo, theta_hi) -> near list;
// above -> far-out list; below theta_lo it was already expanded at that cost
// (every new cost is >= the cost of the item that produced it) -> dropped.
// Distance items are vertices with a mask of pending groups; DP items are
// states.  Items moved to the near list carry the parity of the next round.
// The caller pushes `s` to the near-out list if toN and to the far-out list
// if toF (push_multi, warp-aggregated).
__device__ void split_item(const QDev& q, uint32_t s, bool& toN, bool& toF) {
  uint32_t best = ld_cg(&q.ctl->best);
  toN = toF = false;
  if (q.phase == PH_SSSP && q.rescan) {
    // item = a vertex: its distances are final, and arcs of theirs that led beyond
    // the old reach are still to be relaxed, unless none stays under the cap
    const uint32_t capb = (uint32_t)((unsigned long long)best * q.cap_num / q.cap_den);
    uint32_t r[KMAX], nb = 0;
    load_row(q.dist, s, r);
#pragma unroll
    for (int t = 0; t < KMAX; t++)
      if (t < q.k && r[t] != INF32 && r[t] < capb) nb |= 1u << t;
    // (the next round's parity, which a split round does not flip)
    if (nb) red_or(q.dist + (size_t)s * ROW + FLAGW, nb << near_sh(q.par));
    toN = nb != 0u;
    return;
  }
  if (q.phase == PH_SSSP) {
    uint32_t* fw = q.dist + (size_t)s * ROW + FLAGW;
    const uint32_t capb = (uint32_t)((unsigned long long)best * q.cap_num / q.cap_den);
    const uint32_t fm = (atomicAnd(fw, ~(0xFFu << FAR_SH)) >> FAR_SH) & 0xFFu;
    uint32_t nb = 0, kb = 0;
    for (int t = 0; t < q.k; t++) {
      if (!((fm >> t) & 1u)) continue;
      uint32_t d = ld_cg(q.dist + (size_t)s * ROW + t);
      if (d < q.theta_lo || d == INF32 || d > capb) continue;
      if (d < q.theta_hi)
        nb |= 1u << t;
      else
        kb |= 1u << t;
    }
    // items moved to the near list carry the next round's parity, which a
    // split round does not flip
    const uint32_t psh = near_sh(q.par);
    if (nb | kb) {
      const uint32_t old = atomicOr(fw, (nb << psh) | (kb << FAR_SH));
      toN = nb && ((old >> psh) & 0xFFu) == 0u;
      toF = kb && ((old >> FAR_SH) & 0xFFu) == 0u;
    }
    return;
  }
  uint32_t cost = (uint32_t)(ld_cg(q.table + s) >> 32);
  if (cost < q.theta_lo || cost == INF32 || cost > best) {
    atomicAnd(&q.dflag[s >> 3], ~dflag_bit(s, 2u));
  } else if (cost < q.theta_hi) {
    atomicAnd(&q.dflag[s >> 3], ~dflag_bit(s, 2u));
    uint32_t bit = dflag_bit(s, q.par);
    uint32_t old = atomicOr(&q.dflag[s >> 3], bit);
    toN = !(old & bit);
  } else {
    toF = true;
  }
}

// Member item v*8+j -> distance 0; the vertex enters the first near list
// (the caller pushes v if toN).
__device__ void sseed_item(const QDev& q, uint32_t item, bool& toN) {
  uint32_t v = item >> 3, j = item & 7u;
  q.dist[(size_t)v * ROW + j] = 0;
  const uint32_t psh = near_sh(q.par);
  toN = ((atomicOr(q.dist + (size_t)v * ROW + FLAGW, (1u << j) << psh) >> psh) & 0xFFu) == 0u;
}

// Single append (DP seeding only: once per member state of a query).
__device__ __forceinline__ void push_list(const QDev& q, uint32_t* cnt, uint32_t* buf, uint32_t item) {
  uint32_t pos = atomicAdd(cnt, 1u);
  if (pos < q.cap)
    buf[pos] = item;
  else
    atomicExch(&q.ctl->overflow, 1u);
}

// Cost-0 states: every non-empty subset of a member's mask (DPQ.cu:341-358).
// The member item of the lowest group bit of the mask does the seeding.
__device__ void dseed_item(const QDev& q, uint32_t item) {
  uint32_t v = item >> 3, gi = item & 7u;
  uint32_t m = 0;
  for (int t = 0; t < q.k; t++)
    if (q.dist[(size_t)v * 8 + t] == 0) m |= 1u << t;
  if (m == 0 || (uint32_t)(__ffs(m) - 1) != gi) return;
  for (uint32_t sub = m; sub; sub = (sub - 1u) & m) {
    uint32_t s = q.phase == PH_HOP ? ((v << q.k) | sub) * (uint32_t)q.nd : ((v << q.k) | sub);
    // a seed that its bound rules out is no state (a dead vertex has none)
    if (sub != (uint32_t)q.full &&
        !lb_ok(0u, ld_round(q.lbt + ((size_t)v << q.k) + ((uint32_t)q.full ^ sub)), ld_best(q.ctl)))
      continue;
    q.table[s] = pack(0u, 0u);
    if (sub == (uint32_t)q.full) {  // v is in every query group: a cost-0 tree
      atomicMin(&q.ctl->best, 0u);
      atomicMin(&q.ctl->best_full, q.phase == PH_HOP ? (unsigned long long)(v * 8u) : (unsigned long long)v);
      continue;
    }
    uint32_t bit = dflag_bit(s, q.par);
    if (!(atomicOr(&q.dflag[s >> 3], bit) & bit)) push_list(q, &q.ctl->n_near, q.qbuf[q.out_idx], s);
  }
}

// Tour tables of a query, one warp per starting group i: group-to-group
// distances gd[a][b] = min over members of group a of the (capped) distance to
// group b, then
//   P[i][S][j]  cheapest visiting order of S starting at i, ending at j
//   T2[i][S]    min_j P[i][S][j]
// for the subsets S that hold i, and the span table (replaces the host DP of DPQ.cu:409-483 /
// AllPaths, CPUNONHOP.h:269-386).  Each warp works out gd again (a query has
// few members; four of a lane's rows are in flight at once) and keeps it and
// its 2^(k-1) x k table in shared memory: gd[64], Pi[2^(KMAX-1) * KMAX].  A
// chain of dependent layers; one warp for all of it, through global memory,
// took 127 us for k = 6 and 366 us for k = 7; this takes 20 and 35.
constexpr uint32_t TOUR_WORDS = (1u << (KMAX - 1)) * KMAX;
__device__ __noinline__ void tour_warp(const QDev& q, uint32_t i, uint32_t lane, uint32_t* gd, uint32_t* Pi) {
  const uint32_t k = (uint32_t)q.k, K2 = 1u << k;
  const uint32_t* rows = q.D >= 1 ? q.rows[q.D] : q.dist;
  for (uint32_t t = lane; t < 64; t += 32) gd[t] = BIG;
  __syncwarp();
  constexpr int U = 4;
  for (uint32_t t0 = lane; t0 < q.n_members; t0 += 32 * U) {
    uint32_t item[U], r[U][KMAX];
#pragma unroll
    for (int u = 0; u < U; u++) item[u] = t0 + 32 * u < q.n_members ? __ldg(q.members + t0 + 32 * u) : INF32;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (item[u] != INF32) load_row(rows, item[u] >> 3, r[u]);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (item[u] != INF32) {
#pragma unroll
        for (int j = 0; j < KMAX; j++)
          if (j < (int)k) atomicMin(&gd[(item[u] & 7u) * 8u + j], min(r[u][j], q.cap1));
      }
  }
  __syncwarp();
  // With no feasible tree found yet the distance rounds ran without a cap, so
  // an unreachable pair of groups proves there is no solution at all.
  if (i == 0u && lane == 0 && ld_cg(&q.ctl->best) == INF32) {
    bool cut = false;
    for (uint32_t a = 0; a < k; a++)
      for (uint32_t b = 0; b < k; b++)
        if (a != b && gd[a * 8 + b] >= BIG) cut = true;
    if (cut) q.ctl->infeasible = 1u;
  }
  // subsets that hold i, numbered by their other groups
  const uint32_t n = K2 / 2u;
  auto subset = [&](uint32_t c) { return ((c >> i) << (i + 1u)) | (c & ((1u << i) - 1u)) | (1u << i); };
  for (uint32_t t = lane; t < n * k; t += 32) Pi[t] = t == i ? 0u : BIG;
  __syncwarp();
  for (uint32_t size = 1; size < k; size++) {  // other groups visited
    for (uint32_t t = lane; t < n * k; t += 32) {
      const uint32_t c = t / k, l = t - c * k, S = subset(c);
      if ((uint32_t)__popc(c) != size || l == i || !(S >> l & 1u)) continue;
      const uint32_t cp = c ^ (1u << (l < i ? l : l - 1u));
      uint32_t best = BIG;
      for (uint32_t m = S ^ (1u << l); m; m &= m - 1u) {
        const uint32_t j = __ffs(m) - 1;
        best = min(best, sat_add(Pi[cp * k + j], gd[j * 8u + l]));
      }
      Pi[t] = best;
    }
    __syncwarp();
  }
  uint32_t* P = q.tour + (size_t)i * K2 * k;
  uint32_t* T2 = q.tour + (size_t)k * K2 * k + (size_t)i * K2;
  for (uint32_t t = lane; t < n * k; t += 32) {
    const uint32_t c = t / k;
    P[subset(c) * k + (t - c * k)] = Pi[t];
  }
  unsigned short* span = span_table(q);
  for (uint32_t c = lane; c < n; c += 32) {
    const uint32_t S = subset(c);
    uint32_t m = BIG, tour = BIG;
    for (uint32_t l = 0; l < k; l++) {
      m = min(m, Pi[c * k + l]);
      tour = min(tour, sat_add(Pi[c * k + l], l == i ? 0u : min(gd[l * 8u + i], gd[i * 8u + l])));
    }
    T2[S] = m;
    // half the cheapest closed tour of S (the same from each of its groups)
    if ((S & ((1u << i) - 1u)) == 0u) {
      const uint32_t half = (tour + 1u) >> 1;
      span[S] = (unsigned short)(tour >= BIG ? LB_INF : min(half, LB_INF - 1u));
    }
  }
  if (i == 0u && lane == 0) span[0] = 0;
  __syncwarp();
}

// Lower bound on the cost of connecting a vertex (a lane's own, with group
// distances d[], already capped) to every group of X:
//   one-label  max_j d_j                                   (DPQ.cu:182-188)
//   tour lb1   min_{i,j} ceil((d_i + P[i][X][j] + d_j)/2)   (CPUNONHOP.h:448-466)
//   tour lb2   max_i ceil((d_i + T2[i][X] + min_j d_j)/2)   (CPUNONHOP.h:468-472)
// P[i][S][j] = cheapest order of visiting the groups of S starting at i and
// ending at j with group-to-group distances as step costs; T2 = min_j P.  Every
// lane of the warp evaluates the same X, so the tests on it branch alike, the
// table reads are one broadcast, and with the loops unrolled over all groups the
// distances stay in registers.
//   - Each unordered pair {i, j} is visited once, in the order i < j: a tour can be
//     walked either way, so either order's P bounds it (they are equal unless one
//     of two distances between the same groups was cut off above the cap).  A pair
//     (i, i) only exists for X = {i}, where every bound is d_i.
//   - Each term is a sum of three values <= 2^30, which cannot overflow 32
//     bits, and saturation at BIG and the halving are monotone, so both are
//     applied once to the minimum (lb1) or maximum (lb2) instead of per term.
// Against loops over the set bits with the distances in shared memory and both
// orders read: 48 mixed queries on 3M vertices 96.9 -> 92.7 ms, two of k = 6, 7 on
// 54k vertices 3144 -> 3027 us.
__device__ __forceinline__ uint32_t lower_bound_uniform(const uint32_t (&d)[KMAX], int k, uint32_t X,
                                                        const uint32_t* __restrict__ P,
                                                        const uint32_t* __restrict__ T2) {
  const uint32_t K2 = 1u << k;
  uint32_t lb0 = 0, mind = BIG;
#pragma unroll
  for (int j = 0; j < KMAX; j++)
    if (X >> j & 1u) {
      lb0 = max(lb0, d[j]);
      mind = min(mind, d[j]);
    }
  if ((X & (X - 1u)) == 0u) return lb0;  // a single group
  uint32_t m1 = 0xFFFFFFFFu, m2 = 0;
#pragma unroll
  for (int i = 0; i < KMAX; i++)
    if (X >> i & 1u) {
      const uint32_t* Pi = P + ((size_t)i * K2 + X) * k;
#pragma unroll
      for (int j = i + 1; j < KMAX; j++)
        if (X >> j & 1u) m1 = min(m1, d[i] + ld_round(Pi + j) + d[j]);
      m2 = max(m2, d[i] + ld_round(T2 + (size_t)i * K2 + X) + mind);
    }
  const uint32_t lb1 = (min(m1, BIG) + 1u) >> 1;
  const uint32_t lb2 = (min(m2, BIG) + 1u) >> 1;
  return max(lb0, max(lb1, lb2));
}

// Lower-bound table rows: lbt[v][X] = lower_bound_uniform(d(v), X) for every
// subset X (the per-vertex one_label_lb table of the reference,
// DPQ.cu:174-224, with the tour bounds of CPUNONHOP.h:436-496), saturated to
// 16 bits, which only lowers a bound.  A warp first looks 32 consecutive
// vertices over and drops the dead ones, those in no tree of cost at most the
// incumbent:
//   - a tree through v that reaches every group costs at least the bound of
//     (v, all groups);
//   - a vertex that is no member has two branches in a minimal tree: one
//     reaches the farthest group, another reaches some group, so it costs at
//     least the largest plus the smallest distance.
// A dead vertex's row reads "impossible" and no DP state is ever written,
// flagged or queued at it, so its state table and flags stay uninitialised.
// The live ones' are filled here (16-byte stores over runs of neighbouring
// rows), and their bounds are evaluated 32 at a time from a list that carries
// over from task to task: all lanes evaluate the same subset X, so the bound's
// loops over the groups of X branch alike in every lane and the tour-table
// reads are one broadcast per warp.  Issue-bound: the evaluation is some
// k^2 / 4 table reads per subset and vertex, the look-over one row and one
// bound.  Measured against bounds for every vertex and a state table filled
// at admission: six hop-bounded queries on 2^20 vertices 5.5 -> 4.1 ms (their
// starts had differed by launches alone before), 48 of them in a batch 34.9 ->
// 27.2 ms, 48 mixed queries on 3M vertices 226 -> 202 ms.
__device__ __forceinline__ void lb_row(const QDev& q, bool mine, uint32_t v,
                                             uint32_t (&d)[KMAX], uint32_t& dmin, uint32_t& dmax) {
  uint32_t r[KMAX] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
  if (mine) {
    load_row(q.dist, v, r);
    if (q.D >= 0) {
      // a state at v has at least h hops below it, h the hops from v to the
      // nearest member: the missing groups are within D - h hops
      bool member = false, reached = false;
#pragma unroll
      for (int t = 0; t < KMAX; t++) {
        member = member || (t < q.k && r[t] == 0u);
        reached = reached || (t < q.k && r[t] != INF32);
      }
      if (reached && q.D > 0) {
        uint32_t h = 0;
        if (!member)
          for (h = 1; h < q.push_rounds; h++) {
            load_row(q.rows[h], v, r);
            bool any = false;
#pragma unroll
            for (int t = 0; t < KMAX; t++) any = any || (t < q.k && r[t] != INF32);
            if (any) break;
          }
        if (h < (uint32_t)q.D) {
          load_row(q.rows[(uint32_t)q.D - h], v, r);
        } else {
#pragma unroll
          for (int t = 0; t < KMAX; t++) r[t] = INF32;  // no hop left, and v is no member
        }
      }
    }
  }
  dmin = BIG;
  dmax = 0u;
#pragma unroll
  for (int j = 0; j < KMAX; j++) {
    d[j] = min(r[j], q.cap1);
    if (j < q.k) {
      dmin = min(dmin, d[j]);
      dmax = max(dmax, d[j]);
    }
  }
}

// Bounds of the first `cnt` (at most 32) listed vertices; the rest move up.
__device__ void lb_eval(const QDev* qd, uint32_t cnt, uint32_t lane, LbScratch& lb) {
  const QDev& q = qd[lb.slot];
  const int k = q.k;
  const uint32_t K2 = 1u << k;
  const uint32_t* P = q.tour;
  const uint32_t* T2 = q.tour + (size_t)k * K2 * k;
  const bool mine = lane < cnt;
  const uint32_t v = mine ? lb.v[lane] : 0u;
  uint32_t d[KMAX], dmin, dmax;
  lb_row(q, mine, v, d, dmin, dmax);
  unsigned short* out = q.lbt + ((size_t)v << k);
  for (uint32_t x0 = 0; x0 < K2; x0 += 8u) {
    unsigned long long pk[2] = {0, 0};  // eight entries
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll 1
      for (uint32_t e = 0; e < 4u; e++) {
        const uint32_t X = x0 + 4u * h + e;
        uint32_t bound = 0;
        if (X != 0u && X < K2) bound = lower_bound_uniform(d, k, X, P, T2);
        const uint32_t ent = bound >= BIG ? LB_INF : min(bound, LB_INF - 1u);
        pk[h] |= (unsigned long long)ent << (16u * e);
      }
    if (mine) {
      if (K2 >= 8u) {
        *reinterpret_cast<ulonglong2*>(out + x0) = make_ulonglong2(pk[0], pk[1]);
      } else {
        for (uint32_t X = 0; X < K2; X++) out[X] = (unsigned short)(pk[0] >> (16u * X));
      }
    }
  }
  const uint32_t left = lb.n - cnt;  // at most 31
  const uint32_t mv = lane < left ? lb.v[cnt + lane] : 0u;
  __syncwarp();
  if (lane < left) lb.v[lane] = mv;
  if (lane == 0) lb.n = left;
  __syncwarp();
}

// What is left on the warp's list, at the end of its tasks (every lane).
__device__ __forceinline__ void lb_flush(const QDev* qd, uint32_t lane, LbScratch& lb) {
  __syncwarp();
  if (lb.n) lb_eval(qd, lb.n, lane, lb);
}

__device__ void lbt_rows32(const QDev* qd, const uint32_t* __restrict__ pre, int nslots, uint32_t n_lb,
                           uint32_t task, uint32_t lane, LbScratch& lb) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t it = task * 32u + lane;
  const bool valid = it < n_lb;
  const uint32_t slot = valid ? find_slot_s(pre, nslots, it) : 0xFFFFFFFFu;
  const uint32_t prev = __shfl_up_sync(FULL, slot, 1);
  unsigned runs = __ballot_sync(FULL, valid && (lane == 0u || prev != slot));
  while (runs) {
    const uint32_t i0 = (uint32_t)(__ffs(runs) - 1);
    runs &= runs - 1u;
    const uint32_t si = __shfl_sync(FULL, slot, i0);
    const bool mine = valid && slot == si;
    const QDev& q = qd[si];
    const int k = q.k;
    const uint32_t K2 = 1u << k;
    if (lb.n != 0u && lb.slot != si) lb_flush(qd, lane, lb);
    const uint32_t v = mine ? q.lb_off + (it - pre[si]) : 0u;
    uint32_t d[KMAX], dmin, dmax;
    lb_row(q, mine, v, d, dmin, dmax);
    const uint32_t best = ld_best(q.ctl);
    bool live = mine && dmax < BIG && (dmin == 0u || dmin + dmax <= best);
    if (__any_sync(FULL, live)) {
      const uint32_t all = lower_bound_uniform(d, k, K2 - 1u, q.tour, q.tour + (size_t)k * K2 * k);
      live = live && all < BIG && all <= best;
    }
    const unsigned mm = __ballot_sync(FULL, mine), am = __ballot_sync(FULL, live);
    // every row of the run "impossible" (entry 0, the empty set, is 0); the
    // live ones are written again with their bounds
    const uint32_t v0 = __shfl_sync(FULL, v, i0), nrow = __popc(mm);
    if (K2 >= 8u) {
      uint4* rows = reinterpret_cast<uint4*>(q.lbt + ((size_t)v0 << k));
      const uint32_t per = K2 / 8u;
      for (uint32_t i = lane; i < nrow * per; i += 32u)
        rows[i] = make_uint4((i & (per - 1u)) ? INF32 : 0xFFFF0000u, INF32, INF32, INF32);
    } else if (mine) {
      for (uint32_t X = 0; X < K2; X++) q.lbt[((size_t)v << k) + X] = (unsigned short)(X ? LB_INF : 0u);
    }
    // state table (and flags, where a vertex's are whole words) of the live rows
    for (unsigned left = am; left;) {
      const uint32_t a = (uint32_t)(__ffs(left) - 1);
      const uint32_t len = __popc(left & ~(left + (1u << a)));  // consecutive set bits from a
      const uint32_t va = __shfl_sync(FULL, v, a);
      uint4* tab = reinterpret_cast<uint4*>(q.table + (size_t)va * q.WT);
      for (uint32_t i = lane; i < len * q.WT / 2u; i += 32u) tab[i] = make_uint4(INF32, INF32, INF32, INF32);
      if (K2 >= 8u) {
        uint32_t* fl = q.dflag + (size_t)va * (q.WT / 8u);
        for (uint32_t i = lane; i < len * q.WT / 8u; i += 32u) fl[i] = 0u;
      }
      left &= left + (1u << a);
    }
    if (am) {
      if (live) lb.v[lb.n + __popc(am & ((1u << lane) - 1u))] = v;
      __syncwarp();
      if (lane == 0) {
        lb.n += __popc(am);
        lb.slot = si;
      }
    }
    __syncwarp();
    if (lb.n >= 32u) lb_eval(qd, 32u, lane, lb);
  }
}

// Weight of arc (a -> b): the warp scans a's weight-sorted adjacency, 32
// arcs per step (hub lists hold tens of thousands of arcs).  Every lane calls
// it with the same a and b.
__device__ uint32_t arc_weight_warp(const GraphDev& g, uint32_t a, uint32_t b, uint32_t lane) {
  const uint32_t x0 = __ldg(g.beg + a), x1 = __ldg(g.beg + a + 1);
  for (uint32_t base = x0; base < x1; base += 32u) {
    const uint32_t x = base + lane;
    uint32_t w = INF32;
    if (x < x1) {
      const uint2 arc = __ldg(g.adj + x);
      if (arc.x == b) w = arc.y;
    }
    const unsigned hit = __ballot_sync(0xFFFFFFFFu, w != INF32);
    if (hit) return __shfl_sync(0xFFFFFFFFu, w, __ffs(hit) - 1);
  }
  return INF32;
}

// Whether the list [lo, hi), sorted by (weight, neighbour), holds an arc to b of
// weight w: binary search by one lane.
__device__ __forceinline__ bool has_arc(const GraphDev& g, uint32_t lo, uint32_t hi, uint32_t b, uint32_t w) {
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    const uint2 arc = __ldg(g.adj + mid);
    if (arc.y == w && arc.x == b) return true;
    if (arc.y < w || (arc.y == w && arc.x < b))
      lo = mid + 1u;
    else
      hi = mid;
  }
  return false;
}

// Follow parent words from the best full state, emitting (u, v, w) edges.  Run
// by one warp: every lane holds one state still to follow.  A state's subset
// is non-empty and a merge splits it into two disjoint parts, so at most k
// lanes are ever busy; each step is one trip to the state table for all of
// them, where a single walk took one per state.  An edge's weight is the
// difference of its two states' costs unless the lower one has been lowered
// since (only possible beyond what the bounds let through): afterwards each
// lane checks its edges against the graph, by binary search of the endpoint
// with fewer arcs, and the rare rest is looked up by the whole warp.  A chain
// of dependent loads; measured on a 2^20-vertex R-MAT graph, whose trees run
// through hubs: 0.264 -> 0.022 ms for the round with the slowest extraction of
// a batch.
__device__ __noinline__ void extract_warp(const QDev& q, const GraphDev& g, uint32_t lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  QCtl* ctl = q.ctl;
  const unsigned long long bf = __ldcg(&ctl->best_full);
  if (bf == INF64) {
    if (lane == 0) {
      ctl->status = 1;
      ctl->n_edges = 0;
    }
    return;
  }
  const int k = q.k;
  const bool hop = q.phase == PH_HOP;
  const uint32_t nd = hop ? (uint32_t)q.nd : 1u;
  const uint32_t payload = (uint32_t)bf, root = hop ? payload >> 3 : payload;
  uint32_t s = ((root << k) | (uint32_t)q.full) * nd + (hop ? (payload & 7u) : 0u);
  bool act = lane == 0;
  uint32_t ne = 0, status = 0, steps = 0;
  uint32_t edge = INF32, c_edge = 0;  // the edge that led here: its number and its upper state's cost
  const uint32_t max_steps = 4u * g.V + 64u;
  while (__any_sync(FULL, act)) {
    const unsigned long long e = act ? __ldcg(q.table + s) : 0ull;
    const uint32_t cost = (uint32_t)(e >> 32), par = (uint32_t)e, type = par >> 30;
    const uint32_t d = s % nd, vp = s / nd, v = vp >> k, p = vp & ((1u << k) - 1u);
    if (act && edge < q.max_edges) q.out_edges[3 * edge + 2] = c_edge - cost;
    const bool grow = act && type == 1u, merge = act && type == 2u;
    const uint32_t p1 = par & 0xFFu, p2 = p ^ p1;
    const bool bad = act && (cost == INF32 || type == 3u || (grow && hop && d == 0u) ||
                             (merge && (p1 == 0u || p2 == 0u || (p1 & ~p) != 0u)));
    if (++steps > max_steps || __any_sync(FULL, bad)) {
      status = 2;
      break;
    }
    const unsigned gm = __ballot_sync(FULL, grow), mm = __ballot_sync(FULL, merge);
    edge = INF32;
    uint32_t s2 = 0;
    if (grow) {
      const uint32_t u = par & 0x3FFFFFFFu;
      edge = ne + __popc(gm & ((1u << lane) - 1u));
      c_edge = cost;
      if (edge < q.max_edges) {
        q.out_edges[3 * edge] = u;
        q.out_edges[3 * edge + 1] = v;
      }
      s = ((u << k) | p) * nd + (hop ? d - 1u : 0u);
    } else if (merge) {
      s = ((v << k) | p1) * nd + (hop ? (par >> 8) & 7u : 0u);
      s2 = ((v << k) | p2) * nd + (hop ? (par >> 11) & 7u : 0u);
    }
    ne += __popc(gm);
    act = grow || merge;
    // the second parts go to the free lanes, in order
    const unsigned idle = ~__ballot_sync(FULL, act);
    const uint32_t r = __popc(idle & ((1u << lane) - 1u));
    const bool take = !act && r < (uint32_t)__popc(mm);
    const uint32_t from = take ? __fns(mm, 0, (int)r + 1) : lane;
    const uint32_t got = __shfl_sync(FULL, s2, (int)from);
    if (take) {
      s = got;
      act = true;
    }
  }
  __syncwarp();
  if (status == 0) {
    const uint32_t n = min(ne, q.max_edges);
    for (uint32_t i0 = 0; i0 < n; i0 += 32u) {
      const uint32_t i = i0 + lane;
      bool miss = false;
      uint32_t a = 0, b = 0;
      if (i < n) {
        a = q.out_edges[3 * i];
        b = q.out_edges[3 * i + 1];
        const uint32_t w = q.out_edges[3 * i + 2];
        const uint32_t a0 = __ldg(g.beg + a), a1 = __ldg(g.beg + a + 1), b0 = __ldg(g.beg + b), b1 = __ldg(g.beg + b + 1);
        miss = a1 - a0 <= b1 - b0 ? !has_arc(g, a0, a1, b, w) : !has_arc(g, b0, b1, a, w);
      }
      for (unsigned m = __ballot_sync(FULL, miss); m; m &= m - 1u) {
        const int l = __ffs(m) - 1;
        const uint32_t w = arc_weight_warp(g, __shfl_sync(FULL, b, l), __shfl_sync(FULL, a, l), lane);
        if (lane == (uint32_t)l) q.out_edges[3 * i + 2] = w;
      }
    }
  }
  if (q.host_edges != nullptr && status == 0 && ne <= min(HOST_EDGES, q.max_edges)) {
    __syncwarp();
    for (uint32_t i = lane; i < 3u * ne; i += 32u) q.host_edges[i] = q.out_edges[i];
  }
  if (lane == 0) {
    ctl->status = status;
    ctl->n_edges = ne;
    ctl->root = root;
  }
}

// ---------------------------------------------------------------------------
// Admission of the queries staged for a block of rounds, one launch for all of
// them: blockIdx.y is the query, whose record in `stage` (at off[y]) is its
// descriptor, its control block and its member items, each 64-byte aligned.
// Descriptor and control block go to the query's slot and the members to its
// workspace; the distance rows that the rounds will read are set to "unknown"
// (words 0..6 all ones) with no group pending (word 7 zero), and, for k < 3, the
// state flags to zero (a vertex's flags are not whole words then).  The state
// table, up to
// 7.7 GB at 3M vertices, is not touched: the bound-row pass fills the rows of the
// vertices that can hold a state.  Bound by its HBM writes for large graphs (32
// bytes a vertex and buffer) and by its launch for small ones.  A kernel and three copies
// for each query, two more copies for each finished one and a wait for the block
// launched ahead, against this and trees written to the host by extraction: a
// 90-query batch on 170k vertices 19.8 -> 17.4 ms, 48 hop-bounded queries on
// 2^20 vertices 4.07 -> 3.18 ms, one query on 10k vertices 493 -> 410 us.
// ---------------------------------------------------------------------------
__device__ void init_rows(const QDev& q, const uint32_t* members, size_t tid, size_t stride) {
  const uint4 ones = make_uint4(INF32, INF32, INF32, INF32);
  const uint4 tail = make_uint4(INF32, INF32, INF32, 0u);
  uint4* dist = reinterpret_cast<uint4*>(q.dist);
  uint4* next = reinterpret_cast<uint4*>(q.dist_nx);
  // Unbounded queries have one buffer.  Of a hop-bounded query's two, the first is
  // read and written at the members only when there is one relaxed round
  // (D = 1..3), and the second not at all when there is none (D = 0).  Measured
  // against both buffers always: six queries (D = 2..4) one at a time on 2^20
  // vertices 1457 -> 1417 us, 48 in a batch 3.01 -> 2.86 ms; on 10k vertices the
  // same.
  const bool first = q.push_rounds != 1u || members == nullptr;
  const bool second = next != dist && q.push_rounds != 0u;
  for (size_t i = tid; i < 2 * (size_t)q.nv; i += stride) {
    const uint4 x = (i & 1u) ? tail : ones;
    if (first) dist[i] = x;
    if (second) next[i] = x;
  }
  if (!first)
    for (size_t i = tid; i < q.n_members; i += stride) {
      uint4* row = dist + 2 * (size_t)(members[i] >> 3);
      row[0] = ones;
      row[1] = tail;
    }
  if (q.k < 3)
    for (size_t i = tid; i < ((size_t)q.nv * q.WT + 7) / 8; i += stride) q.dflag[i] = 0u;
}

__global__ void __launch_bounds__(256) k_admit(const unsigned char* __restrict__ stage,
                                               const uint32_t* __restrict__ off, QDev* qd, QCtl* ctl, RoundDesc* rd) {
  const unsigned char* rec = stage + off[blockIdx.y];
  const QDev& q = *reinterpret_cast<const QDev*>(rec);
  const unsigned char* rc = rec + (sizeof(QDev) + 63) / 64 * 64;
  const uint32_t* rm = reinterpret_cast<const uint32_t*>(rc + (sizeof(QCtl) + 63) / 64 * 64);
  const size_t stride = (size_t)gridDim.x * blockDim.x, tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.x == 0) {
    const uint32_t slot = (uint32_t)(q.ctl - ctl);
    for (uint32_t i = threadIdx.x; i < sizeof(QDev) / 8; i += blockDim.x)
      reinterpret_cast<unsigned long long*>(qd + slot)[i] = reinterpret_cast<const unsigned long long*>(rec)[i];
    for (uint32_t i = threadIdx.x; i < sizeof(QCtl) / 8; i += blockDim.x)
      reinterpret_cast<unsigned long long*>(q.ctl)[i] = reinterpret_cast<const unsigned long long*>(rc)[i];
    // one more for the next control step to look at, beside those that the last
    // one left running (the distance windows go by the number of live queries)
    if (threadIdx.x == 0) atomicAdd(&rd->n_live, 1u);
  }
  uint32_t* members = const_cast<uint32_t*>(q.members);
  for (size_t i = tid; i < q.n_members; i += stride) members[i] = rm[i];
  init_rows(q, rm, tid, stride);
}

// The same for the allocation-free query, whose descriptor and control block are
// in place already.  Its members may still be on their way (the copy overlaps
// this: waiting for it cost 2 us of 548), so all of the first buffer is set.
__global__ void __launch_bounds__(256) k_init_workspace(const QDev* qd) {
  init_rows(*qd, nullptr, (size_t)blockIdx.x * blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x);
}

// ---------------------------------------------------------------------------
// Control: one thread per slot.  Absorbs the previous round's counters,
// decides this round's action, and publishes per-type item counts as
// exclusive prefix sums over slots (pre[t][0..nslots]).
// ---------------------------------------------------------------------------
// What a control step reads of a query's control block, loaded at once: read
// where they are needed, the words would cost a trip to L2 each.
struct CtlIn {
  uint32_t best, infeasible, center, n_near, n_far, n_far2, overflow, deferred, status, cancel;
  unsigned long long best_full;
  __device__ explicit CtlIn(const QCtl& c)
      : best(c.best), infeasible(c.infeasible), center(c.center), n_near(c.n_near), n_far(c.n_far), n_far2(c.n_far2),
        overflow(c.overflow), deferred(c.deferred), status(c.status), cancel(c.cancel), best_full(c.best_full) {}
};

// After a distance round of a hop-bounded query: the passes over its rows.
__device__ __forceinline__ void hop_round_over(QRun& q) {
  if (q.D < 2) return;
  if (q.hops == q.center_h + 1u) q.center_done = 1u;  // the pass ran during this round
  if (q.hops < (uint32_t)q.D &&
      (q.hops + 2u <= q.push_rounds || q.hops == q.star_h || q.hops == q.center_h))
    q.rows_h = q.hops;
}

__device__ __forceinline__ void absorb(QRun& q, QDev& qg, QCtl& c, const CtlIn& in) {
  if (in.cancel) {  // the host withdrew the request
    q.st = J_DONE;
    c.final_status = 12;  // GST_CANCELLED
    c.done = 1;
    return;
  }
  if (in.overflow) {
    q.st = J_DONE;
    c.final_status = 6;  // GST_QUEUE_OVERFLOW
    c.done = 1;
    return;
  }
  int t;
  q.rows_h = 0;  // a pass over rows scheduled last round has run
  switch (q.act) {
    case A_SSEED:
      t = q.in_idx; q.in_idx = q.out_idx; q.out_idx = t;
      q.n_in = in.n_near;
      q.n_far = 0;
      q.st = J_SSSP;
      if (q.D >= 0) {  // the lists of the exact rounds are kept: list h is qbuf[h]
        q.in_idx = 0;
        q.out_idx = 1;
        q.n_list[0] = in.n_near;
      }
      break;
    case A_WORK:
      t = q.in_idx; q.in_idx = q.out_idx; q.out_idx = t;
      q.n_in = in.n_near;
      q.n_far = in.n_far;
      q.par ^= 1u;  // producers of the round flagged the next items with the other parity
      if (q.st == J_SSSP) {
        q.hops++;
        if (q.D >= 0) {  // exact rounds: the rows just written become the current ones
          uint32_t* x = q.dist;
          q.dist = q.dist_nx;
          q.dist_nx = x;
          q.in_idx = (int32_t)q.hops;
          q.out_idx = (int32_t)min(q.hops + 1u, 3u);
#pragma unroll
          for (uint32_t b = 1; b <= 3u; b++)
            if (b == q.hops) q.n_list[b] = in.n_near;
          // the last two relaxed rounds' rows stay in the two buffers, earlier
          // ones are copied to their own while the next round runs
          if (q.hops + 2u > q.push_rounds) qg.rows[q.hops] = q.dist;
        }
        hop_round_over(q);
      }
      break;
    case A_PULL:
      q.hops++;
      hop_round_over(q);
      break;
    case A_SPLIT:
      t = q.in_idx; q.in_idx = q.out_idx; q.out_idx = t;
      t = q.far_idx; q.far_idx = q.far2_idx; q.far2_idx = t;
      q.n_in = in.n_near;
      q.n_far = in.n_far2;
      break;
    case A_TOUR:
      q.st = in.infeasible ? J_EXTRACT : J_LB;  // disconnected groups: straight to "no solution"
      break;
    case A_LB:
      // the bound table is filled in chunks of LB_CHUNK entries per round
      q.lb_off += min(q.nv - q.lb_off, LB_CHUNK);
      if (q.lb_off >= q.nv) q.st = J_DPSEED;
      break;
    case A_DSEED:
      t = q.in_idx; q.in_idx = q.out_idx; q.out_idx = t;
      q.n_in = in.n_near;
      q.n_far = 0;
      q.st = J_DP;
      break;
    case A_EXTRACT:
      q.st = J_DONE;
      c.final_status = in.status == 1 ? 1u : (in.status != 0 ? 8u : 0u);  // NO_SOLUTION / INTERNAL / OK
      c.done = 1;
      break;
    default:
      break;
  }
  if (q.act != A_NONE) atomicAdd(&c.stat[ST_ROUNDS], 1ull);
  q.act = A_NONE;
}

// End of a hop-bounded query's distance rounds.  Every tree of hop diameter
// <= D has a vertex with all its vertices within ceil(D/2) hops (a centre of
// the tree), so when the exact rows of that many hops showed no vertex with
// every group in reach, the query has no solution.
__device__ __forceinline__ void hop_rounds_done(QRun& q, QDev& qg, QCtl& c, const CtlIn& in) {
  if (q.center_h != 0u && q.center_done && in.center == 0u && in.best == INF32) c.infeasible = 1u;
  q.dist_nx = q.dist;
  // rounds that converged early: the rows over more hops are the last ones
  for (uint32_t b = q.hops + 1u; b <= (uint32_t)q.D; b++) qg.rows[b] = q.dist;
}

// Upper end of the near window that starts at lo.
//
// DP, exact query: everything up to the incumbent in one window (without an
// incumbent, 16 widths).  A window's end costs a split round, and re-expanding
// a state whose cost drops later costs little next to the incumbent's pruning:
// windows of 8 / 64 / 128 gave 3570 / 2016 / 1857 us for four hop-bounded
// queries on 10k vertices, 5990 / 4446 / 4287 us for two of k = 6, 7 on 54k,
// and 19.9 / 19.0 / 18.9 ms for a 90-query batch on 170k.  Progressive queries
// keep the narrow windows: the window's lower end is the bound they stop on.
//
// Distances: narrow while there is no incumbent, because nothing else bounds
// what is relaxed then (windows of 64 from the start cost six queries on 170k
// vertices 5615 -> 6075 us); four times as wide after a window of at most
// LIGHT_ITEMS items over all live queries, whose rounds are launch and latency;
// and the rest in one window once an incumbent caps them.  Only arcs that lead
// below the reach, two widths, are relaxed at first: without an incumbent a
// vertex's heavy arcs lead to distances that almost never matter.  Should the
// incumbent turn out beyond it (or none be found), every vertex reached relaxes
// all its arcs once more.  The reach took 90 queries on 170k vertices from 15.5 to
// 14.8 ms and 48 mixed ones on 3M from 104 to 96; relaxing below the window's own
// end only, with a look at every vertex for each new window, halved the arcs but
// cost the serving mixes 2-6%.  LIGHT_ITEMS is some four items a warp of the whole
// GPU; a quarter of it costs two queries of k = 6, 7 on 54k vertices 1% (2942 us
// against 2915), four times as many changes nothing.
constexpr uint32_t LIGHT_ITEMS = 16384;
__device__ __forceinline__ uint32_t window_end(const QRun& q, uint32_t lo, uint32_t best, uint32_t limit) {
  uint32_t w = q.delta;
  if (q.phase == PH_SSSP) {
    if (best != INF32 && limit >= lo) w = max(w, limit - lo + 1u);
  } else if (q.ratio_num == 0u) {
    w = best == INF32 ? (w > BIG / 16u ? BIG : 16u * w) : max(w, (best > lo ? best - lo : 0u) + 1u);
  }
  return lo + min(w, INF32 - lo);
}

__device__ __forceinline__ void decide(QRun& q, QDev& qg, QCtl& c, const CtlIn& in, uint32_t n_live) {
  for (int guard = 0; guard < 8; guard++) {
    switch (q.st) {
      case J_INIT:
        q.phase = PH_SSSP;
        q.theta_lo = 0;
        // a hop-bounded query runs its distance rounds as Bellman-Ford rounds
        // (one window holding everything): after D rounds every path of at
        // most D hops has been relaxed
        q.theta_hi = q.D >= 0 ? INF32 : q.delta_sssp;
        q.reach = q.D >= 0 ? INF32 : (q.delta_sssp > BIG / 2u ? INF32 : 2u * q.delta_sssp);
        q.delta = q.delta_sssp;
        q.win_items = 0;
        q.hops = 0;
        c.n_near = 0;
        q.act = A_SSEED;
        return;
      case J_SSSP:
      case J_DP: {
        if (q.st == J_SSSP && q.D >= 0 && q.hops >= (uint32_t)q.D) {
          // hop-bounded distances: d_j(v) <= the cheapest path of at most D
          // hops from group j to v, INF if there is none.  Every path of the
          // final tree has at most D hops, so these are valid lower bounds,
          // and an unreached vertex cannot join a group
          q.cap1 = BIG;
          hop_rounds_done(q, qg, c, in);
          q.st = J_TOUR;
          continue;
        }
        if (q.st == J_SSSP && q.D >= 0 && q.hops >= q.push_rounds && (q.hops > q.push_rounds || q.n_in > 0)) {
          q.act = A_PULL;
          return;
        }
        if (q.st == J_DP && q.phase == PH_DP && q.ratio_num != 0u && in.best_full != INF64) {
          // Progressive exit (CPUNONHOP.h:730-755, in exact integer
          // arithmetic).  Every state of cost below lo (theta_lo, or theta_hi
          // once the window's near list is empty) has been expanded at its
          // final cost.  The optimum's derivation has no state costlier than
          // the optimum, so an optimum below lo would already be recorded:
          // opt >= min(best_full, lo).  Stop once best_full <= ratio * lo.
          const unsigned long long lo = q.n_in > 0 ? q.theta_lo : q.theta_hi;
          const unsigned long long bf = in.best_full >> 32;
          if (bf * q.ratio_den <= lo * q.ratio_num) {
            c.early = 1u;
            c.lb_exit = (uint32_t)(bf < lo ? bf : lo);
            q.st = J_EXTRACT;
            continue;
          }
        }
        if (q.n_in > 0) {
          q.win_items = min(q.win_items + min(q.n_in, BIG), BIG);
          c.n_near = 0;
          c.n_far = q.n_far;
          q.act = A_WORK;
          return;
        }
        uint32_t next_lo = q.theta_hi;
        // distance rounds only matter up to cap(best); DP rounds up to best
        unsigned long long limit = in.best;
        if (q.st == J_SSSP && in.best != INF32) limit = (unsigned long long)in.best * q.cap_num / q.cap_den;
        // arcs beyond the reach are left: what comes next is every vertex again
        const bool again = q.st == J_SSSP && q.n_far == 0 && in.deferred != 0u && limit >= q.reach;
        bool exhausted = (q.n_far == 0 && !again) || next_lo > limit;
        q.rescan = 0;
        if (!exhausted) {
          if (again) {
            q.rescan = 1;
            q.reach = INF32;
            c.deferred = 0;
          }
          if (q.st == J_SSSP && (unsigned long long)q.win_items * n_live <= LIGHT_ITEMS && q.delta < BIG / 4u)
            q.delta *= 4u;
          q.win_items = 0;
          q.theta_lo = next_lo;
          q.theta_hi = window_end(q, next_lo, in.best, (uint32_t)limit);
          if (q.st == J_SSSP) q.theta_hi = min(q.theta_hi, q.reach);
          c.n_near = 0;
          c.n_far2 = 0;
          q.act = A_SPLIT;
          return;
        }
        if (q.st == J_SSSP) {
          if (q.D >= 0) hop_rounds_done(q, qg, c, in);  // its rounds converged before D
          // every distance below theta_hi is exact and every distance <=
          // cap(best), which is below the reach if arcs were left, was
          // discovered; unknown ones are >= min(theta_hi, cap+1)
          unsigned long long b1 = in.best == INF32 ? (unsigned long long)INF32 : limit + 1;
          unsigned long long cap1 = q.n_far == 0 ? b1 : (q.theta_hi < b1 ? q.theta_hi : b1);
          q.cap1 = (uint32_t)(cap1 < BIG ? cap1 : BIG);
          q.st = J_TOUR;
          continue;
        }
        q.st = J_EXTRACT;
        continue;
      }
      case J_TOUR:
        q.act = A_TOUR;
        return;
      case J_LB:
        q.act = A_LB;
        return;
      case J_DPSEED:
        q.phase = q.D < 0 ? PH_DP : PH_HOP;
        q.theta_lo = 0;
        q.delta = q.delta_dp;
        q.theta_hi = window_end(q, 0u, in.best, in.best);
        q.in_idx = 0;
        q.out_idx = 1;
        q.far_idx = 2;
        q.far2_idx = 3;
        q.n_in = 0;
        q.n_far = 0;
        c.n_near = 0;
        c.n_far = 0;
        q.act = A_DSEED;
        return;
      case J_EXTRACT:
        q.act = A_EXTRACT;
        return;
      default:
        q.act = A_NONE;
        return;
    }
  }
}

// Bounds of a small round, per warp of the cluster (k_small).  Half and twice each,
// against these: one k = 4 query on 10k vertices through the allocation-free call
// (no arc chunks, launches not in a graph) 551 and 533 us for SMALL_ARCS, 554 and
// 531 for SMALL_DP, 556 and 533 for SMALL_TASKS (532); four hop-bounded ones there
// 1158 and 1181, 1176 and 1169, 1190 and 1164 (1166); two of k = 6, 7 on 54k
// vertices 2953 and 2873, 2927 and 2899, 2902 and 2915 (2915); SMALL_CHUNKS, and
// all four on 170k and 2^20 vertices, within 1.1%.
constexpr uint32_t SMALL_ARCS = 256, SMALL_DP = 2, SMALL_TASKS = 2, SMALL_CHUNKS = 4;

// Shared memory of one control step.
struct CtlSmem {
  uint32_t wsum[32][NT];  // per-warp inclusive totals, then their scan
  uint32_t carry[NT];     // items of the slots in earlier chunks
  uint32_t live_cnt, used_hi;
};

// The round's description staged in shared memory (every thread of the block
// calls it, a barrier follows): a task reads a dozen of its words, one after
// another, and from L2 each would cost a trip.  `rd` beside a staged copy `sd`
// is the global one, whose n_big the tasks count up.
constexpr uint32_t RD_WORDS = sizeof(RoundDesc) / 4;
static_assert(sizeof(RoundDesc) % 4 == 0, "copied by words");
__device__ __forceinline__ void stage_rd(RoundDesc& sd, const RoundDesc* rd) {
  for (uint32_t i = threadIdx.x; i < RD_WORDS; i += blockDim.x)
    reinterpret_cast<uint32_t*>(&sd)[i] = __ldcg(reinterpret_cast<const uint32_t*>(rd) + i);
}

// One control step over slots [0, nslots) by all threads of one block
// (blockDim.x a multiple of 32, at most 1024).  Slots go in chunks of
// blockDim.x; the per-type prefixes carry from one chunk to the next, so any
// block size gives the same prefixes.  Fewer than 32 slots are one warp's
// work, without the block-wide scan and its barriers.
//
// small_warps: warps of the cluster that runs small rounds itself (0: none).
// A round that is small for them is laid out for them and marked small.
// sd: the block's staged copy of the round description; on return it holds
// the new one, which has been written to *rd.
__device__ void control_step(QDev* qd, QCtl* ctl, int nslots, RoundDesc* rd, uint32_t* pre, CtlSmem& sm, RoundDesc& sd,
                             uint32_t small_warps = 0) {
  const int tid = threadIdx.x, B = blockDim.x;
  const uint32_t lane = tid & 31, wid = tid >> 5, nw = (uint32_t)B >> 5;
  stage_rd(sd, rd);
  if (tid == 0) sm.live_cnt = sm.used_hi = 0;
  if (tid < NT) sm.carry[tid] = 0;
  __syncthreads();
  if (sd.slot_hi != 0u) nslots = min(nslots, (int)sd.slot_hi);
  const bool one_warp = nslots < 32;
  for (int base = 0; base <= nslots; base += B) {
    if (one_warp && wid != 0u) break;
    const int s = base + tid;
    uint32_t cnt[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) cnt[t] = 0;
    if (s < nslots) {
      // (a free slot's words are loaded too: its state alone first would put
      // another trip to L2 in front of every live one's)
      QDev& qg = qd[s];
      QRun q = qg;
      QCtl& c = ctl[s];
      const CtlIn in(c);
      if (q.st != J_FREE) atomicMax(&sm.used_hi, (uint32_t)s + 1u);
      if (q.st != J_FREE && q.st != J_DONE) {
        absorb(q, qg, c, in);
        if (q.st != J_DONE) decide(q, qg, c, in, sd.n_live);
        const uint32_t n01 = q.n_list[0] + q.n_list[1], n012 = n01 + q.n_list[2];
        switch (q.act) {
          case A_SSEED:
          case A_DSEED: cnt[T_ITEM] = q.n_members; break;
          case A_SPLIT: cnt[T_ITEM] = q.rescan ? q.nv : q.n_far; break;
          case A_PULL: {  // round hops + 1: the lists 0 .. D - (hops + 1)
            const uint32_t h = (uint32_t)q.D - q.hops - 1u;
            cnt[T_PULL] = h == 0u ? q.n_list[0] : (h == 1u ? n01 : (h == 2u ? n012 : n012 + q.n_list[3]));
            break;
          }
          case A_TOUR: cnt[T_TOUR] = (uint32_t)qg.k; break;
          case A_LB: cnt[T_LB] = min(q.nv - q.lb_off, LB_CHUNK); break;
          case A_EXTRACT: cnt[T_EXTRACT] = 1; break;
          case A_WORK:
            cnt[q.phase == PH_SSSP ? T_SSSP : (q.phase == PH_DP ? T_DP : T_HOP)] = q.n_in;
            break;
          default: break;
        }
        // the pass over the rows of round rows_h: a copy of all of them, or a
        // look at the vertices within push_rounds hops of a member
        if (q.rows_h)
          cnt[T_ROWS] = q.rows_h + 2u <= q.push_rounds
                            ? q.nv
                            : (q.push_rounds == 1u ? n01 : (q.push_rounds == 2u ? n012 : n012 + q.n_list[3]));
        if (q.st != J_DONE) atomicAdd(&sm.live_cnt, 1u);
        static_cast<QRun&>(qg) = q;
      }
    }
    // exclusive scan over the chunk's slots, per task type
    uint32_t incl[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) {
      uint32_t x = cnt[t];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      incl[t] = x;
      if (lane == 31) sm.wsum[wid][t] = x;
    }
    if (one_warp) {
#pragma unroll
      for (int t = 0; t < NT; t++) {
        if (s <= nslots) pre[t * (MAX_SLOTS + 1) + s] = incl[t] - cnt[t];
        if (lane == 31) sm.carry[t] = incl[t];
      }
      break;
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
      for (int t = 0; t < NT; t++) {
        uint32_t x = lane < nw ? sm.wsum[lane][t] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
          if (lane >= (uint32_t)o) x += y;
        }
        sm.wsum[lane][t] = x;  // inclusive over warps
      }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < NT; t++) {
      uint32_t before = sm.carry[t] + (wid ? sm.wsum[wid - 1][t] : 0u) + incl[t] - cnt[t];
      if (s <= nslots) pre[t * (MAX_SLOTS + 1) + s] = before;
    }
    __syncthreads();  // carry and wsum read by every thread
    if (tid < NT) sm.carry[tid] += sm.wsum[nw - 1][tid];
    __syncthreads();
  }
  __syncwarp();
  if (tid == 0) {
    const unsigned long long n_sssp = sm.carry[T_SSSP];
    const unsigned long long n_dp = (unsigned long long)sm.carry[T_DP] + sm.carry[T_HOP];
    // A small round: at most SMALL_ARCS arcs a warp of the cluster at the
    // graph's average degree, SMALL_DP states and SMALL_TASKS other tasks
    const uint32_t n_other =
        (sm.carry[T_ITEM] + 31u) / 32u + (sm.carry[T_LB] + 31u) / 32u + (sm.carry[T_ROWS] + 31u) / 32u;
    const bool small = small_warps != 0u && sm.live_cnt != 0u &&
                       (n_sssp + sm.carry[T_PULL]) * sd.avg_deg <= SMALL_ARCS * small_warps &&
                       n_dp <= SMALL_DP * small_warps && n_other <= SMALL_TASKS * small_warps;
    sd.small = small ? 1u : 0u;
    const uint32_t lw = small ? small_warps : sd.light_warps;
    // distance items per warp task: 4 while that leaves at most two tasks per
    // light warp, more (up to sssp_wmax) in rounds with many items
    uint32_t w = 4;
    while (w < min(sd.sssp_wmax, SSSP_WMAX) && n_sssp > 2ull * w * lw) w <<= 1;
    sd.sssp_w = w;
    // DP states per warp task: 1 while that leaves at most two tasks per
    // light warp (every state gets a warp), more (up to dp_wmax) in rounds
    // with many states
    uint32_t wd = 1;
    while (wd < sd.dp_wmax && n_dp > 2ull * wd * lw) wd <<= 1;
    sd.dp_w = wd;
    const uint32_t per_task[NT] = {32, 1, 1, w, wd, wd, 32 / PULL_LANES, 32, 32};
    uint32_t off = 0;
#pragma unroll
    for (int t = 0; t < NT; t++) {
      uint32_t tot = sm.carry[t];
      sd.items[t] = tot;
      if (t == T_LB) {
        sd.light_tasks = off;
        off = 0;
      }
      sd.task_off[t] = off;
      off += (tot + per_task[t] - 1) / per_task[t];
    }
    sd.task_off[NT] = off;
    sd.heavy_tasks = off;
    sd.n_live = sm.live_cnt;
    sd.nslots = sm.used_hi;  // slots the round kernels search (all later ones are free)
    sd.n_big = 0;
    sd.next_light = 0;
    sd.next_heavy = 0;
    // hub chunking pays off only when the round is too small to fill the GPU
    const uint32_t n_items = (uint32_t)(n_sssp + n_dp);
    sd.hub_on = (sd.big != nullptr && n_items < sd.hub_max_items) ? 1u : 0u;
    // distance items: every hub in small rounds; in larger ones (a single
    // query's dense rounds) only the biggest hubs, whose one warp would
    // otherwise finish long after the rest: at least hub_big_deg arcs and
    // more than 1/hub_share_div of a warp's share of the round's arcs
    uint32_t big_deg = sd.hub_big_deg;
    if (sd.hub_share_div != 0u) {
      const unsigned long long share =
          (unsigned long long)n_items * sd.avg_deg / max(1u, sd.light_warps) / sd.hub_share_div;
      big_deg = (uint32_t)max((unsigned long long)big_deg, min(share, (unsigned long long)INF32 - 1ull));
    }
    sd.hub_deg = sd.hub_on ? sd.hub_min_deg
                           : ((sd.big != nullptr && n_items < sd.hub_max_items2) ? big_deg : INF32);
    // DP tasks that hold several states hand their hub grows out in every
    // round: a task with a few hub states would otherwise grow them one
    // after another on one warp
    sd.grow_chunks = (sd.big != nullptr && (sd.hub_on || wd > 1u)) ? 1u : 0u;
  }
  __syncthreads();
  for (uint32_t i = tid; i < RD_WORDS; i += B)
    reinterpret_cast<uint32_t*>(rd)[i] = reinterpret_cast<const uint32_t*>(&sd)[i];
}

// ---------------------------------------------------------------------------
// Round work, one warp task at a time.  The separate round kernels (k_light,
// k_heavy) and the persistent one (k_rounds) run the same tasks.
// ---------------------------------------------------------------------------

// Light task `task` (types T_ITEM .. T_PULL: splits and seeds, tour tables,
// extraction, distance items, DP states, gathered rows).  s_pre / s_dp / s_hop: the per-slot
// prefixes of the distance, DP and hop items, staged in shared memory.
__device__ __forceinline__ void light_task(const QDev* qd, const RoundDesc& sd, RoundDesc* rd, const uint32_t* pre,
                                           const uint32_t* s_pre, const uint32_t* s_dp, const uint32_t* s_hop,
                                           int nslots, const GraphDev& g, uint32_t task, uint32_t lane,
                                           WarpStat& ws, WarpBuf& wb, WarpScratch& sc) {
  int t = 0;
  while (t < T_PULL && task >= sd.task_off[t + 1]) t++;
  const uint32_t local = task - sd.task_off[t];
  const uint32_t* P = pre + t * (MAX_SLOTS + 1);
  const uint32_t total = sd.items[t];
  if (t == T_SSSP) {
    sssp_task(qd, s_pre, nslots, total, local, sd.sssp_w, g, lane, ws, sd, rd, sc.hdr, wb);
  } else if (t == T_DP || t == T_HOP) {
    dp_task(qd, t == T_DP ? s_dp : s_hop, nslots, total, local, sd.dp_w, t == T_HOP, g, lane, sd, rd, ws, wb, &sc.mg);
  } else if (t == T_PULL) {
    pull_task(qd, P, nslots, total, local, g, lane, ws, sd, rd);
  } else if (t == T_TOUR) {
    // (the tables' scratch: the warp's append buffer, emptied first)
    static_assert(sizeof(wb.it) >= TOUR_WORDS * 4 && sizeof(WarpScratch) >= 256, "tour scratch");
    const uint32_t slot = find_slot(P, nslots, local);
    wb_flush(wb, lane);
    tour_warp(qd[slot], local - __ldcg(P + slot), lane, reinterpret_cast<uint32_t*>(&sc), wb.it);
  } else if (t == T_EXTRACT) {
    extract_warp(qd[find_slot(P, nslots, local)], g, lane);
  } else {
    const uint32_t it = local * 32u + lane;
    bool toN = false, toF = false;
    uint32_t slot = 0, item = 0;
    if (it < total) {
      slot = find_slot(P, nslots, it);
      const QDev& q = qd[slot];
      const uint32_t idx = it - __ldcg(P + slot);
      if (q.act == A_SPLIT) {
        item = q.rescan ? idx : q.qbuf[q.far_idx][idx];
        split_item(q, item, toN, toF);
      } else if (q.act == A_SSEED) {
        const uint32_t m = __ldg(q.members + idx);
        item = m >> 3;
        sseed_item(q, m, toN);
      } else {
        dseed_item(q, __ldg(q.members + idx));
      }
    }
    push_multi(toN, item, 0u, qd[slot], slot, lane);
    push_multi(toF, item, 1u, qd[slot], slot, lane);
  }
}

// Heavy task `ht` that does not depend on the round's light tasks: bound-table
// rows (one vertex per lane) and passes over hop-bounded queries' distance rows.
__device__ __forceinline__ void heavy_static_task(const QDev* qd, const uint32_t* pre, const uint32_t* s_lb,
                                                  int nslots, uint32_t ht, uint32_t rows0, uint32_t n_lb,
                                                  uint32_t n_rows, uint32_t lane, LbScratch& lb) {
  if (ht < rows0) {
    lbt_rows32(qd, s_lb, nslots, n_lb, ht, lane, lb);
    return;
  }
  // a pass over a hop-bounded query's distance rows, one row per lane
  const uint32_t it = (ht - rows0) * 32u + lane;
  if (it < n_rows) {
    const uint32_t* P = pre + T_ROWS * (MAX_SLOTS + 1);
    const uint32_t slot = find_slot(P, nslots, it);
    const QDev& q = qd[slot];
    const uint32_t h = q.rows_h;
    if (h + 2u <= q.push_rounds) {  // copy: its buffer is written again two rounds later
      const uint32_t v = it - __ldcg(P + slot);
      const uint4* src = reinterpret_cast<const uint4*>(q.dist + (size_t)v * ROW);
      uint4* dst = reinterpret_cast<uint4*>(q.rows[h] + (size_t)v * ROW);
      const uint4 a = __ldcg(src), b = __ldcg(src + 1);
      dst[0] = a;
      dst[1] = b;
      return;
    }
    // the rows are the exact distances over paths of at most h hops
    uint32_t l, r[KMAX];
    const uint32_t v = list_item(q, it - __ldcg(P + slot), l);
    load_row(q.rows[h], v, r);
    bool all = true;
    unsigned long long sum = 0;
#pragma unroll
    for (int t = 0; t < KMAX; t++)
      if (t < q.k) {
        all = all && r[t] != INF32;
        sum += r[t];
      }
    if (all && h == q.center_h && __ldca(&q.ctl->center) == 0u) atomicExch(&q.ctl->center, 1u);
    // v joined to every group by its cheapest path of at most star_h
    // hops: a breadth-first tree from v inside their union has depth <=
    // star_h, so diameter <= 2 * star_h <= D, at cost <= sum
    if (all && h == q.star_h && sum < ld_best(q.ctl)) atomicMin(&q.ctl->best, (uint32_t)sum);
  }
}

// Whether the round's light tasks may hand arc chunks over.
__device__ __forceinline__ bool has_chunks(const RoundDesc& sd) {
  return sd.big != nullptr && (sd.hub_deg != INF32 || sd.grow_chunks != 0u || sd.items[T_PULL] != 0u);
}

// Arc chunk `i` that a light task handed over this round (hub vertex of a
// distance item, or a high-degree DP state's grow).
__device__ __forceinline__ void chunk_task(const QDev* qd, const RoundDesc& sd, const GraphDev& g, uint32_t i,
                                           uint32_t lane, RelaxHdr* hub, WarpStat& ws, WarpBuf& wb) {
  const uint4 it = __ldcg(sd.big + i);
  if (it.x & CH_PULL)
    pull_chunk(qd, it, g, lane, ws);
  else if (it.x & CH_GROW)
    grow_chunk(qd, it, g, lane, ws, wb);
  else
    hub_chunk(qd, it, g, lane, hub, ws, wb);
}

// Light round kernel: the round's light tasks.  NW warps per block (4 or
// 8); the occupancy bound keeps 24 warps per SM at 80 registers.
#ifndef GSTB_LIGHT_MIN_BLOCKS
#define GSTB_LIGHT_MIN_BLOCKS 3  // blocks of 8 warps
#endif
template <int NW>
__global__ void __launch_bounds__(NW * 32, GSTB_LIGHT_MIN_BLOCKS * 8 / NW)
    k_light(const QDev* __restrict__ qd, RoundDesc* __restrict__ rd, const uint32_t* __restrict__ pre, int nslots,
            GraphDev g) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  __shared__ RoundDesc sd;
  stage_rd(sd, rd);
  __syncthreads();
  const uint32_t ntasks = sd.light_tasks;
  if (ntasks == 0u) return;
  nslots = min(nslots, (int)sd.nslots);
  // prefixes over slots of the item types with many items, staged once per block
  __shared__ uint32_t s_pre[MAX_SLOTS + 1], s_dp[MAX_SLOTS + 1], s_hop[MAX_SLOTS + 1];
  __shared__ WarpScratch s_sc[NW];
  __shared__ WarpStat s_ws[NW];
  __shared__ WarpBuf s_wb[NW];
  WarpStat& ws = s_ws[threadIdx.x >> 5];
  WarpBuf& wb = s_wb[threadIdx.x >> 5];
  if (lane == 0) {
    ws_init(ws);
    wb_init(wb);
  }
  for (int i = threadIdx.x; i <= nslots; i += blockDim.x) {
    s_pre[i] = __ldcg(pre + T_SSSP * (MAX_SLOTS + 1) + i);
    s_dp[i] = __ldcg(pre + T_DP * (MAX_SLOTS + 1) + i);
    s_hop[i] = __ldcg(pre + T_HOP * (MAX_SLOTS + 1) + i);
  }
  __syncthreads();
#if GSTB_STEAL
  for (uint32_t task = warp; task < ntasks; task = next_task(&rd->next_light, nwarps, lane))
#else
  for (uint32_t task = warp; task < ntasks; task += nwarps)
#endif
    light_task(qd, sd, rd, pre, s_pre, s_dp, s_hop, nslots, g, task, lane, ws, wb, s_sc[threadIdx.x >> 5]);
  wb_flush(wb, lane);
  if (lane == 0) ws_flush(ws);
}

// Heavy round kernel: the arc chunks k_light handed over this round, then
// bound-table rows and passes over distance rows.
template <int NW>
__global__ void __launch_bounds__(NW * 32, 24 / NW)
    k_heavy(const QDev* __restrict__ qd, RoundDesc* __restrict__ rd, const uint32_t* __restrict__ pre, int nslots,
            GraphDev g) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  __shared__ RoundDesc sd;
  stage_rd(sd, rd);
  __syncthreads();
  const uint32_t nbig = sd.big ? min(sd.n_big, sd.big_cap) : 0u;
  const uint32_t ntasks = sd.heavy_tasks + nbig;
  if (ntasks == 0u) return;
  nslots = min(nslots, (int)sd.nslots);
  __shared__ uint32_t s_lb[MAX_SLOTS + 1];
  __shared__ RelaxHdr s_hub[NW];
  __shared__ LbScratch s_lbs[NW];
  __shared__ WarpStat s_ws[NW];
  __shared__ WarpBuf s_wb[NW];
  WarpStat& ws = s_ws[threadIdx.x >> 5];
  WarpBuf& wb = s_wb[threadIdx.x >> 5];
  LbScratch& lb = s_lbs[threadIdx.x >> 5];
  if (lane == 0) {
    ws_init(ws);
    wb_init(wb);
    lb.n = 0;
  }
  for (int i = threadIdx.x; i <= nslots; i += blockDim.x) s_lb[i] = __ldcg(pre + T_LB * (MAX_SLOTS + 1) + i);
  __syncthreads();
  const uint32_t n_lb = sd.items[T_LB], n_rows = sd.items[T_ROWS];
  const uint32_t rows0 = sd.task_off[T_ROWS];  // heavy tasks before the passes over rows
#if GSTB_STEAL
  for (uint32_t task = warp; task < ntasks; task = next_task(&rd->next_heavy, nwarps, lane)) {
#else
  for (uint32_t task = warp; task < ntasks; task += nwarps) {
#endif
    if (task < nbig)
      chunk_task(qd, sd, g, task, lane, &s_hub[threadIdx.x >> 5], ws, wb);
    else
      heavy_static_task(qd, pre, s_lb, nslots, task - nbig, rows0, n_lb, n_rows, lane, lb);
  }
  lb_flush(qd, lane, lb);
  wb_flush(wb, lane);
  if (lane == 0) ws_flush(ws);
}

// ---------------------------------------------------------------------------
// Persistent round loop: R rounds in one cooperative launch (every block
// resident at once).  Block 0 runs the first control step; the last block to
// finish a round's work runs the next one.  A round is
//   wait for its control step (epoch) -> light tasks and the static heavy
//   tasks (bound rows, passes over rows), taken by warp striding -> every block done
//   with those (phase1: the arc chunks the light tasks handed over are all
//   written; skipped in rounds that hand out none) -> the chunks -> arrive;
//   the last block to arrive runs the next control step and publishes it.
// Every wait is bounded by pc->timeout_ns (and an iteration limit): when one
// expires the launch sets pc->err and every block returns, the host fails
// the admitted queries with GST_DEVICE_TIMEOUT and the context stays usable.
// ---------------------------------------------------------------------------
// The waits poll with relaxed loads (read at L2, leaving the SM's L1 alone)
// and order what follows with one fence once the flag is seen: an acquire at
// every poll would invalidate the L1 of an SM whose other blocks are still
// working from it.
__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One thread: wait until *flag >= target, then fence (the acquire).  False
// when the launch has failed (another wait expired) or this one expires.
__device__ bool wait_geq(const uint32_t* flag, uint32_t target, PersistCtl* pc, uint32_t where) {
  const unsigned long long t0 = global_ns(), lim = pc->timeout_ns;
  uint32_t ns = 32;
  for (uint32_t it = 0; it < (1u << 25); it++) {
    if (ld_relaxed_gpu(flag) >= target) {
      __threadfence();
      return true;
    }
    if (ld_relaxed_gpu(&pc->err)) return false;
    if (global_ns() - t0 > lim) break;
    if (it >= 64u) {  // a short wait polls back to back, a long one backs off to 1 us
      __nanosleep(ns);
      if (ns < 1024u) ns <<= 1;
    }
  }
  atomicCAS(&pc->err_where, 0u, where);
  atomicExch(&pc->err, 1u);
  return false;
}

// Publish control step `e` (after its writes).  One thread.
__device__ __forceinline__ void publish(PersistCtl* pc, uint32_t e) {
  __threadfence();
  if (!pc->hold) st_release_gpu(&pc->epoch, e);
}

template <int NW>
struct RoundSmem {
  uint32_t pre_sssp[MAX_SLOTS + 1], pre_dp[MAX_SLOTS + 1], pre_hop[MAX_SLOTS + 1], pre_lb[MAX_SLOTS + 1];
  WarpScratch w[NW];
  WarpStat ws[NW];
  WarpBuf wb[NW];
  CtlSmem ctl;
  RoundDesc rd;
  uint32_t ok, last;
};

// ---------------------------------------------------------------------------
// Control and small rounds: one cluster (SMALL_NW warps per CTA), the first
// kernel of every round.  CTA 0 runs the control step.  While the round it
// lays out is small the cluster runs it itself and goes on to the next, with
// hardware cluster barriers between the steps; the first round that is not
// (or whose arc chunks are too many) is left to the k_light and k_heavy
// launches that follow.  Most rounds of a query hold a few hundred items and
// are a chain of dependent accesses: as three launches over the whole GPU
// such a round costs its launches, a scan of every slot and three grid
// start-ups.  The cluster also leaves when a query has finished, so that the
// host sees it, and after `rounds` rounds, so that waiting ones are admitted.
// Every CTA of a cluster is resident, so the barriers cannot wait for ever.
// What the rounds write is read with ordinary weak loads after a barrier
// (release / acquire), as in the persistent launch.  Measured against a
// one-block control kernel before k_light and k_heavy in every round: one
// k = 3 query on 10k vertices 1063 -> 746 us, four hop-bounded ones 5360 ->
// 3837 us, six on 170k vertices 7559 -> 6757 us, a 90-query batch there
// unchanged (21.8 -> 21.7 ms: its rounds are large).
// ---------------------------------------------------------------------------
constexpr int SMALL_NW = 16;
constexpr int SMALL_SLOTS = 8;  // query descriptors kept in shared memory

struct SmallSmem {
  RoundSmem<SMALL_NW> r;
  QDev qd[SMALL_SLOTS];
};

__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(SMALL_NW * 32, 1)
    k_small(QDev* qd, QCtl* ctl, int nslots_ctl, RoundDesc* rd, uint32_t* pre, GraphDev g, uint32_t rounds) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  SmallSmem& ss = *reinterpret_cast<SmallSmem*>(s_raw);
  RoundSmem<SMALL_NW>& sm = ss.r;
  const RoundDesc& sd = sm.rd;
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  // consecutive tasks go to different SMs
  const uint32_t nwarps = gridDim.x * SMALL_NW, warp = wib * gridDim.x + blockIdx.x;
  WarpStat& ws = sm.ws[wib];
  WarpBuf& wb = sm.wb[wib];
  uint32_t live0 = 0;
  if (lane == 0) {
    ws_init(ws);
    wb_init(wb);
  }
  // nothing admitted since the last control step found no live query: the round
  // described is empty, and stays so (every CTA reads the same word, which no one
  // writes before they have all passed the first barrier)
  if (__ldcg(&rd->n_live) == 0u) return;
  cluster_barrier();
  for (uint32_t r = 0;; r++) {
    if (blockIdx.x == 0) control_step(qd, ctl, nslots_ctl, rd, pre, sm.ctl, sm.rd, r < rounds ? nwarps : 0u);
    cluster_barrier();
    // the round's description, the first slots' prefixes and descriptors in
    // one trip to L2 (with few slots in use they are all there is)
    stage_rd(sm.rd, rd);
    auto stage_pre = [&](int i) {
      sm.pre_sssp[i] = __ldcg(pre + T_SSSP * (MAX_SLOTS + 1) + i);
      sm.pre_dp[i] = __ldcg(pre + T_DP * (MAX_SLOTS + 1) + i);
      sm.pre_hop[i] = __ldcg(pre + T_HOP * (MAX_SLOTS + 1) + i);
      sm.pre_lb[i] = __ldcg(pre + T_LB * (MAX_SLOTS + 1) + i);
    };
    if (threadIdx.x <= SMALL_SLOTS) stage_pre(threadIdx.x);
    const uint32_t qw = min(nslots_ctl, SMALL_SLOTS) * (uint32_t)(sizeof(QDev) / 8);
    for (uint32_t i = threadIdx.x; i < qw; i += blockDim.x)
      reinterpret_cast<unsigned long long*>(ss.qd)[i] = __ldcg(reinterpret_cast<const unsigned long long*>(qd) + i);
    __syncthreads();
    if (r == 0) live0 = sd.n_live;
    // every CTA reads the same words, so all of them leave here together
    if (!sd.small || sd.n_live < live0) return;
    const int nslots = min(nslots_ctl, (int)sd.nslots);
    const QDev* q = qd;
    if (nslots <= SMALL_SLOTS) {
      q = ss.qd;
    } else {
      for (int i = SMALL_SLOTS + 1 + threadIdx.x; i <= nslots; i += blockDim.x) stage_pre(i);
      __syncthreads();
    }
    const uint32_t ntl = sd.light_tasks, nth = sd.heavy_tasks;
    const uint32_t n_lb = sd.items[T_LB], n_rows = sd.items[T_ROWS], rows0 = sd.task_off[T_ROWS];
    bool lb_used = false;  // the warp's scratch holds a list of bound rows (its light tasks come first)
    for (uint32_t task = warp; task < ntl + nth; task += nwarps) {
      if (task >= ntl && !lb_used) {
        lb_used = true;
        __syncwarp();
        if (lane == 0) sm.w[wib].lb.n = 0;
        __syncwarp();
      }
      if (task < ntl)
        light_task(q, sd, rd, pre, sm.pre_sssp, sm.pre_dp, sm.pre_hop, nslots, g, task, lane, ws, wb, sm.w[wib]);
      else
        heavy_static_task(q, pre, sm.pre_lb, nslots, task - ntl, rows0, n_lb, n_rows, lane, sm.w[wib].lb);
    }
    if (lb_used) lb_flush(q, lane, sm.w[wib].lb);
    bool handover = false;
    if (has_chunks(sd)) {
      cluster_barrier();  // the chunk list is complete
      const uint32_t nbig = sd.big ? min(__ldcg(&rd->n_big), sd.big_cap) : 0u;
      handover = nbig > SMALL_CHUNKS * nwarps;  // too many for the cluster: k_heavy takes them
      if (!handover)
        for (uint32_t i = warp; i < nbig; i += nwarps) chunk_task(q, sd, g, i, lane, &sm.w[wib].hdr[0], ws, wb);
    }
    wb_flush(wb, lane);
    if (lane == 0) {
      wb.q = nullptr;  // the descriptors are staged again
      ws_flush(ws);
    }
    cluster_barrier();  // the round's work is done and visible to the next control step
    if (handover) {
      if (blockIdx.x == 0 && threadIdx.x == 0) rd->light_tasks = rd->heavy_tasks = 0u;
      return;
    }
  }
}

template <int NW>
__global__ void __launch_bounds__(NW * 32, 24 / NW)
    k_rounds(QDev* qd, QCtl* ctl, int nslots_ctl, RoundDesc* rd, uint32_t* pre, GraphDev g, uint32_t R,
             PersistCtl* pc) {
  __shared__ RoundSmem<NW> sm;
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + wib;
  const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
  WarpStat& ws = sm.ws[wib];
  WarpBuf& wb = sm.wb[wib];
  uint32_t p1 = 0;  // rounds with a chunk phase so far (the same in every block)
  if (blockIdx.x == 0) {
    control_step(qd, ctl, nslots_ctl, rd, pre, sm.ctl, sm.rd);
    __syncthreads();
    if (threadIdx.x == 0) publish(pc, 1u);
  }
  for (uint32_t r = 0; r < R; r++) {
    if (threadIdx.x == 0) sm.ok = wait_geq(&pc->epoch, r + 1u, pc, 1u) ? 1u : 0u;
    __syncthreads();
    if (!sm.ok) return;
    stage_rd(sm.rd, rd);
    __syncthreads();
    const RoundDesc& sd = sm.rd;
    // a round with no live query does nothing, nor do the rest: every block
    // reads the same count, so every block leaves here together
    if (sd.n_live == 0u) return;
    const int nslots = min(nslots_ctl, (int)sd.nslots);
    for (int i = threadIdx.x; i <= nslots; i += blockDim.x) {
      sm.pre_sssp[i] = __ldcg(pre + T_SSSP * (MAX_SLOTS + 1) + i);
      sm.pre_dp[i] = __ldcg(pre + T_DP * (MAX_SLOTS + 1) + i);
      sm.pre_hop[i] = __ldcg(pre + T_HOP * (MAX_SLOTS + 1) + i);
      sm.pre_lb[i] = __ldcg(pre + T_LB * (MAX_SLOTS + 1) + i);
    }
    if (lane == 0) {
      ws_init(ws);
      wb_init(wb);
    }
    __syncthreads();
    const uint32_t ntl = sd.light_tasks, nth = sd.heavy_tasks;
    const uint32_t n_lb = sd.items[T_LB], n_rows = sd.items[T_ROWS], rows0 = sd.task_off[T_ROWS];
    // light tasks, then the static heavy ones, as one list dealt out over
    // the warps (two lists dealt out one after the other would leave the
    // warps with the heaviest light tasks also the first heavy ones)
    bool lb_used = false;  // the warp's scratch holds a list of bound rows (its light tasks come first)
    for (uint32_t task = warp; task < ntl + nth; task += nwarps) {
      if (task >= ntl && !lb_used) {
        lb_used = true;
        __syncwarp();
        if (lane == 0) sm.w[wib].lb.n = 0;
        __syncwarp();
      }
      if (task < ntl)
        light_task(qd, sd, rd, pre, sm.pre_sssp, sm.pre_dp, sm.pre_hop, nslots, g, task, lane, ws, wb, sm.w[wib]);
      else
        heavy_static_task(qd, pre, sm.pre_lb, nslots, task - ntl, rows0, n_lb, n_rows, lane, sm.w[wib].lb);
    }
    if (lb_used) lb_flush(qd, lane, sm.w[wib].lb);
    // phase 1 done in this block: its chunk entries are written.  Rounds
    // that hand out no chunks (every block reads the same flags) skip the
    // grid-wide wait for the others
    if (has_chunks(sd)) {
      p1++;
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&pc->phase1, 1u);
        sm.ok = wait_geq(&pc->phase1, p1 * gridDim.x, pc, 2u) ? 1u : 0u;
      }
    }
    __syncthreads();
    if (sm.ok) {
      const uint32_t nbig = sd.big ? min(__ldcg(&rd->n_big), sd.big_cap) : 0u;
      for (uint32_t i = warp; i < nbig; i += nwarps) chunk_task(qd, sd, g, i, lane, &sm.w[wib].hdr[0], ws, wb);
    }
    wb_flush(wb, lane);
    if (lane == 0) ws_flush(ws);
    __syncthreads();
    if (!sm.ok) return;
    if (threadIdx.x == 0) {
      __threadfence();
      const uint32_t old = atomicAdd(&pc->arrive, 1u);
      sm.last = old == (r + 1u) * gridDim.x - 1u ? 1u : 0u;
      if (sm.last) {
        __threadfence();  // every block's round work is visible from here on
        pc->rounds = r + 1u;
      }
    }
    __syncthreads();
    if (sm.last && r + 1u < R) {
      control_step(qd, ctl, nslots_ctl, rd, pre, sm.ctl, sm.rd);
      __syncthreads();
      if (threadIdx.x == 0) publish(pc, r + 2u);
    }
    __syncthreads();  // sm.ok and sm.last are rewritten next round
  }
}

// Host side: the round kernels of one block size, 128 or 256 threads (null
// for any other; 512-thread blocks would need more than the 48 KB of static
// shared memory a block can hold: each warp stages its appends in 2 KB).
const void* light_kernel(int threads) {
  return threads == 128 ? (const void*)k_light<4> : threads == 256 ? (const void*)k_light<8> : nullptr;
}
const void* heavy_kernel(int threads) {
  return threads == 128 ? (const void*)k_heavy<4> : threads == 256 ? (const void*)k_heavy<8> : nullptr;
}
const void* small_kernel(int* threads, size_t* smem) {
  *threads = SMALL_NW * 32;
  *smem = sizeof(SmallSmem);
  return (const void*)k_small;
}
const void* rounds_kernel(int threads) {
  return threads == 128 ? (const void*)k_rounds<4> : threads == 256 ? (const void*)k_rounds<8> : nullptr;
}

}  // namespace gstb
