// Motif enumeration for sm_100a: one task = (v0, range of second vertices) or a donated DFS
// prefix, run by a warp whose lanes form 32/W virtual warps ("groups") of W lanes.
//
// Semantics follow the reference's motif driver (src/main/motifs_DM_WCLB.cu:9-36): every
// connected induced k-subgraph is enumerated once, from its lowest-id vertex v0, along the one
// vertex order the reference's canonical filter accepts (extend(0,k), DuMatoGPU.cu:1702-1721;
// canonicalFilter2, 989-1012: an extension x whose first adjacent prefix vertex is v_src must
// exceed every prefix vertex after v_src), and classified through the quick code
// (forward_induce 846-869, aggregate_pattern 930-967) looked up in the dictionary.
//
// That filter makes the extension sets incremental. If E_t is the valid extension set of
// prefix (v_0..v_t) and w = v_{t+1} is taken from it, then
//     E_{t+1} = { e in E_t : e > w }  U  excl(w),
//     excl(w) = { x in N(w) : x > v0, x not in N(v_0) U .. U N(v_t) }
// (the inherited members keep their source, and the only new constraint is "> w"; the new
// members have w as their source). Every member carries its adjacency mask to the prefix
// (bit i = edge to v_i), so quick codes come from masks, not from the reference's per-leaf
// adjacency scans. The excluded set U_t = N(v_0..v_t) cap (v0, inf) is kept as disjoint
// sorted runs (run 0 = N(v0) above v0, run i = excl(v_i)). E_t is kept sorted by vertex id, so
// the inherited members are the suffix of E_t after w.
//
// The last two vertices are counted in bulk (leaf_sweep): once E_{k-3} of a (k-2)-prefix is
// materialised, no member is expanded. With R_a the number of members of mask a, the pairs
// (w, x) of members contribute R_a R_b (C(R_a,2) for a = b) subgraphs of masks a, b, of which
// those joined by an edge are moved to the joined class; and a member w adds its neighbours above
// v0 that lie outside U_{k-3}. So the sweep only walks the members' rows above v0 once, testing
// each neighbour against the two bitmaps, and adds to the class counters once per prefix and
// mask pair. The rows of W members are laid end to end, one entry per lane, so rows shorter than
// the group waste no lanes. Expanding every member w on its own (its row scanned, its leaf
// masks looked up and flushed) took 12.6 ms for k = 5 on a Chung-Lu graph of 3,000 vertices and
// 18,000 edges, 10.4 ms for k = 6 on a random graph of 2,000 / 10,000, 387 ms for a batch of 24
// graphs; the sweep takes 7.0, 5.2 and 86 ms.
//
// Virtual warps (the reference's DM_WCV variant, src/DM_WCV/DuMatoGPU.cu:12-37): with W < 32
// the groups of a warp take second vertices of the same task from its shared item range and
// run their subtrees independently, each with its own DFS state and arena; every collective
// uses the group's lane mask. Small extension sets (small graphs, low degree) keep more
// lanes busy this way.
//
// Load balancing (lb.cuh): idle warps get donated work, either a range of second vertices
// or, when one second vertex roots most of the work (a hub), a DFS prefix - the path to some
// level's extension set and a range of its members, which the receiver rebuilds by replaying
// the path (each level's set is a deterministic function of the path).
#pragma once

#include <climits>

#include "engine.hpp"
#include "gpm.cuh"
#include "lb.cuh"

namespace dmb {

constexpr int MOTIF_KMAX = 7;

__host__ __device__ constexpr int quick_off(int p) { return (p - 2) * (p + 1) / 2; }

// DFS state of one group.
struct alignas(16) MotifGroup {
  int n[MOTIF_KMAX];           // extension-set sizes per level
  int pos[MOTIF_KMAX];         // next member to expand per level
  int lim[MOTIF_KMAX];         // members [pos, lim) of a level are still this group's to expand
  int runn[MOTIF_KMAX];        // run sizes per level
  unsigned quick[MOTIF_KMAX];  // quick code of the prefix ending at level t
  int spill_lo, spill_hi;      // second vertices split off when the queue was full
};

// Sweep state of one group: class counters of its task, and by mask over E_{k-3} the members swept
// (rest: those after the swept range), their neighbours outside U, and the joined pairs.
template <int K>
struct alignas(16) MotifSweep {
  static constexpr int MASKS = 1 << (K > 3 ? K - 2 : 2);
  unsigned swept[MASKS], rest[MASKS], fresh[MASKS];
  unsigned joined[K > 3 ? MASKS * MASKS : 1];
  unsigned mh[8];              // k = 3: leaf-mask histogram
};

// 64-bit class counters: in shared memory (w, as pairs of 32-bit words, low word first: a 64-bit
// add to shared memory is a compare-and-swap loop, and many lanes add to the same few classes;
// two 32-bit adds with the carry taken from the first one's old value are native), else in
// global memory (g).
struct ClassHist {
  unsigned* w;
  unsigned long long* g;
  __device__ __forceinline__ void add(int c, unsigned long long v) const {
    if (w) {
      const unsigned lo = (unsigned)v;
      unsigned hi = (unsigned)(v >> 32);
      const unsigned old = atomicAdd(w + 2 * c, lo);
      hi += old + lo < old ? 1u : 0u;
      if (hi) atomicAdd(w + 2 * c + 1, hi);
    } else {
      atomicAdd(g + c, v);
    }
  }
};

// Task state shared by the groups of one warp.
struct alignas(16) MotifShared {
  unsigned long long range;    // second vertices not taken yet (pack_range)
  int donations_left;          // donation budget of the running task
  int busy;                    // serialises level-0 splits
};

template <int K, int W>
__host__ __device__ constexpr size_t motif_warp_smem() {
  return sizeof(MotifShared) + (sizeof(MotifGroup) + sizeof(MotifSweep<K>)) * (32 / W);
}

// Everything a motif task needs besides its own (v0, range) or prefix.
struct MotifCtx {
  GraphView g;                 // undirected CSR, rows sorted
  LBArgs lb;
  const int32_t* q2c;          // quick code -> class
  int sym;                     // the class does not depend on the order of the last two vertices
  int maxdeg;                  // bound on every degree in g (arena sizing)
  int arena_stride;            // int2 slots per group
  unsigned long long* per_root;  // optional: subgraphs found under each v0 (subtree logger)
  int bit_base;                // membership bitmaps index vertex x at bit x - bit_base
  int bit_words;               // 32-bit words per bitmap (0 = no bitmaps: binary searches only)
};

// Membership bitmaps of one group (bit_words pairs of words, all zero between tasks; word 2i of
// U and word 2i + 1 of E, so that one 8-byte load answers both questions): U holds
// U_t = N(v_0..v_t) above v0 for the levels materialised on the current path, E holds E_{k-3}.
// They turn the sweep and the exclusion test into one probe per neighbour instead of binary
// searches over the runs (k >= 4).
__device__ __forceinline__ bool bit_test(const uint32_t* b, int x) { return (b[2 * (x >> 5)] >> (x & 31)) & 1u; }

template <int W>
__device__ __forceinline__ void bits_flip_ids(uint32_t* b, int base, const int32_t* ids, int n, bool set, int gl) {
  for (int i = gl; i < n; i += W) {
    const int x = __ldg(ids + i) - base;
    if (set) atomicOr(b + 2 * (x >> 5), 1u << (x & 31));
    else atomicAnd(b + 2 * (x >> 5), ~(1u << (x & 31)));
  }
}

template <int W>
__device__ __forceinline__ void bits_flip_list(uint32_t* b, int base, const int2* list, int n, bool set, int gl) {
  for (int i = gl; i < n; i += W) {
    const int x = list[i].x - base;
    if (set) atomicOr(b + 2 * (x >> 5), 1u << (x & 31));
    else atomicAnd(b + 2 * (x >> 5), ~(1u << (x & 31)));
  }
}

// int2 slots of one group's arena: extension levels 1..k-3 (level t holds at most
// (t+1) * maxdeg members) then runs 1..k-3 (at most maxdeg each).
__host__ __device__ inline size_t motif_group_stride(int k, int maxdeg) {
  size_t s = 0;
  for (int t = 1; t <= k - 3; ++t) s += (size_t)(t + 1) * maxdeg + 32;
  for (int t = 1; t <= k - 3; ++t) s += (size_t)maxdeg + 32;
  return s < 1 ? 1 : s;
}

// First index in [lo, hi) of an id-sorted (vertex, mask) list whose vertex is >= x.
__device__ __forceinline__ int lower_bound2(const int2* a, int lo, int hi, int32_t x) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid].x < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ int ilog2p1(int x) { return 32 - __clz(x | 1); }

// Membership of x in the disjoint sorted runs 0..t (run 0 is the CSR suffix of v0; run i >= 1
// starts at runs1 + (i - 1) * rstride).
__device__ __forceinline__ bool in_runs(int32_t x, const int32_t* run0, int n0, const int2* runs1, size_t rstride,
                                        const int* runn, int t) {
  if (contains(run0, n0, x)) return true;
  for (int i = 1; i <= t; ++i) {
    const int2* r = runs1 + (size_t)(i - 1) * rstride;
    const int nr = runn[i];
    const int j = lower_bound2(r, 0, nr, x);
    if (j < nr && r[j].x == x) return true;
  }
  return false;
}

// Adds the masks of list[lo, hi) to the group's 32-entry histogram h (aggregated per mask).
template <int W>
__device__ __forceinline__ void mask_hist(const int2* list, int lo, int hi, unsigned* h, int gl, unsigned gmask) {
  for (int i0 = lo; i0 < hi; i0 += W) {
    const int i = i0 + gl;
    const bool v = i < hi;
    dm_gpm::aggregate_pattern<W>(h, v ? list[i].y : 0, v);
  }
  __syncwarp(gmask);
}

// Sweeps members [lo, *lim) of the materialised set E = E_{K-3} (n members, sorted by id) of the
// prefix whose quick code is quick_t: every subgraph with at least one of its last two vertices
// in the range, the other one after it in E or new, is added to hist. `between` runs after every
// batch of W members with the next position (group-uniform; it may lower *lim). Returns this
// lane's share of the subgraphs counted.
//
// Bound by instruction issue: a step of about 45 instructions takes W row entries (an owner
// search by shuffles, one load of the entry, one 8-byte load of both bitmaps, one ballot).
template <int K, int W, class Between>
__device__ __forceinline__ unsigned long long leaf_sweep(const MotifCtx& c, const ClassHist& hist, MotifSweep<K>* sw,
                                                         const int2* E, int n, int lo, const int* lim, int v0,
                                                         unsigned quick_t, const uint32_t* Ub, const int32_t* E0,
                                                         int n0, const int2* runs1, size_t rstride, const int* runn,
                                                         int gl, int gsrc, unsigned gmask, Between&& between) {
  constexpr int P = K - 2;  // position of the first of the two vertices; the second is at K - 1
  constexpr int MASKS = MotifSweep<K>::MASKS;
  unsigned long long counted = 0;
  auto code = [&](unsigned a, unsigned b) -> unsigned {
    return quick_t + (P >= 2 ? a << quick_off(P) : 0u) + (b << quick_off(K - 1));
  };
  if (!c.sym) {
    // pairs in id order, one member at a time: the masks of the members after it
    mask_hist<W>(E, lo, n, sw->rest, gl, gmask);
  }
  int i0 = lo;
  while (i0 < *reinterpret_cast<const volatile int*>(lim)) {
    const int end = min(*reinterpret_cast<const volatile int*>(lim), i0 + W);
    const bool valid = i0 + gl < end;
    int2 wm = make_int2(0, 0);
    int base = 0, len = 0;
    if (valid) {
      wm = E[i0 + gl];
      const int r = __ldg(c.g.row + wm.x);
      const int d = __ldg(c.g.deg + wm.x);
      const int s = lower_bound(c.g.adj + r, 0, d, v0 + 1);
      base = r + s;
      len = d - s;
    }
    int off = len;
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
      const int y = __shfl_up_sync(gmask, off, o, W);
      if (gl >= o) off += y;
    }
    const int total = __shfl_sync(gmask, off, W - 1, W);
    off -= len;
    unsigned inside = 0;  // this lane's member: its neighbours in U
    for (int f0 = 0; f0 < total; f0 += W) {
      const int f = f0 + gl;
      // owner: the last member whose entries start at or before f
      int j = 0;
#pragma unroll
      for (int h = W / 2; h >= 1; h >>= 1) {
        const int o = __shfl_sync(gmask, off, j + h, W);
        j = o <= f ? j + h : j;
      }
      const int ob = __shfl_sync(gmask, base, j, W) + (f - __shfl_sync(gmask, off, j, W));
      const int ow = __shfl_sync(gmask, wm.x, j, W);
      const int om = __shfl_sync(gmask, wm.y, j, W);
      bool in_u = false, in_e = false;
      int x = 0;
      if (f < total) {
        x = __ldg(c.g.adj + ob);
        if (Ub) {
          const int xb = x - c.bit_base;
          const uint2 ue = *reinterpret_cast<const uint2*>(Ub + 2 * (xb >> 5));
          in_u = (ue.x >> (xb & 31)) & 1u;
          in_e = x > ow && ((ue.y >> (xb & 31)) & 1u);
        } else {
          in_u = in_runs(x, E0, n0, runs1, rstride, runn, K - 3);
          in_e = in_u && x > ow;
        }
      }
      const unsigned bal = __ballot_sync(gmask, in_u) >> gsrc;
      const int a0 = min(max(off - f0, 0), W), a1 = min(max(off + len - f0, 0), W);
      const unsigned upto1 = a1 >= 32 ? 0xffffffffu : (1u << a1) - 1u;
      const unsigned upto0 = a0 >= 32 ? 0xffffffffu : (1u << a0) - 1u;
      inside += __popc(bal & upto1 & ~upto0);
      if (in_e) {
        const int q = lower_bound2(E, i0 + j + 1, n, x);
        if (q < n) {
          const int2 y = E[q];
          if (y.x == x) atomicAdd(&sw->joined[om * MASKS + y.y], 1u);
        }
      }
    }
    if (valid) {
      if (len > (int)inside) atomicAdd(&sw->fresh[wm.y], (unsigned)len - inside);
      atomicAdd(&sw->swept[wm.y], 1u);
    }
    __syncwarp(gmask);
    if (!c.sym) {
      for (int i = i0; i < end; ++i) {
        const int m = E[i].y;
        if (gl == 0) sw->rest[m] -= 1u;
        __syncwarp(gmask);
        for (int b = gl; b < MASKS; b += W) {
          const unsigned t = sw->rest[b];
          if (t) {
            hist.add(__ldg(c.q2c + code(m, b)), (unsigned long long)t);
            counted += t;
          }
        }
        __syncwarp(gmask);
      }
    }
    i0 = end;
    between(end);
  }
  if (c.sym && i0 < n) mask_hist<W>(E, i0, n, sw->rest, gl, gmask);
  __syncwarp(gmask);
  // every (a, b) to a lane
  for (int ab = gl; ab < MASKS * MASKS; ab += W) {
    const int a = ab / MASKS, b = ab % MASKS;
    const unsigned ra = sw->swept[a];
    if (ra == 0) continue;
    unsigned long long pairs = 0;
    if (c.sym) {
      const unsigned long long rb = sw->swept[b];
      if (b == a) pairs = (rb & 1) ? rb * ((rb - 1) >> 1) : (rb >> 1) * (rb - 1);
      else if (b > a) pairs = (unsigned long long)ra * rb;
      pairs += (unsigned long long)ra * sw->rest[b];
    }
    const unsigned join = sw->joined[ab];
    if (join) {
      sw->joined[ab] = 0u;
      hist.add(__ldg(c.q2c + code(a, b | (1 << P))), (unsigned long long)join);
    }
    // (a pair joined in the order (a, b) was taken in that order or, with equal classes, in the
    // other: the difference may be negative here, the class total is not)
    if (pairs != join) hist.add(__ldg(c.q2c + code(a, b)), pairs - join);
    counted += pairs;
  }
  for (int a = gl; a < MASKS; a += W) {
    const unsigned fr = sw->fresh[a];
    if (fr) {
      sw->fresh[a] = 0u;
      hist.add(__ldg(c.q2c + code(a, 1 << P)), (unsigned long long)fr);
      counted += fr;
    }
  }
  __syncwarp(gmask);
  for (int m = gl; m < MASKS; m += W) sw->swept[m] = sw->rest[m] = 0u;
  __syncwarp(gmask);
  return counted;
}

// k = 3: flushes the group's leaf-mask histogram (masks below 4) into the class counters.
template <int W>
__device__ __forceinline__ void flush_masks(unsigned* mh, const int32_t* q2c, const ClassHist& hist,
                                            unsigned long long& task_cnt, int gl, unsigned gmask) {
  for (int m = gl; m < 4; m += W) {
    const unsigned c = mh[m];
    if (c) {
      mh[m] = 0;
      hist.add(__ldg(q2c + m), (unsigned long long)c);
      task_cnt += c;
    }
  }
  __syncwarp(gmask);
}

// The group leader's view of the demand for work: the hungry and queued counters as loaded at the
// previous check. The loads complete while the group works on, so a check never waits for them.
struct MotifDemand {
  int hungry = 0;
  int queued = 0;
};

__device__ __forceinline__ void motif_sample(const LBArgs& lb, MotifDemand& dm) {
  if (lb.hungry_trigger <= 0) return;
  dm.hungry = vload(&lb.ctr->hungry);
  dm.queued = vload(&lb.ctr->queued);
}

// Whether this task should hand work out now, by the previous sample; takes the next one.
__device__ __forceinline__ bool motif_wanted(const LBArgs& lb, const MotifShared* ws, MotifDemand& dm, long long t_start) {
  if (lb.hungry_trigger <= 0) return false;
  const bool wanted = dm.hungry - dm.queued >= lb.hungry_trigger;
  motif_sample(lb, dm);
  if (!wanted || *reinterpret_cast<const volatile int*>(&ws->donations_left) <= 0) return false;
  return global_ns() - t_start >= lb.donate_after_ns;
}

// Group leader, between two expansions of a task whose lowest own level is `floor` (1 for an
// item task; L for a donated DFS prefix of level L) and whose deepest materialised level is
// t, when work is wanted: hands the upper half of the shallowest level that still has
// unexpanded members to the queue. Level 0 is the task's second-vertex range (cost-aware
// split, shared by the groups); a level s >= 1 goes out as (root, s, path to E_s, position
// range), the path being the second vertex's index `it` and the index picked at each level
// 1..s-1.
__device__ __forceinline__ void motif_donate(const LBArgs& lb, MotifShared* ws, MotifGroup* sg, int v0, int floor, int t,
                                             int it, int n0) {
  if (floor == 1) {
    const unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&ws->range);
    const int next = (int)(unsigned)cur, end = (int)(unsigned)(cur >> 32);
    if (end - next >= 2) {
      // inside a running item even two untaken second vertices are worth handing out
      if (sg->spill_lo >= sg->spill_hi) {
        int ob = 0, oe = 0;
        if (range_split_donate(lb, &ws->range, v0, &ws->donations_left, &ws->busy, ob, oe, n0, 2, 0, nullptr)) {
          // the queue was full: this group runs the split-off second vertices itself
          sg->spill_lo = ob;
          sg->spill_hi = oe;
        }
      }
      return;
    }
  }
  for (int s = floor; s <= t; ++s) {
    const int ps = sg->pos[s], lim = sg->lim[s];
    if (lim - ps >= 2) {
      // E_s is sorted by id: member i inherits the n - i - 1 members above it
      const int mid = split_mid(ps, lim, sg->n[s]);
      int path[QPATH];
      path[0] = it;
      for (int j = 1; j < s && j < QPATH; ++j) path[j] = sg->pos[j] - 1;
      if (lb_donate_deep(lb, v0, s, path, mid, lim)) {
        sg->lim[s] = mid;
        atomicSub(&ws->donations_left, 1);
      }
      return;
    }
  }
}

// k = 3: the subgraphs (v0, w, x) with w the member of E_0 = N(v0) above v0 at index it.
template <int W>
__device__ __forceinline__ void leaf_pairs(const MotifCtx& c, unsigned* mh, const int32_t* E0, int n0, int it, int v0,
                                           const ClassHist& hist, unsigned long long& task_cnt, int gl,
                                           unsigned gmask) {
  const int w = __ldg(E0 + it);
  const int32_t* Nw = c.g.adj + __ldg(c.g.row + w);
  const int dw = __ldg(c.g.deg + w);
  const int start = it + 1, n_inh = n0 - start;
  const int sw0 = lower_bound(Nw, 0, dw, v0 + 1);
  const int above = dw - sw0;
  const int gt = lower_bound(Nw, 0, dw, w + 1);
  const int dgt = dw - gt;
  // members of E_0 after w that are adjacent to w: probe each of them in N(w), or each
  // neighbour above w in E_0, whichever side is cheaper
  unsigned adj = 0;
  if ((long long)dgt * ilog2p1(n_inh) < (long long)n_inh * ilog2p1(dw)) {
    for (int i = gt + gl; i < dw; i += W) adj += contains(E0 + start, n_inh, Nw[i]) ? 1u : 0u;
  } else {
    for (int i = start + gl; i < n0; i += W) adj += contains(Nw, dw, __ldg(E0 + i)) ? 1u : 0u;
  }
  // new vertices: N(w) above v0 minus N(v0)
  unsigned inter = 0;
  if (n0 <= above) {
    for (int i = gl; i < n0; i += W) inter += contains(Nw, dw, __ldg(E0 + i)) ? 1u : 0u;
  } else {
    for (int i = sw0 + gl; i < dw; i += W) inter += contains(E0, n0, Nw[i]) ? 1u : 0u;
  }
  for (int o = W / 2; o > 0; o >>= 1) {
    adj += __shfl_xor_sync(gmask, adj, o);
    inter += __shfl_xor_sync(gmask, inter, o);
  }
  if (gl == 0) {
    mh[1] = (unsigned)n_inh - adj;
    mh[2] = (unsigned)above - inter;
    mh[3] = adj;
  }
  __syncwarp(gmask);
  flush_masks<W>(mh, c.q2c, hist, task_cnt, gl, gmask);
}

// Runs one task on the calling warp (all 32 lanes). level 0: second vertices [bb, ee) of v0
// (task_range encoding); level L >= 1: replay path[0..L-1], then expand positions [bb, ee) of
// E_L (group 0 only). Adds the task's subgraphs to hist; nodes counts expansions (every
// lane of a group counts the same nodes; the caller keeps group leaders' counts only).
template <int K, int W>
__device__ __forceinline__ void motif_run_task(const MotifCtx& c, const ClassHist& hist, MotifShared* ws,
                                               int2* warp_arena, uint32_t* warp_bits, int v0, int bb, int ee,
                                               int level, const int* path, unsigned long long& nodes) {
  static_assert(W == 8 || W == 16 || W == 32, "virtual warp width must be 8, 16 or 32");
  const int lane = lane_id();
  const int gl = lane & (W - 1);
  const int gi = lane / W;
  const unsigned gmask = (W == 32) ? FULL_MASK : (((1u << W) - 1u) << (gi * W));
  const int gsrc = gi * W;  // the group leader's lane
  // the warp's words: MotifShared | a MotifGroup per group | a MotifSweep per group
  MotifGroup* sg = reinterpret_cast<MotifGroup*>(ws + 1) + gi;
  MotifSweep<K>* sw = reinterpret_cast<MotifSweep<K>*>(reinterpret_cast<MotifGroup*>(ws + 1) + 32 / W) + gi;
  // level t (1..K-3): extension list E_t at ext_at(t); run t at run_at(t) (no pointer
  // tables, so nothing indexed dynamically lives in local memory)
  int2* const arena = warp_arena + (size_t)gi * c.arena_stride;
  const size_t md = (size_t)c.maxdeg;
  auto ext_at = [&](int t) -> int2* { return arena + md * (size_t)(t * (t + 1) / 2 - 1) + 32 * (size_t)(t - 1); };
  int2* const runs1 = ext_at(K - 2);
  const size_t rstride = md + 32;
  auto run_at = [&](int t) -> int2* { return runs1 + (size_t)(t - 1) * rstride; };
  // (k = 3 has a single level: setting and clearing E_0's bits per task costs more than the
  // binary searches it saves)
  const bool use_bits = K >= 4 && warp_bits != nullptr && c.bit_words > 0;
  uint32_t* const Ub = use_bits ? warp_bits + (size_t)gi * 2 * c.bit_words : nullptr;
  uint32_t* const Eb = use_bits ? Ub + 1 : nullptr;
  int bdepth = 0;  // levels 1..bdepth have their run (and, at level k-3, E) bits set
  unsigned long long task_cnt = 0;
  const long long t_start = global_ns();
  // E_0 = run 0 = N(v0) above v0: a suffix of the sorted CSR row
  const int32_t* row0 = c.g.adj + __ldg(c.g.row + v0);
  const int deg0 = __ldg(c.g.deg + v0);
  const int s0 = lower_bound(row0, 0, deg0, v0 + 1);
  const int32_t* E0 = row0 + s0;
  const int n0 = deg0 - s0;
  const int floor = level > 0 ? level : 1;
  int lo = 0, hi = 0;
  if (level == 0) task_range(bb, ee, n0, lo, hi);
  __syncwarp();
  if (lane == 0) {
    ws->range = pack_range(lo, hi);
    ws->donations_left = c.lb.max_donations;
    ws->busy = 0;
  }
  if (gl == 0) {
    sg->quick[0] = 0;
    sg->spill_lo = sg->spill_hi = 0;
  }
  for (int m = gl; m < (int)(sizeof(MotifSweep<K>) / sizeof(unsigned)); m += W) reinterpret_cast<unsigned*>(sw)[m] = 0u;
  if (use_bits) bits_flip_ids<W>(Ub, c.bit_base, E0, n0, true, gl);
  MotifDemand dm;  // group leader
  if (gl == 0) motif_sample(c.lb, dm);
  unsigned long long checked = nodes;
  __syncwarp();
  // drops the bits of levels from..bdepth (the group's lanes, then a group barrier)
  auto drop_levels = [&](int from) {
    for (int L = bdepth; L >= from; --L) {
      bits_flip_list<W>(Ub, c.bit_base, run_at(L), sg->runn[L], false, gl);
      if (L == K - 3) bits_flip_list<W>(Eb, c.bit_base, ext_at(L), sg->n[L], false, gl);
    }
    if (bdepth >= from) bdepth = from - 1;
    __syncwarp(gmask);
  };
  bool replay_item = level > 0 && gi == 0;
  while (true) {
    int it = 0;
    if (level > 0) {
      if (!replay_item) break;
      replay_item = false;
      it = path[0];
      if (it < 0 || it >= n0) {
        if (gl == 0) set_err(c.lb.ctr, ERR_BAD_TASK);
        break;
      }
    } else {
      if (gl == 0) {
        it = range_take(&ws->range);
        if (it < 0) {
          if (sg->spill_lo < sg->spill_hi) it = sg->spill_lo++;
        } else if (sg->spill_lo >= sg->spill_hi) {
          int ob = 0, oe = 0;
          if (motif_wanted(c.lb, ws, dm, t_start) &&
              range_split_donate(c.lb, &ws->range, v0, &ws->donations_left, &ws->busy, ob, oe, n0, 0, 0, nullptr)) {
            sg->spill_lo = ob;
            sg->spill_hi = oe;
          }
        }
      }
      it = __shfl_sync(gmask, it, gsrc);
      if (it < 0) break;
    }
    if constexpr (K == 3) {
      ++nodes;
      if (gl == 0 && (nodes & 255) == 0) atomicAdd(&c.lb.ctr->progress, 256ull);
      leaf_pairs<W>(c, sw->mh, E0, n0, it, v0, hist, task_cnt, gl, gmask);
    } else {
      // prefix (v0, w1); the members of E_0 after w1 are the inherited part
      int t = 0;
      int w = __ldg(E0 + it);
      int wmask = 1;
      bool bad = false;
      // hands work away when it is wanted (checked every 64 expansions)
      auto give = [&]() {
        if (nodes - checked >= 64) {
          checked = nodes;
          if (gl == 0 && motif_wanted(c.lb, ws, dm, t_start)) motif_donate(c.lb, ws, sg, v0, floor, t, it, n0);
          __syncwarp(gmask);
        }
      };
      // depth-first over levels; level t's current vertex is w with mask wmask
      while (true) {
        // here the prefix is v_0..v_t plus w = v_{t+1}
        const int p = t + 1;  // position of w
        if (p > level) {
          // nodes at or above a donated prefix's level belong to the donor
          ++nodes;
          if (gl == 0 && (nodes & 255) == 0) atomicAdd(&c.lb.ctr->progress, 256ull);
        }
        unsigned quick_p = (t == 0) ? 0u : sg->quick[t];
        if (p >= 2) quick_p += ((unsigned)wmask & ((1u << p) - 1u)) << quick_off(p);
        const int32_t* Nw = c.g.adj + __ldg(c.g.row + w);
        const int dw = __ldg(c.g.deg + w);
        // inherited members: e in E_t with e > w. E_t is sorted by vertex id and w is its
        // member at position pos[t] - 1 (E_0: index it), so they are the suffix from there.
        const int2* Et = t == 0 ? nullptr : ext_at(t);
        const int nE = (t == 0) ? n0 : sg->n[t];
        const int startE = (t == 0) ? it + 1 : sg->pos[t];
        // materialise E_{p} = inherited + excl(w), merged by vertex id; excl(w) is also run
        // p. Both parts are sorted and disjoint, so each member's place is its index in its
        // own part plus the number of smaller members of the other part.
        int2* Ep = ext_at(p);
        int2* Rp = run_at(p);
        if (use_bits) drop_levels(p);  // the previous member's sets at levels >= p
        const int sw0 = dw <= 2 * W ? 0 : lower_bound(Nw, 0, dw, v0 + 1);
        int rn = 0;
        for (int i0 = sw0; i0 < dw; i0 += W) {
          const int i = i0 + gl;
          int32_t x = 0;
          bool nw = false;
          if (i < dw && Nw[i] > v0) {
            x = Nw[i];
            nw = use_bits ? !bit_test(Ub, x - c.bit_base) : !in_runs(x, E0, n0, runs1, rstride, sg->runn, t);
          }
          const unsigned bal = __ballot_sync(gmask, nw) >> gsrc;
          if (nw) Rp[rn + __popc(bal & ((1u << gl) - 1u))] = make_int2(x, 0);
          rn += __popc(bal);
        }
        __syncwarp(gmask);
        for (int i = startE + gl; i < nE; i += W) {
          int ev, em;
          if (t == 0) {
            ev = __ldg(E0 + i);
            em = 1;
          } else {
            const int2 x = Et[i];
            ev = x.x;
            em = x.y;
          }
          if (contains(Nw, dw, ev)) em |= 1 << p;
          Ep[(i - startE) + lower_bound2(Rp, 0, rn, ev)] = make_int2(ev, em);
        }
        for (int j = gl; j < rn; j += W) {
          const int32_t x = Rp[j].x;
          const int cnt_lt = (t == 0) ? lower_bound(E0, 0, n0, x) : lower_bound2(Et, 0, nE, x);
          Ep[j + max(0, cnt_lt - startE)] = make_int2(x, 1 << p);
        }
        const int m = (nE - startE) + rn;
        __syncwarp(gmask);
        if (use_bits) {
          bits_flip_list<W>(Ub, c.bit_base, Rp, rn, true, gl);
          if (p == K - 3) bits_flip_list<W>(Eb, c.bit_base, Ep, m, true, gl);
          bdepth = p;
          __syncwarp(gmask);
        }
        if (p < level) {
          // replaying a donated prefix: the path fixes the member expanded at level p
          const int idx = (p < QPATH) ? path[p] : -1;
          if (idx < 0 || idx >= m) {
            if (gl == 0) set_err(c.lb.ctr, ERR_BAD_TASK);
            bad = true;
            break;
          }
          const int2 x = Ep[idx];
          if (gl == 0) {
            sg->n[p] = m;
            sg->pos[p] = idx + 1;
            sg->lim[p] = idx + 1;
            sg->runn[p] = rn;
            sg->quick[p] = quick_p;
          }
          __syncwarp(gmask);
          t = p;
          w = x.x;
          wmask = x.y;
          continue;
        }
        const int first_pos = p == level ? min(bb, m) : 0;
        if (gl == 0) {
          sg->n[p] = m;
          sg->pos[p] = first_pos;
          sg->lim[p] = p == level ? min(ee, m) : m;
          sg->runn[p] = rn;
          sg->quick[p] = quick_p;
        }
        __syncwarp(gmask);
        t = p;  // descend
        if (p == K - 3) {
          // the last two vertices in bulk
          int last = first_pos;
          task_cnt += leaf_sweep<K, W>(c, hist, sw, Ep, m, first_pos, &sg->lim[p], v0, quick_p, Ub, E0, n0, runs1, rstride,
                                       sg->runn, gl, gsrc, gmask, [&](int next) {
                                         const unsigned long long before = nodes;
                                         nodes += (unsigned long long)(next - last);
                                         last = next;
                                         if (gl == 0) {
                                           sg->pos[p] = next;
                                           if ((nodes ^ before) >> 8) atomicAdd(&c.lb.ctr->progress, 256ull);
                                         }
                                         __syncwarp(gmask);
                                         give();
                                       });
        }
        give();
        // next vertex: advance the deepest level that still has members
        bool found = false;
        while (t >= floor) {
          const int ps = sg->pos[t];
          if (ps < sg->lim[t]) {
            const int2 x = ext_at(t)[ps];
            __syncwarp(gmask);
            if (gl == 0) sg->pos[t] = ps + 1;
            __syncwarp(gmask);
            w = x.x;
            wmask = x.y;
            found = true;
            break;
          }
          --t;
        }
        if (!found) break;
      }
      if (use_bits) drop_levels(1);
      if (bad) break;
    }
  }
  if (use_bits) bits_flip_ids<W>(Ub, c.bit_base, E0, n0, false, gl);
  __syncwarp();
  if (c.per_root) {
    const unsigned long long tsum = warp_sum_u64(task_cnt);
    if (lane == 0 && tsum) atomicAdd(c.per_root + v0, tsum);
  }
  if (lane == 0) lb_task_time(c.lb, t_start, v0);
}

}  // namespace dmb
