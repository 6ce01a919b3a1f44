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
// adjacency scans. The excluded set U_t = N(v_0..v_t) cap (v0, inf) is kept as disjoint runs
// (run 0 = N(v0) above v0, run i = excl(v_i)); E_t lists the inherited members in E_{t-1}'s order,
// then excl(v_t) ascending, so it is a deterministic function of the path.
//
// The last two vertices are counted in bulk (leaf_sweep): once E_{k-3} of a (k-2)-prefix is
// materialised, no member is expanded. With R_a the number of members of mask a, the pairs
// (w, x) of members contribute R_a R_b (C(R_a,2) for a = b) subgraphs of masks a, b, of which
// those joined by an edge are moved to the joined class; and a member w adds its neighbours above
// v0 that lie outside U_{k-3}. So the sweep only walks the members' rows above v0 once, looking
// each neighbour up in the bitmaps, and adds to the class counters once per prefix and mask pair. The rows of W members are laid end to end, one entry per lane, so rows shorter than
// the group waste no lanes. Expanding every member w on its own (its row scanned, its leaf
// masks looked up and flushed) took 12.6 ms for k = 5 on a Chung-Lu graph of 3,000 vertices and
// 18,000 edges, 10.4 ms for k = 6 on a random graph of 2,000 / 10,000, 387 ms for a batch of 24
// graphs; the sweep took 6.5, 5.3 and 86 ms while the sets were sorted lists in global memory that
// masks and adjacency were searched in, and takes 3.5, 4.2 and 51 ms with one bitmap per mask bit
// and the sets of level k-3 in shared memory.
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
  // k = 7: 16-bit counters, two to a word (32-bit ones took 4 KB of each group: one block per SM with
  // groups of 8 lanes). They hold the pairs of a set of up to 255 members; larger sets do without.
  static constexpr bool NARROW = K == 7;
  static constexpr int NARROW_SET = 255;
  unsigned joined[K > 3 ? MASKS * MASKS / (NARROW ? 2 : 1) : 1];
  __device__ __forceinline__ void join(int at) {
    if constexpr (NARROW) atomicAdd(joined + (at >> 1), 1u << (16 * (at & 1)));
    else atomicAdd(joined + at, 1u);
  }
  __device__ __forceinline__ unsigned take(int at) {  // reads and zeroes a counter
    unsigned v;
    if constexpr (NARROW) {
      unsigned short* h = reinterpret_cast<unsigned short*>(joined) + at;
      if ((v = *h)) *h = 0;
    } else {
      if ((v = joined[at])) joined[at] = 0u;
    }
    return v;
  }
};

// 64-bit class counters: in shared memory (w, as pairs of 32-bit words, low word first: a 64-bit
// add to shared memory is a compare-and-swap loop, and many lanes add to the same few classes;
// two 32-bit adds with the carry taken from the first one's old value are native), else in
// global memory (g).
struct ClassHist {
  unsigned* w;
  unsigned long long* g;
  __device__ __forceinline__ void add(int c, unsigned long long v) const {
    if (!w) {
      atomicAdd(g + c, v);
      return;
    }
    const unsigned lo = (unsigned)v;
    unsigned hi = (unsigned)(v >> 32);
    const unsigned old = atomicAdd(w + 2 * c, lo);
    hi += old + lo < old ? 1u : 0u;
    if (hi) atomicAdd(w + 2 * c + 1, hi);
  }
};

// Task state shared by the groups of one warp.
struct alignas(16) MotifShared {
  unsigned long long range;    // second vertices not taken yet (pack_range)
  int donations_left;          // donation budget of the running task
  int busy;                    // serialises level-0 splits
};

// The lists of level k-3 of one group, in shared memory while they fit (arena otherwise): they are
// written and read back at once, and a global store read back by the same warp costs a trip to L2.
template <int W>
struct alignas(16) MotifLists {
  static constexpr int CAP = 4 * W;
  int2 ext[CAP];
  int run[CAP];
};

// A warp's shared memory: MotifShared | a MotifGroup, a MotifSweep and a MotifLists per group.
template <int K, int W>
__host__ __device__ constexpr size_t motif_warp_smem() {
  // (k = 3 sweeps nothing and keeps no lists)
  return sizeof(MotifShared) +
         (sizeof(MotifGroup) + (K > 3 ? sizeof(MotifSweep<K>) + sizeof(MotifLists<W>) : 0)) * (32 / W);
}

// Zeroes a warp's sweep counters (all 32 lanes; every sweep leaves them zero). Once per launch where the
// memory holds nothing else, else before each task.
template <int K, int W>
__device__ __forceinline__ void motif_zero_sweeps(MotifShared* ws) {
  if constexpr (K == 3) return;
  unsigned* const s = reinterpret_cast<unsigned*>(reinterpret_cast<MotifGroup*>(ws + 1) + 32 / W);
  for (int i = lane_id(); i < (int)(sizeof(MotifSweep<K>) / sizeof(unsigned)) * (32 / W); i += 32) s[i] = 0u;
  __syncwarp();
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
  int bit_words;               // 32-bit words per bitmap
};

// Vertex bitmaps of one group (k >= 4), all zero between tasks: the words of 32 vertices lie
// together, so one or three vector loads answer everything about a vertex. Word 0: U_t above v0
// for the levels materialised on the current path; word 1 + i: the members of E_{k-3} adjacent to
// v_i (a member's mask, bit by bit). Word k - 2 (i = k - 3) also marks N(w) while a set is built.
__host__ __device__ constexpr int motif_bit_stride(int k) { return k <= 5 ? 4 : 6; }

template <int K>
struct MotifBits {
  static constexpr int STRIDE = motif_bit_stride(K);
  static constexpr int MARK = K - 2;
  uint32_t* b;
  int base;
  __device__ __forceinline__ uint32_t* at(int x) const { return b + STRIDE * ((x - base) >> 5); }
  __device__ __forceinline__ uint32_t bit(int x) const { return 1u << ((x - base) & 31); }
  // (x in U, mask of x in E_{k-3})
  __device__ __forceinline__ void look(int x, bool& in_u, unsigned& mask) const {
    const int s = (x - base) & 31;
    if constexpr (STRIDE == 4) {
      const uint4 v = *reinterpret_cast<const uint4*>(at(x));
      in_u = (v.x >> s) & 1u;
      mask = ((v.y >> s) & 1u) | (((v.z >> s) & 1u) << 1);
      if constexpr (K >= 5) mask |= ((v.w >> s) & 1u) << 2;
    } else {
      const uint2* q = reinterpret_cast<const uint2*>(at(x));
      const uint2 v0 = q[0], v1 = q[1], v2 = q[2];
      in_u = (v0.x >> s) & 1u;
      mask = ((v0.y >> s) & 1u) | (((v1.x >> s) & 1u) << 1) | (((v1.y >> s) & 1u) << 2) | (((v2.x >> s) & 1u) << 3);
      if constexpr (K >= 7) mask |= ((v2.y >> s) & 1u) << 4;
    }
  }
  __device__ __forceinline__ void set(int x, int word) const { atomicOr(at(x) + word, bit(x)); }
  __device__ __forceinline__ void clear(int x, int word) const { atomicAnd(at(x) + word, ~bit(x)); }
};

// int2 slots of one group's arena: extension levels 1..k-3 (level t holds at most
// (t+1) * maxdeg members) then runs 1..k-3 (at most maxdeg each).
__host__ __device__ inline size_t motif_group_stride(int k, int maxdeg) {
  size_t s = 0;
  for (int t = 1; t <= k - 3; ++t) s += (size_t)(t + 1) * maxdeg + 32;
  for (int t = 1; t <= k - 3; ++t) s += (size_t)maxdeg + 32;
  return s < 1 ? 1 : s;
}

__device__ __forceinline__ int ilog2p1(int x) { return 32 - __clz(x | 1); }

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

// Tables whose classes depend on the order of the last two vertices: the pairs of member i of
// E (n members) with every member of a larger id, in that order (a member list per mask first).
template <int K, int W>
__device__ __noinline__ unsigned long long leaf_ordered(const MotifCtx& c, const ClassHist& hist, MotifSweep<K>* sw,
                                                        const int2* E, int n, int i, unsigned quick_t, int gl,
                                                        unsigned gmask) {
  unsigned long long counted = 0;
  const int2 w = E[i];
  for (int j0 = 0; j0 < n; j0 += W) {
    const int j = j0 + gl;
    const int2 x = j < n ? E[j] : make_int2(-1, 0);
    dm_gpm::aggregate_pattern<W>(sw->rest, x.y, x.x > w.x);
  }
  __syncwarp(gmask);
  for (int b = gl; b < MotifSweep<K>::MASKS; b += W) {
    const unsigned t = sw->rest[b];
    sw->rest[b] = 0u;
    if (t) {
      const unsigned q = quick_t + ((unsigned)w.y << quick_off(K - 2)) + ((unsigned)b << quick_off(K - 1));
      hist.add(__ldg(c.q2c + q), (unsigned long long)t);
      counted += t;
    }
  }
  __syncwarp(gmask);
  return counted;
}

// Sweeps members [lo, *lim) of the materialised set E = E_{K-3} (n members) of the prefix whose
// quick code is quick_t: every pair of a swept member with a member after it in E, and of a swept
// member with a new vertex, is added to hist (an edge between two members is credited to the
// one of smaller id, wherever that one is swept). `between` runs after every batch of W
// members with the next position (group-uniform; it may lower *lim). Returns this lane's share of
// the subgraphs counted.
//
// Bound by instruction issue: a step of about 40 instructions takes W row entries (an owner
// search by shuffles, one load of the entry, one lookup in the bitmaps, one ballot).
template <int K, int W, bool ROWS, class Between>
__device__ __forceinline__ unsigned long long leaf_sweep(const MotifCtx& c, const ClassHist& hist, MotifSweep<K>* sw,
                                                         const int2* E, int n, int lo, const int* lim, int v0,
                                                         unsigned quick_t, const MotifBits<K>& bits, int gl, int gsrc,
                                                         unsigned gmask, Between&& between) {
  constexpr int P = K - 2;  // position of the first of the two vertices; the second is at K - 1
  constexpr int MASKS = MotifSweep<K>::MASKS;
  unsigned long long counted = 0;
  auto code = [&](unsigned a, unsigned b) -> unsigned {
    return quick_t + (a << quick_off(P)) + (b << quick_off(K - 1));
  };
  // moves a pair of members with masks a, b to the joined class
  auto join = [&](unsigned a, unsigned b) {
    if (MotifSweep<K>::NARROW && n > MotifSweep<K>::NARROW_SET) {
      hist.add(__ldg(c.q2c + code(a, b | (1 << P))), 1ull);
      hist.add(__ldg(c.q2c + code(a, b)), ~0ull);
    } else {
      sw->join((int)(a * MASKS + b));
    }
  };
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
    // narrow groups, rows of similar length: a row per lane, which needs no owners (k = 6, random graph of
    // 9,000 / 16,000, 8 lanes: 4.22 -> 3.51 ms; k = 7, 16,000 / 18,000, 16 lanes: 4.46 -> 3.93; k = 5
    // with 16 lanes is no faster by rows)
    constexpr bool BY_ROW = ROWS && (W == 8 || (W == 16 && K >= 6));
    int longest = INT_MAX;
    if constexpr (BY_ROW) {
      longest = len;
#pragma unroll
      for (int o = W / 2; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(gmask, longest, o));
    }
    const bool by_row = BY_ROW && longest * W <= 2 * total;
    if (by_row) {
      for (int i = 0; i < longest; ++i) {
        if (i < len) {
          const int x = __ldg(c.g.adj + base + i);
          bool in_u;
          unsigned xm;
          bits.look(x, in_u, xm);
          if (xm && x > wm.x) join((unsigned)wm.y, xm);
          inside += in_u ? 1u : 0u;
        }
      }
    }
    for (int f0 = by_row ? total : 0; f0 < total; f0 += W) {
      const int f = f0 + gl;
      // owner: the last member whose entries start at or before f
      int j = 0;
#pragma unroll
      for (int h = W / 2; h >= 1; h >>= 1) {
        const int o = __shfl_sync(gmask, off, j + h, W);
        j = o <= f ? j + h : j;
      }
      const int ob = __shfl_sync(gmask, base - off, j, W) + f;
      const int ow = __shfl_sync(gmask, wm.x, j, W);
      const int om = __shfl_sync(gmask, wm.y, j, W);
      bool in_u = false;
      unsigned xm = 0;
      if (f < total) {
        const int x = __ldg(c.g.adj + ob);
        bits.look(x, in_u, xm);
        if (xm && x > ow) join((unsigned)om, xm);
      }
      const unsigned bal = __ballot_sync(gmask, in_u) >> gsrc;
      const int a0 = min(max(off - f0, 0), W), a1 = min(max(off + len - f0, 0), W);
      const unsigned upto1 = a1 >= 32 ? 0xffffffffu : (1u << a1) - 1u;
      const unsigned upto0 = a0 >= 32 ? 0xffffffffu : (1u << a0) - 1u;
      inside += __popc(bal & upto1 & ~upto0);
    }
    if (valid) {
      if (len > (int)inside) atomicAdd(&sw->fresh[wm.y], (unsigned)len - inside);
      atomicAdd(&sw->swept[wm.y], 1u);
    }
    __syncwarp(gmask);
    if (!c.sym)
      for (int i = i0; i < end; ++i) counted += leaf_ordered<K, W>(c, hist, sw, E, n, i, quick_t, gl, gmask);
    i0 = end;
    between(end);
  }
  if (c.sym && i0 < n) mask_hist<W>(E, i0, n, sw->rest, gl, gmask);
  __syncwarp(gmask);
  auto settle = [&](int a, int b, unsigned ra) {
    unsigned long long pairs = 0;
    if (c.sym) {
      const unsigned long long rb = sw->swept[b];
      if (b == a) pairs = (rb & 1) ? rb * ((rb - 1) >> 1) : (rb >> 1) * (rb - 1);
      else if (b > a) pairs = (unsigned long long)ra * rb;
      pairs += (unsigned long long)ra * sw->rest[b];
    }
    const unsigned joins = sw->take(a * MASKS + b);
    // (a pair joined in the order (a, b) may have been counted in the other order, or in another
    // range of E: the difference may be negative here, the class total is not)
    if (pairs != joins) hist.add(__ldg(c.q2c + code(a, b)), pairs - joins);
    if (joins) hist.add(__ldg(c.q2c + code(a, b | (1 << P))), (unsigned long long)joins);
    counted += pairs;
  };
  if constexpr (MASKS * MASKS <= 4 * W) {
    // every (a, b) to a lane
    for (int ab = gl; ab < MASKS * MASKS; ab += W) {
      const unsigned ra = sw->swept[ab / MASKS];
      if (ra) settle(ab / MASKS, ab % MASKS, ra);
    }
  } else {
    // only the masks that were swept (few of them: most sets are small), their b over the lanes: up to
    // 1,024 pairs were looked at per prefix for k = 7
    unsigned present = 0;
#pragma unroll
    for (int m = 0; m < MASKS; m += W)
      present |= (__ballot_sync(gmask, m + gl < MASKS && sw->swept[m + gl] != 0u) >> gsrc) << m;
    for (; present; present &= present - 1) {
      const int a = __ffs(present) - 1;
      const unsigned ra = sw->swept[a];
      for (int b = gl; b < MASKS; b += W) settle(a, b, ra);
    }
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
      const int mid = split_mid(ps, lim, 0);
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

// k = 3: the subgraphs (v0, w, x) with w the member of E_0 = N(v0) above v0 at index it, by leaf mask
// m in s[m - 1]. A lane's own sums may be negative; the group's are the counts. One pass over E_0 or
// over N(w) above v0, whichever searches less, gives both the neighbours of w in E_0 and those of them
// after w. The lanes meet after every search: drifting apart they loaded one row in more and smaller pieces
// (k = 3 of a Chung-Lu graph of 18,700 vertices with groups of 8 / 16 / 32 lanes: 1.83 / 1.38 / 0.82 ms per
// call with a pass for each and no meeting, 0.62 / 0.50 / 0.54 now).
template <int W>
__device__ __forceinline__ void leaf_pairs(const MotifCtx& c, const int32_t* E0, int n0, int it, int v0, int gl,
                                           unsigned gmask, long long (&s)[3]) {
  const int w = __ldg(E0 + it);
  const int32_t* Nw = c.g.adj + __ldg(c.g.row + w);
  const int dw = __ldg(c.g.deg + w);
  const int sw0 = lower_bound(Nw, 0, dw, v0 + 1);
  const int above = dw - sw0;
  int adj = 0, inter = 0;
  if ((long long)n0 * ilog2p1(above) <= (long long)above * ilog2p1(n0)) {
    for (int i0 = 0; i0 < n0; i0 += W) {
      const int i = i0 + gl;
      if (i < n0 && contains(Nw + sw0, above, __ldg(E0 + i))) {
        ++inter;
        adj += i > it ? 1 : 0;
      }
      __syncwarp(gmask);
    }
  } else {
    for (int i0 = sw0; i0 < dw; i0 += W) {
      const int i = i0 + gl;
      const int x = i < dw ? Nw[i] : 0;
      if (i < dw && contains(E0, n0, x)) {
        ++inter;
        adj += x > w ? 1 : 0;
      }
      __syncwarp(gmask);
    }
  }
  s[0] += (gl == 0 ? n0 - it - 1 : 0) - adj;
  s[1] += (gl == 0 ? above : 0) - inter;
  s[2] += adj;
}

// Runs one task on the calling warp (all 32 lanes). level 0: second vertices [bb, ee) of v0
// (task_range encoding); level L >= 1: replay path[0..L-1], then expand positions [bb, ee) of
// E_L (group 0 only). The sweep counters are zero (motif_zero_sweeps). ROWS: narrow groups may sweep a row
// per lane (the batch kernel, short of registers, leaves that out: k = 4 with 8 lanes 1.15 ms with it,
// 1.05 without). Adds the task's subgraphs to hist; nodes counts expansions (every
// lane of a group counts the same nodes; the caller keeps group leaders' counts only).
template <int K, int W, bool ROWS = true>
__device__ __forceinline__ void motif_run_task(const MotifCtx& c, const ClassHist& hist, MotifShared* ws,
                                               int2* warp_arena, uint32_t* warp_bits, int v0, int bb, int ee,
                                               int level, const int* path, unsigned long long& nodes) {
  static_assert(W == 8 || W == 16 || W == 32, "virtual warp width must be 8, 16 or 32");
  const int lane = lane_id();
  const int gl = lane & (W - 1);
  const int gi = lane / W;
  const unsigned gmask = (W == 32) ? FULL_MASK : (((1u << W) - 1u) << (gi * W));
  const int gsrc = gi * W;  // the group leader's lane
  // the warp's words (motif_warp_smem)
  MotifGroup* const groups = reinterpret_cast<MotifGroup*>(ws + 1);
  MotifSweep<K>* const sweeps = reinterpret_cast<MotifSweep<K>*>(groups + 32 / W);
  MotifGroup* sg = groups + gi;
  MotifSweep<K>* sw = sweeps + gi;
  MotifLists<W>* const sl = reinterpret_cast<MotifLists<W>*>(sweeps + 32 / W) + gi;
  // level t (1..K-3): extension list E_t at ext_at(t); run t at run_at(t) (no pointer
  // tables, so nothing indexed dynamically lives in local memory)
  int2* const arena = warp_arena + (size_t)gi * c.arena_stride;
  const size_t md = (size_t)c.maxdeg;
  auto ext_at = [&](int t) -> int2* { return arena + md * (size_t)(t * (t + 1) / 2 - 1) + 32 * (size_t)(t - 1); };
  int2* const runs1 = ext_at(K - 2);
  auto run_at = [&](int t) -> int* { return reinterpret_cast<int*>(runs1 + (size_t)(t - 1) * (md + 32)); };
  // (k = 3 has a single level and uses binary searches only)
  constexpr bool use_bits = K >= 4;
  const MotifBits<K> bits{use_bits ? warp_bits + (size_t)gi * MotifBits<K>::STRIDE * c.bit_words : nullptr, c.bit_base};
  int bdepth = 0;         // levels 1..bdepth have their bits set
  bool top_small = true;  // the lists of level K-3 are in shared memory
  auto ext_of = [&](int t) -> int2* { return t == K - 3 && top_small ? sl->ext : ext_at(t); };
  auto run_of = [&](int t) -> int* { return t == K - 3 && top_small ? sl->run : run_at(t); };
  unsigned long long task_cnt = 0;
  long long pairs3[3] = {0, 0, 0};  // k = 3
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
  if constexpr (use_bits)
    for (int i = gl; i < n0; i += W) bits.set(__ldg(E0 + i), 0);
  MotifDemand dm;  // group leader
  if (K > 3 && gl == 0) motif_sample(c.lb, dm);
  // k = 3: no look at the demand before a donation is allowed, then one every 2,048 cycles (a look waits
  // for words that every idle warp polls)
  long long look = clock64() + (c.lb.donate_after_ns == 0 ? 0 : 2 * c.lb.donate_after_ns);
  unsigned long long checked = nodes;
  __syncwarp();
  // drops the bits of levels from..bdepth (the group's lanes, then a group barrier)
  auto drop_levels = [&](int from) {
    for (int L = bdepth; L >= from; --L) {
      const int* Rl = run_of(L);
      for (int i = gl; i < sg->runn[L]; i += W) bits.clear(Rl[i], 0);
      if (L == K - 3) {
        const int2* El = ext_of(L);
        for (int i = gl; i < sg->n[L]; i += W) {
          const int2 e = El[i];
#pragma unroll
          for (int q = 0; q <= K - 3; ++q)
            if ((e.y >> q) & 1) bits.clear(e.x, 1 + q);
        }
      }
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
          bool kept = false;
          if constexpr (K == 3) {
            if (clock64() >= look) {
              kept = range_maybe_donate(c.lb, &ws->range, v0, &ws->donations_left, t_start, &ws->busy, ob, oe, n0);
              look = clock64() + (c.lb.donate_after_ns == 0 ? 0 : 2048);
            }
          } else {
            kept = motif_wanted(c.lb, ws, dm, t_start) &&
                   range_split_donate(c.lb, &ws->range, v0, &ws->donations_left, &ws->busy, ob, oe, n0, 0, 0, nullptr);
          }
          if (kept) {
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
      leaf_pairs<W>(c, E0, n0, it, v0, gl, gmask, pairs3);
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
        // inherited members: e in E_t with e > w (E_0 is sorted: those after index it)
        const int2* Et = t == 0 ? nullptr : ext_at(t);
        const int nE = t == 0 ? n0 : sg->n[t];
        drop_levels(p);  // the previous member's sets at levels >= p
        const int sw0 = dw <= 2 * W ? 0 : lower_bound(Nw, 0, dw, v0 + 1);
        if (p == K - 3) top_small = (t == 0 ? n0 - it - 1 : nE) + (dw - sw0) <= MotifLists<W>::CAP;
        int2* const Ep = ext_of(p);
        int* const Rp = run_of(p);
        // N(w) above v0: marked, and listed as run p where outside U_t
        int rn = 0;
        for (int i0 = sw0; i0 < dw; i0 += W) {
          const int i = i0 + gl;
          const int x = i < dw ? __ldg(Nw + i) : 0;
          const bool above = i < dw && x > v0;
          bool nw = false;
          if (above) {
            nw = !(bits.at(x)[0] & bits.bit(x));
            bits.set(x, MotifBits<K>::MARK);
          }
          const unsigned bal = __ballot_sync(gmask, nw) >> gsrc;
          if (nw) Rp[rn + __popc(bal & ((1u << gl) - 1u))] = x;
          rn += __popc(bal);
        }
        __syncwarp(gmask);
        // the inherited members, with their bit for w
        int m = 0;
        for (int i0 = t == 0 ? it + 1 : 0; i0 < nE; i0 += W) {
          const int i = i0 + gl;
          int2 e = make_int2(-1, 0);
          if (i < nE) e = t == 0 ? make_int2(__ldg(E0 + i), 1) : Et[i];
          const bool keep = e.x > w;
          const unsigned bal = __ballot_sync(gmask, keep) >> gsrc;
          if (keep) {
            if (p == K - 3) {
#pragma unroll
              for (int q = 0; q < K - 3; ++q)
                if ((e.y >> q) & 1) bits.set(e.x, 1 + q);
            }
            if (bits.at(e.x)[MotifBits<K>::MARK] & bits.bit(e.x)) e.y |= 1 << p;
            Ep[m + __popc(bal & ((1u << gl) - 1u))] = e;
          }
          m += __popc(bal);
        }
        __syncwarp(gmask);
        // the marks: dropped, but at level K - 3 they stay as the members' bit for w (new vertices and
        // inherited members; a vertex of U_t that is no member has no other bit)
        for (int i = sw0 + gl; i < dw; i += W) {
          const int x = __ldg(Nw + i);
          if (x <= v0) continue;
          bool stays = false;
          if (p == K - 3) {
            bool in_u;
            unsigned mask;
            bits.look(x, in_u, mask);
            stays = !in_u || (mask & ((1u << (K - 3)) - 1u)) != 0u;
          }
          if (!stays) bits.clear(x, MotifBits<K>::MARK);
        }
        __syncwarp(gmask);
        for (int j = gl; j < rn; j += W) {
          const int x = Rp[j];
          Ep[m + j] = make_int2(x, 1 << p);
          bits.set(x, 0);
        }
        m += rn;
        bdepth = p;
        __syncwarp(gmask);
        if (p < level) {
          // replaying a donated prefix: the path fixes the member expanded at level p
          const int idx = (p < QPATH) ? path[p] : -1;
          if (idx < 0 || idx >= m) {
            if (gl == 0) set_err(c.lb.ctr, ERR_BAD_TASK);
            bdepth = p - 1;  // (its lists are not recorded; the host clears the bits of a failed call)
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
          task_cnt += leaf_sweep<K, W, ROWS>(c, hist, sw, Ep, m, first_pos, &sg->lim[p], v0, quick_p, bits, gl, gsrc, gmask,
                                       [&](int next) {
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
      drop_levels(1);
      if (bad) break;
    }
  }
  if constexpr (use_bits)
    for (int i = gl; i < n0; i += W) bits.clear(__ldg(E0 + i), 0);
  __syncwarp();
  if constexpr (K == 3) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const unsigned long long x = warp_sum_u64((unsigned long long)pairs3[m]);
      if (lane == 0 && x) {
        hist.add(__ldg(c.q2c + m + 1), x);
        task_cnt += x;
      }
    }
  }
  if (c.per_root) {
    const unsigned long long tsum = warp_sum_u64(task_cnt);
    if (lane == 0 && tsum) atomicAdd(c.per_root + v0, tsum);
  }
  if (lane == 0) lb_task_time(c.lb, t_start, v0);
}

}  // namespace dmb
