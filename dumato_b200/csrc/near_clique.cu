// The reference's pattern-aware queries q4..q13 (src/main/q4_PA.cu .. q13_PA.cu; extension
// steps DuMatoGPU.cu:1222-1445): query q_n grows an (n-2)-clique v_0 < .. < v_{n-3}
// (extend_single from v_0 above v_0, then `intersect` of the previous set with N(v_l) above
// v_l), then takes v_{n-2} from the common neighbourhood of the clique (extend_single +
// intersect_unique over every clique vertex) and v_{n-1} from the same set above v_{n-2}
// (copy_extensions), counting at the last level. Every embedding it counts is therefore an
// (n-2)-clique C plus an unordered pair of vertices adjacent to all of C - a non-induced copy
// of K_n minus one edge - and the count is
//     q_n = sum over (n-2)-cliques C of  t_C (t_C - 1) / 2,   t_C = |common neighbourhood of C|.
//
// Here an (n-2)-clique C is found once on the degree-ordered DAG, from its two lowest-ranked
// vertices r -> v, and one warp takes each DAG edge. Every other vertex of C and every common
// neighbour of C lies in N(r) cap N(v), the edge's triangles, so the warp lists that universe
// (the members of it that r and v both point to first: the candidates for C, ascending), builds
// one bitmap row over the universe per candidate, and from there only ANDs rows:
// X = the universe cap the rows of the members chosen so far holds both the candidates left and
// the common neighbours, and t_C = popc(X & row of the last member), one last member per lane.
// Edges are numbered by descending out-degree of r, so the heaviest start first, and claimed in
// runs from a cursor. A claim is laid out with an edge per lane, and where out-degrees are small the
// candidates of all its edges are searched side by side first, since most edges of a sparse graph have
// too few: one edge after the other, q_5 of a random graph of 50,000 / 200,000 took 320 us, now 129
// (claims of one to three edges go on directly: q_6 of the R-MAT graph below 66 us, 70 with the search).
//
// Bound by the dependent loads of the membership searches that build the rows (one binary search
// in an out-row per universe vertex and candidate, 32 side by side); the counting is AND + popc
// from shared memory. Taking a whole root per warp and intersecting undirected adjacency lists
// for every clique again, as this kernel did before, read whole rows per clique and left the
// heaviest roots on one warp each: q_6 on an R-MAT graph of 1,377 vertices and 8,000 edges took
// 7,867 us per call, now 64 us (41 us of them this kernel).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <string>

#include "engine.hpp"
#include "gpm.cuh"
#include "lb.cuh"

namespace dmb {

struct NearArgs {
  GraphView dag;            // rank-space out-lists
  const int32_t* in_end;    // in-lists (census_in_lists)
  const int32_t* in_deg;
  const int2* in;
  const int32_t* roots;     // by descending out-degree
  const int4* steps;        // (first item, first root, out-degree): runs of equal out-degree
  int n_steps, n_items;
  LBArgs lb;
  DevCounters* out;         // page-locked host memory: the counters at the end of the launch
  DevCounters* next;        // the next launch's counters, zeroed by this one
  int32_t* arena;           // per warp: list, rows, sets that do not fit shared memory; or null
  size_t arena_ints;
  int list_cap;             // universe vertices an edge can have
  int max_claim;            // of light items a warp claims up to half its share, at most these (<= 32)
};

constexpr int NEAR_WARPS = 8;
// shared memory of a warp: universes of up to 256 vertices and 1,024 row words (the rest of the
// edges, a few around hubs, use the arena)
constexpr int NEAR_LIST = 256;
constexpr int NEAR_ROWS = 1024;
constexpr int NEAR_SETS = 9;  // nested sets X (n = 13 chooses nine members from the candidates)
constexpr int NEAR_WARP_INTS = NEAR_LIST + NEAR_ROWS + NEAR_SETS * (NEAR_LIST / 32);
constexpr int PAIR_CHUNK = 256;       // pairs of out-neighbours a warp takes together (q_4)
constexpr int NEAR_LIGHT = 32;        // out-degrees up to which a claim's candidates are searched together
constexpr unsigned NEAR_TELL = 64;  // steps of an item between two reports of progress

// Adds t (t - 1) / 2 over the cliques that extend the members chosen so far by LEFT more
// candidates from index `start` on. X: the candidates and common neighbours left (null: the whole
// universe); sets: room for the sets below. Warp-uniform but for the last member. `nodes` counts the
// members chosen before the last two; every NEAR_TELL of them are reported as progress.
template <int LEFT>
__device__ __forceinline__ void near_dfs(const uint32_t* rows, int W, int m, const uint32_t* X, uint32_t* sets, int start,
                                         unsigned long long& total, unsigned& nodes, DevCounters* ctr) {
  const int lane = lane_id();
  if constexpr (LEFT == 1) {
    for (int j = start + lane; j < m; j += 32) {
      if (X && !((X[j >> 5] >> (j & 31)) & 1u)) continue;
      unsigned t = 0;
      for (int w = 0; w < W; ++w) t += __popc(rows[j * W + w] & (X ? X[w] : 0xffffffffu));
      total += (t & 1) ? (unsigned long long)t * ((t - 1) >> 1) : (unsigned long long)(t >> 1) * (t - 1u);
    }
  } else {
    for (int j = start; j <= m - LEFT; ++j) {
      if (X && !((X[j >> 5] >> (j & 31)) & 1u)) continue;
      if constexpr (LEFT >= 3) {
        if (++nodes % NEAR_TELL == 0u && lane == 0) atomicAdd(&ctr->progress, (unsigned long long)NEAR_TELL);
      }
      const uint32_t* Y = rows + (size_t)j * W;
      if (X) {
        for (int w = lane; w < W; w += 32) sets[w] = X[w] & Y[w];
        __syncwarp();
        Y = sets;
      }
      // candidates left above j
      int left = 0;
      for (int w = (j + 1) >> 5; w <= (m - 1) >> 5; ++w) {
        uint32_t b = Y[w];
        if (w == (j + 1) >> 5) b &= 0xffffffffu << ((j + 1) & 31);
        if (w == (m - 1) >> 5) b &= 0xffffffffu >> (31 - ((m - 1) & 31));
        left += __popc(b);
      }
      if (left >= LEFT - 1) near_dfs<LEFT - 1>(rows, W, m, Y, X ? sets + W : sets, j + 1, total, nodes, ctr);
      __syncwarp();
    }
  }
}

template <int C>
__global__ void __launch_bounds__(32 * NEAR_WARPS) near_clique_kernel(const __grid_constant__ NearArgs a) {
  __shared__ int32_t smem[NEAR_WARPS][NEAR_WARP_INTS];
  const int lane = lane_id();
  const int wib = warp_in_block();
  const int total_warps = gridDim.x * NEAR_WARPS;
  int32_t* own = smem[wib];
  int32_t* arena = a.arena ? a.arena + (size_t)(blockIdx.x * NEAR_WARPS + wib) * a.arena_ints : nullptr;
  DevCounters* ctr = a.lb.ctr;
  unsigned long long total = 0;
  unsigned nodes = 0;
  while (true) {
    int first = 0, count = 0;
    if (lane == 0) {
      const int left = a.n_items - vload(&ctr->cursor);
      const int chunk = max(1, max(min(16, left / (8 * total_warps)), min(a.max_claim, left / (2 * total_warps))));
      first = left > 0 ? atomicAdd(&ctr->cursor, chunk) : a.n_items;
      count = min(chunk, a.n_items - first);
    }
    first = __shfl_sync(FULL_MASK, first, 0);
    count = __shfl_sync(FULL_MASK, count, 0);
    if (count <= 0) break;
    // lane l: item first + l, out-edge i of a root, found through the runs of roots of equal out-degree
    int my_d = 0, my_i = 0, my_nin = 0, my_row = 0, my_v = 0, my_rv = 0, my_nb = 0, my_in = 0;
    if (lane < count) {
      const int e = first + lane;
      int lo = 0, hi = a.n_steps;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&a.steps[mid].x) <= e) lo = mid; else hi = mid;
      }
      const int4 st = __ldg(a.steps + lo);
      my_d = st.z;
      const int o = (e - st.x) / my_d;
      my_i = (e - st.x) - o * my_d;
      if (my_d - 1 - my_i >= C - 2) {
        const int r = __ldg(a.roots + st.y + o);
        my_row = __ldg(a.dag.row + r);
        my_nin = __ldg(a.in_deg + r);
        my_in = __ldg(a.in_end + r) - my_nin;
        my_v = __ldg(a.dag.adj + my_row + my_i);
        my_rv = __ldg(a.dag.row + my_v);
        my_nb = __ldg(a.dag.deg + my_v);
      }
    }
    bool mine = lane < count && my_d - 1 - my_i >= C - 2;
    if (C > 2 && count >= 4 && __shfl_sync(FULL_MASK, my_d, 0) <= NEAR_LIGHT) {
      // light items: all their candidates side by side first, and only those with enough of them on
      const int len = mine ? my_d - 1 - my_i : 0;
      int off = len;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int y = __shfl_up_sync(FULL_MASK, off, s);
        if (lane >= s) off += y;
      }
      const int all = __shfl_sync(FULL_MASK, off, 31);
      off -= len;
      int found = 0;
      for (int f0 = 0; f0 < all; f0 += 32) {
        const int f = f0 + lane;
        int j = 0;  // owner: the last item whose candidates start at or before f
#pragma unroll
        for (int h = 16; h >= 1; h >>= 1) {
          const int x = __shfl_sync(FULL_MASK, off, j + h);
          j = x <= f ? j + h : j;
        }
        const int at = __shfl_sync(FULL_MASK, my_row + my_i + 1 - off, j) + f;
        const int rv = __shfl_sync(FULL_MASK, my_rv, j), nb = __shfl_sync(FULL_MASK, my_nb, j);
        const bool hit = f < all && contains(a.dag.adj + rv, nb, __ldg(a.dag.adj + at));
        const unsigned bal = __ballot_sync(FULL_MASK, hit);
        const int a0 = min(max(off - f0, 0), 32), a1 = min(max(off + len - f0, 0), 32);
        const unsigned upto1 = a1 >= 32 ? 0xffffffffu : (1u << a1) - 1u;
        const unsigned upto0 = a0 >= 32 ? 0xffffffffu : (1u << a0) - 1u;
        found += __popc(bal & upto1 & ~upto0);
      }
      mine = mine && found >= C - 2;
    }
    for (unsigned todo = __ballot_sync(FULL_MASK, mine); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const int d = __shfl_sync(FULL_MASK, my_d, src), i = __shfl_sync(FULL_MASK, my_i, src);
      const int nin = __shfl_sync(FULL_MASK, my_nin, src), v = __shfl_sync(FULL_MASK, my_v, src);
      const int nb = __shfl_sync(FULL_MASK, my_nb, src);
      const int32_t* L = a.dag.adj + __shfl_sync(FULL_MASK, my_row, src);
      const int32_t* B = a.dag.adj + __shfl_sync(FULL_MASK, my_rv, src);
      const int2* I = a.in + __shfl_sync(FULL_MASK, my_in, src);
      int32_t* uni = d + nin <= NEAR_LIST ? own : arena;
      // candidates: above v, and out-neighbours of both
      int m = 0;
      for (int j0 = i + 1; j0 < d; j0 += 32) {
        const int j = j0 + lane;
        const int y = j < d ? __ldg(L + j) : 0;
        m += compact(uni, m, y, j < d && contains(B, nb, y));
      }
      if (m < C - 2) continue;
      // the other common neighbours lie below v: v is in their out-row
      int u = m;
      for (int j0 = 0; j0 < i; j0 += 32) {
        const int j = j0 + lane;
        const int y = j < i ? __ldg(L + j) : 0;
        u += compact(uni, u, y, j < i && contains(a.dag.adj + __ldg(a.dag.row + y), __ldg(a.dag.deg + y), v));
      }
      for (int j0 = 0; j0 < nin; j0 += 32) {
        const int j = j0 + lane;
        const int y = j < nin ? __ldg(&I[j].x) : 0;
        u += compact(uni, u, y, j < nin && contains(a.dag.adj + __ldg(a.dag.row + y), __ldg(a.dag.deg + y), v));
      }
      __syncwarp();
      if constexpr (C == 2) {
        if (lane == 0) total += (u & 1) ? (unsigned long long)u * ((u - 1) >> 1) : (unsigned long long)(u >> 1) * (u - 1);
      } else {
        const int W = (u + 31) >> 5;
        const bool small = u <= NEAR_LIST && m * W <= NEAR_ROWS;
        uint32_t* rows = reinterpret_cast<uint32_t*>(small ? own + NEAR_LIST : arena + a.list_cap);
        uint32_t* sets = small ? rows + NEAR_ROWS : rows + (size_t)m * W;
        for (int w = 0; w < W; ++w) {
          const int q = w * 32 + lane;
          const int y = q < u ? uni[q] : 0;
          const int32_t* Ny = a.dag.adj + __ldg(a.dag.row + y);
          const int ny = __ldg(a.dag.deg + y);
          for (int j = 0; j < m; ++j) {
            const int c = uni[j];
            bool adj = false;
            if (q < u && y < c) adj = contains(Ny, ny, c);
            if (q < u && y > c) adj = contains(a.dag.adj + __ldg(a.dag.row + c), __ldg(a.dag.deg + c), y);
            const unsigned bits = __ballot_sync(FULL_MASK, adj);
            if (lane == 0) rows[j * W + w] = bits;
          }
          if ((w & 63) == 63 && lane == 0) atomicAdd(&ctr->progress, 64ull);
        }
        __syncwarp();
        near_dfs<C - 2>(rows, W, m, nullptr, sets, 0, total, nodes, ctr);
      }
      __syncwarp();
    }
    if (lane == 0) atomicSub(&ctr->pending, count);
  }
  if (lane == 0 && a.lb.test_stall) lb_stall(a.lb);
  total = warp_sum_u64(total);
  if (lane == 0 && total) atomicAdd(&ctr->count, total);
  counters_to_host(ctr, a.next, a.out);
}

template <int C>
static int launch_near(const NearArgs& a, LaunchCtx& ctx, int* grid_out) {
  const int block = 32 * NEAR_WARPS;
  auto kern = near_clique_kernel<C>;
  static LaunchCache cache;
  int occ = 0;
  DM_CUDA(cached_occupancy(cache, kern, ctx.device, block, 0, &occ));
  if (occ < 1) return fail(DM_EINVAL, "near-clique kernel does not fit on an SM");
  int grid = std::min(ctx.num_sms * occ, (a.n_items + NEAR_WARPS - 1) / NEAR_WARPS);
  if (ctx.threads > 0) grid = std::max(1, std::min(grid, (ctx.threads + block - 1) / block));
  if (a.arena && grid * NEAR_WARPS > ctx.arena_warps) grid = std::max(1, ctx.arena_warps / NEAR_WARPS);
  kern<<<grid, block, 0, ctx.stream>>>(a);
  ctx.launches++;
  *grid_out = grid;
  DM_CUDA(cudaGetLastError());
  return DM_OK;
}

// ---------------- q_4: pairs of triangles on an edge ----------------

// q_4 = sum over edges of t (t - 1) / 2 with t the triangles on the edge. Every triangle is found once
// on the DAG, from its lowest vertex r: a pair (v, y) of r's out-neighbours, v < y, joined by an edge,
// which is found at its place in v's row; it adds one to the counters of its three edges. The pairs of
// all roots are numbered end to end (pair_step: the first pair of each run of roots of equal
// out-degree), so a root of any size spreads over the grid.
//
// Bound by the dependent loads of the searches, one per pair of out-neighbours. Edge by edge
// (near_clique_kernel<2>), every neighbour of a vertex is searched for each of its out-edges and every
// triangle is met three times: q_4 takes 6.9 ms on an R-MAT graph of 98,552 vertices / 1.08M edges,
// 0.52 on a Chung-Lu graph of 18,700 / 198,000 and 13.7 on a random graph of 4,000 with edge
// probability 0.1, here 0.31, 0.053 and 1.3 (a warp per root, merging undirected lists, took
// 3.5, 0.36 and 3.5). On small graphs one launch is faster than two (engine.cu NEAR4_STEPS).
__global__ void __launch_bounds__(256) near_triangle_kernel(const __grid_constant__ NearArgs a, unsigned* tri,
                                                            const long long* pair_step, long long n_pairs) {
  const int lane = lane_id();
  const long long warps = (long long)gridDim.x * NEAR_WARPS;
  unsigned chunks = 0;
  for (long long q0 = ((long long)blockIdx.x * NEAR_WARPS + warp_in_block()) * PAIR_CHUNK; q0 < n_pairs;
       q0 += warps * PAIR_CHUNK) {
    // the run of the chunk's first pair
    int s = 0, hi = a.n_steps;
    while (hi - s > 1) {
      const int mid = (s + hi) >> 1;
      if (__ldg(pair_step + mid) <= q0) s = mid; else hi = mid;
    }
    for (int c = 0; c < PAIR_CHUNK; c += 32) {
      const long long q = q0 + c + lane;
      if (q >= n_pairs) break;
      while (__ldg(pair_step + s + 1) <= q) ++s;
      const int4 st = __ldg(a.steps + s);
      const int d = st.z;
      const long long rel = q - __ldg(pair_step + s);
      const unsigned P = (unsigned)((long long)d * (d - 1) / 2);
      unsigned o, p;
      if (rel <= 0xffffffffll) {
        o = (unsigned)rel / P;
        p = (unsigned)rel - o * P;
      } else {
        o = (unsigned)(rel / P);
        p = (unsigned)(rel - (long long)o * P);
      }
      // p = m (m - 1) / 2 + b with 0 <= b < m: v is the m-th out-neighbour from the end
      unsigned m = (unsigned)((1.f + sqrtf(1.f + 8.f * (float)p)) * 0.5f);
      while ((unsigned long long)m * (m - 1) / 2 > p) --m;
      while ((unsigned long long)m * (m + 1) / 2 <= p) ++m;
      const int i = d - 1 - (int)m, j = i + 1 + (int)(p - (unsigned)((unsigned long long)m * (m - 1) / 2));
      const int rr = __ldg(a.dag.row + __ldg(a.roots + st.y + (int)o));
      const int v = __ldg(a.dag.adj + rr + i), y = __ldg(a.dag.adj + rr + j);
      const int rv = __ldg(a.dag.row + v), nv = __ldg(a.dag.deg + v);
      const int at = lower_bound(a.dag.adj + rv, 0, nv, y);
      if (at < nv && __ldg(a.dag.adj + rv + at) == y) {
        atomicAdd(tri + rr + i, 1u);
        atomicAdd(tri + rr + j, 1u);
        atomicAdd(tri + rv + at, 1u);
      }
    }
    __syncwarp();
    if ((++chunks & 63u) == 0u && lane == 0) atomicAdd(&a.lb.ctr->progress, 64ull * PAIR_CHUNK);
  }
}

// The sum over all edges (padding holds no triangle), or over those of the listed roots (a shard).
__global__ void __launch_bounds__(256) near_pairs_kernel(const __grid_constant__ NearArgs a, const unsigned* tri, int64_t n,
                                                         const int32_t* roots, int n_roots) {
  const int t = blockIdx.x * 256 + threadIdx.x, T = gridDim.x * 256;
  auto pairs = [](unsigned x) -> unsigned long long {
    return (x & 1) ? (unsigned long long)x * ((x - 1) >> 1) : (unsigned long long)(x >> 1) * (x - 1u);
  };
  unsigned long long total = 0;
  if (roots) {
    for (int i = t >> 5; i < n_roots; i += T >> 5) {
      const int r = __ldg(roots + i), b = __ldg(a.dag.row + r), d = __ldg(a.dag.deg + r);
      for (int j = lane_id(); j < d; j += 32) total += pairs(tri[b + j]);
    }
  } else {
    for (int64_t i = t; i < n; i += T) total += pairs(tri[i]);
  }
  if (lane_id() == 0 && a.lb.test_stall) lb_stall(a.lb);
  total = warp_sum_u64(total);
  if (lane_id() == 0 && total) atomicAdd(&a.lb.ctr->count, total);
  if (t == 0) {
    atomicSub(&a.lb.ctr->pending, a.n_items);
    atomicAdd(&a.lb.ctr->progress, (unsigned long long)a.n_items);
  }
  counters_to_host(a.lb.ctr, a.next, a.out);
}

static int launch_near4(const NearArgs& a, const NearLaunch& L, LaunchCtx& ctx, int* grid_out) {
  auto grid_for = [&](int64_t blocks) {
    if (ctx.threads > 0) blocks = std::min<int64_t>(blocks, (ctx.threads + 255) / 256);
    return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, ctx.num_sms * 8));
  };
  DM_CUDA(cudaMemsetAsync(L.tri, 0, sizeof(unsigned) * L.tri_words, ctx.stream));
  const int grid = grid_for((L.n_pairs + PAIR_CHUNK * NEAR_WARPS - 1) / (PAIR_CHUNK * NEAR_WARPS));
  if (L.n_pairs > 0) {
    near_triangle_kernel<<<grid, 256, 0, ctx.stream>>>(a, L.tri, L.pair_step, L.n_pairs);
    ctx.launches++;
    DM_CUDA(cudaGetLastError());
  }
  const int64_t work = L.shard ? (int64_t)L.shard_roots * 32 : (int64_t)L.tri_words;
  near_pairs_kernel<<<grid_for((work + 1023) / 1024), 256, 0, ctx.stream>>>(a, L.tri, (int64_t)L.tri_words, L.shard,
                                                                           L.shard_roots);
  ctx.launches++;
  *grid_out = grid;
  DM_CUDA(cudaGetLastError());
  return DM_OK;
}

int near_clique_launch(const NearLaunch& L, LaunchCtx& ctx, int* grid) {
  NearArgs a;
  a.dag = L.dag;
  a.in_end = L.in_end;
  a.in_deg = L.in_deg;
  a.in = reinterpret_cast<const int2*>(L.in);
  a.roots = L.roots;
  a.steps = reinterpret_cast<const int4*>(L.steps);
  a.n_steps = L.n_steps;
  a.n_items = L.n_items;
  a.lb = LBArgs{};
  a.lb.ctr = L.ctr;
  a.lb.timeout_ns = (long long)ctx.timeout_ms * 1000000ll;
  a.lb.test_stall = ctx.test_stall;
  a.out = L.out;
  a.next = L.next;
  a.arena = L.arena;
  a.arena_ints = L.arena_ints;
  a.list_cap = L.list_cap;
  a.max_claim = L.max_claim;
  if (L.tri) return launch_near4(a, L, ctx, grid);
  switch (L.c) {
    case 2: return launch_near<2>(a, ctx, grid);
    case 3: return launch_near<3>(a, ctx, grid);
    case 4: return launch_near<4>(a, ctx, grid);
    case 5: return launch_near<5>(a, ctx, grid);
    case 6: return launch_near<6>(a, ctx, grid);
    case 7: return launch_near<7>(a, ctx, grid);
    case 8: return launch_near<8>(a, ctx, grid);
    case 9: return launch_near<9>(a, ctx, grid);
    case 10: return launch_near<10>(a, ctx, grid);
    case 11: return launch_near<11>(a, ctx, grid);
    default: return fail(DM_EINVAL, "near-clique queries take n in [4, 13]");
  }
}

// Ints of a warp's arena for edges of roots of out-degree d and degree `deg` (0: shared memory
// holds every edge's universe, rows and sets).
size_t near_clique_rows(int d, int deg) {
  const size_t W = ((size_t)deg + 31) / 32, rows = (size_t)std::max(d - 1, 0) * W;
  return deg <= NEAR_LIST && rows <= NEAR_ROWS ? 0 : rows + NEAR_SETS * W;
}

}  // namespace dmb
