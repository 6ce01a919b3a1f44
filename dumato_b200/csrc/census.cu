// Census of the connected 3- and 4-vertex classes of a whole graph without enumerating them
// (k = 3, 4 motifs with the plain schedule, unsharded, no subtree log).
//
// The enumerating kernel (motif.cuh) visits every connected (k-1)-subgraph; on a graph with hubs
// that is billions of prefixes. The class counts of k <= 4 follow exactly from a few sums over
// edges, triangles, 4-cliques and 4-cycles (inclusion-exclusion between copies and induced
// copies; the formulas are the ones of the 4-vertex graphlet counts of Ahmed, Neville, Rossi and
// Duffield, "Efficient graphlet counting for large networks", ICDM 2015):
//   T   triangles, K4 4-cliques, C4 4-cycles (copies), t_e triangles on edge e, d degrees
//   k=3: triangle T; wedge  sum C(d,2) - 3 T
//   k=4: diamond dia = sum_e C(t_e,2) - 6 K4;  cycle cyc = C4 - dia - 3 K4
//        paw     paw = sum over triangles (d_a + d_b + d_c - 6) - 4 dia - 12 K4
//        path    sum_e (d_a - 1)(d_b - 1) - 3 T - 2 paw - 4 cyc - 6 dia - 12 K4
//        star    sum C(d,3) - paw - 2 dia - 4 K4
// Every sum is taken modulo 2^64 without a division, so the results are exact modulo 2^64.
//
// T, t_e and K4 come from the clique index (rows = local adjacency bitmaps of the degree-ordered
// DAG); C4 and the rest of t_e from a walk over two-paths: for every vertex u, each two-path
// u - v - x with v, x below u in rank adds one to a counter c_u[x]. A 4-cycle is counted once,
// at its highest vertex u and the vertex x opposite to it (sum of C(c_u[x], 2), taken as the sum
// of the counters' old values), and c_u[w] for an edge (w, u) is the number of triangles on it
// whose third vertex is below u; those with the third vertex above u are the popcount of row u
// of w's bitmap (`up`). Since the walk only goes down in degree order it makes
// sum over edges of min-degree-bounded steps (Chiba and Nishizeki 1985).
//
// What bounds it: random 4- and 8-byte gathers that hit L2 (the arrays are far below 126 MB) and
// shared-memory atomics, one pair per two-path. Vertices with few two-paths (most of them) are
// taken by one warp each with a hash table of its own (SMALL_PATHS); the others by a block each
// with direct 16-bit counters over the ranks below u, cleared in a few 16-byte stores per thread.
// Measured per call, enumeration before: k = 3 on an R-MAT graph of 98,552 vertices and 1.08M edges
// 2,981 -> 29 us; k = 4 on a Chung-Lu graph of 18,700 vertices and 198,000 edges 12,994 -> 157 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <string>

#include "engine.hpp"
#include "gpm.cuh"

namespace dmb {

// sums[]: k = 4: rows kernel, then the two-path kernels; k = 3: triangles, wedges
enum { CENSUS_STAR, CENSUS_TRI, CENSUS_EDGE, CENSUS_PAW, CENSUS_K4, CENSUS_C4, CENSUS_DIA, CENSUS_PAW_TOP };
enum { FLAT_TRI, FLAT_WEDGE, FLAT_SUMS };
static_assert(CENSUS_PAW_TOP + 1 == CENSUS_SUMS, "engine.hpp sizes the buffer");

// A vertex's in-list entry: v -> u, and the place of u in v's padded out-row (the edge's id).
using InEdge = int2;

struct CensusArgs {
  GraphView g;               // rank-space DAG (padded out-rows)
  const int32_t* ud;         // degree by rank
  const uint4* blocks;       // clique index
  const uint32_t* boff;
  const int32_t* in_end;     // in-list of u: entries [in_end[u] - in_deg[u], in_end[u])
  const int32_t* in_deg;
  const InEdge* in;
  uint32_t* up;              // by edge id: triangles on the edge whose third vertex is above both
  unsigned long long* sums;  // CENSUS_SUMS
  int* list;                 // vertices left to the block kernel
  int* ctl;                  // [0] length of list, [1] warp cursor, [2] block cursor, [3] blocks done
  unsigned long long* out;   // page-locked host memory: the sums at the end of the launches
  const int32_t* order;      // ranks by descending out-degree
  int n_wide;                // of them, those with 32 or more out-neighbours
  int base;                  // first rank with degree >= 2 (lower ranks lie on no cycle)
};

// ---------------- in-lists (laid out once per device copy) ----------------

__global__ void __launch_bounds__(256) in_count_kernel(GraphView g, int32_t* __restrict__ deg) {
  // (eight threads per rank: beyond 32 bits from 2^29 ranks on)
  const int r = (int)((blockIdx.x * 256ll + threadIdx.x) >> 3), l = threadIdx.x & 7;
  if (r >= g.n) return;
  const int32_t* L = g.adj + g.row[r];
  for (int i = l; i < g.deg[r]; i += 8) atomicAdd(deg + L[i], 1);
}

// Each in-list takes a run of the pool; the order of the runs does not matter, so one bump
// pointer (an atomic per warp) stands in for a scan. pos: the next free place of each list.
__global__ void __launch_bounds__(256) in_place_kernel(const int32_t* __restrict__ deg, int n,
                                                       int32_t* __restrict__ pos, int* __restrict__ pool) {
  const int v = blockIdx.x * 256 + threadIdx.x, lane = lane_id();
  const int d = v < n ? deg[v] : 0;
  int s = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL_MASK, s, o);
    if (lane >= o) s += y;
  }
  int b = 0;
  if (lane == 31 && s) b = atomicAdd(pool, s);
  b = __shfl_sync(FULL_MASK, b, 31);
  if (v < n) pos[v] = b + s - d;
}

__global__ void __launch_bounds__(256) in_fill_kernel(GraphView g, int32_t* __restrict__ pos,
                                                      InEdge* __restrict__ in) {
  // (eight threads per rank: beyond 32 bits from 2^29 ranks on)
  const int r = (int)((blockIdx.x * 256ll + threadIdx.x) >> 3), l = threadIdx.x & 7;
  if (r >= g.n) return;
  const int b = g.row[r];
  for (int i = l; i < g.deg[r]; i += 8) in[atomicAdd(pos + g.adj[b + i], 1)] = make_int2(r, b + i);
}

int census_in_lists(const GraphView& g, int32_t* in_end, int32_t* in_deg, void* in, int* pool, LaunchCtx& ctx) {
  if (g.n <= 0) return DM_OK;
  DM_CUDA(cudaMemsetAsync(in_deg, 0, sizeof(int32_t) * g.n, ctx.stream));
  DM_CUDA(cudaMemsetAsync(pool, 0, sizeof(int), ctx.stream));
  const unsigned by8 = (unsigned)(((int64_t)g.n * 8 + 255) / 256);
  in_count_kernel<<<by8, 256, 0, ctx.stream>>>(g, in_deg);
  in_place_kernel<<<(g.n + 255) / 256, 256, 0, ctx.stream>>>(in_deg, g.n, in_end, pool);
  in_fill_kernel<<<by8, 256, 0, ctx.stream>>>(g, in_end, reinterpret_cast<InEdge*>(in));
  ctx.launches += 3;
  DM_CUDA(cudaGetLastError());
  return DM_OK;
}

// ---------------- sums over vertices and over the index ----------------

// Adds one block's per-thread partial sums to sums[first ..].
template <int N>
__device__ __forceinline__ void add_sums(unsigned long long (&s)[N], unsigned long long* sums) {
  __shared__ unsigned long long tot[N];
  if (threadIdx.x < N) tot[threadIdx.x] = 0ull;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const unsigned long long v = warp_sum_u64(s[q]);
    if (lane_id() == 0 && v) atomicAdd(tot + q, v);
  }
  __syncthreads();
  if (threadIdx.x < N && tot[threadIdx.x]) atomicAdd(sums + threadIdx.x, tot[threadIdx.x]);
}

__device__ __forceinline__ unsigned long long choose2(unsigned long long d) {
  // one of d, d - 1 is even: halve that one, so the product is exact modulo 2^64
  return (d & 1) ? d * ((d - 1) >> 1) : (d >> 1) * (d - 1);
}

__device__ __forceinline__ unsigned long long choose3(unsigned long long d) {
  if (d < 3) return 0ull;
  unsigned long long a = d, b = d - 1, c = d - 2;
  if (d & 1) b >>= 1;
  else a >>= 1;
  if (a % 3 == 0) a /= 3;
  else if (b % 3 == 0) b /= 3;
  else c /= 3;
  return a * b * c;
}

// One root's share of the k = 4 sums by G lanes (l of G): stars from the degree; for every edge the popcount t of its index row (the triangles on it whose third vertex is above both);
// the 4-cliques above it, the paths' edge sum, the paws at the two lower vertices of those
// triangles, and t itself in `up`.
template <int G>
__device__ __forceinline__ void census_root(const CensusArgs& a, int r, int l, unsigned long long (&s)[5]) {
  const int d = __ldg(a.g.deg + r);
  const unsigned long long du = (unsigned long long)__ldg(a.ud + r);
  if (l == 0) s[CENSUS_STAR] += choose3(du);
  const int nw = (d + 63) >> 6;
  const uint64_t* rows = d >= 2 ? reinterpret_cast<const uint64_t*>(a.blocks + __ldg(a.boff + r)) : nullptr;
  const int b = __ldg(a.g.row + r);
  for (int i = l; i < d; i += G) {
    unsigned t = 0, q = 0;
    if (rows) {
      const uint64_t* ri = rows + (size_t)i * nw;
      for (int w = 0; w < nw; ++w) {
        uint64_t m = __ldg(ri + w);
        t += __popcll(m);
        // (members are numbered in rank order, so row j holds no bit at or below j)
        while (m) {
          const uint64_t* rj = rows + (size_t)(w * 64 + __ffsll((long long)m) - 1) * nw;
          m &= m - 1;
          for (int x = w; x < nw; ++x) q += __popcll(__ldg(ri + x) & __ldg(rj + x));
        }
      }
    }
    const unsigned long long dv = (unsigned long long)__ldg(a.ud + __ldg(a.g.adj + b + i));
    a.up[b + i] = t;
    s[CENSUS_TRI] += t;
    s[CENSUS_EDGE] += (du - 1) * (dv - 1);
    s[CENSUS_PAW] += (unsigned long long)t * (du + dv - 4);
    s[CENSUS_K4] += q;
  }
}

// All ranks in descending out-degree order: a warp per root for the wide ones (at least 32 rows),
// eight lanes per root for the others.
__global__ void __launch_bounds__(256) census_rows_kernel(const __grid_constant__ CensusArgs a) {
  unsigned long long s[5] = {0ull, 0ull, 0ull, 0ull, 0ull};
  const int t = blockIdx.x * 256 + threadIdx.x, T = gridDim.x * 256;
  for (int i = t >> 5; i < a.n_wide; i += T >> 5) census_root<32>(a, __ldg(a.order + i), t & 31, s);
  for (int i = a.n_wide + (t >> 3); i < a.g.n; i += T >> 3) census_root<8>(a, __ldg(a.order + i), t & 7, s);
  add_sums(s, a.sums);
}

// End of a call's last kernel: its last block hands the n sums to the host and zeroes them and the
// cursors for the next call, which then needs no copy before or after its launches.
__device__ __forceinline__ void census_finish(unsigned long long* sums, int* ctl, int n, unsigned long long* out) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ctl + 3, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if ((int)threadIdx.x < n) {
    volatile unsigned long long* v = sums + threadIdx.x;
    out[threadIdx.x] = *v;
    *v = 0ull;
  }
  if (threadIdx.x < 4) ctl[threadIdx.x] = 0;
}

// k = 3: triangles as the popcount of the whole index (every row bit is one triangle; the blocks
// lie end to end and their padding is zero), and with ud the wedges from the degrees. A stream of
// 16-byte loads, four in flight per thread, where staging the blocks root by root pays for the
// task list, the cursor and the wait for the last warp: triangles of a graph of 2,000 vertices took
// 35.5 us per call, now 23.7; the census of 98,552 vertices (a 20 MB index) 53 us, now 29 (9 us of
// them this kernel, 2.2 TB/s out of L2).
__global__ void __launch_bounds__(256) census_flat_kernel(const uint4* __restrict__ blocks, uint64_t units,
                                                          const int32_t* __restrict__ ud, int n,
                                                          unsigned long long* sums, int* ctl, unsigned long long* out) {
  unsigned long long s[FLAT_SUMS] = {0ull, 0ull};
  const uint64_t T = gridDim.x * 256ull, t = blockIdx.x * 256ull + threadIdx.x;
  for (uint64_t i = t; i < units; i += 4 * T) {
    uint4 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = i + q * T < units ? __ldg(blocks + i + q * T) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int q = 0; q < 4; ++q) s[FLAT_TRI] += (unsigned)(__popc(v[q].x) + __popc(v[q].y) + __popc(v[q].z) + __popc(v[q].w));
  }
  if (ud)
    for (uint64_t i = t; i < (uint64_t)n; i += T) s[FLAT_WEDGE] += choose2((unsigned long long)__ldg(ud + i));
  add_sums(s, sums);
  census_finish(sums, ctl, FLAT_SUMS, out);
}

// ---------------- two-paths below u ----------------

// One 32-entry batch of u's in-list: lane l holds in-neighbour v; the two-paths through the
// batch's vertices are numbered 0..total-1 through the exclusive prefix `off` of their row
// lengths, so the lanes stay busy whatever the rows' lengths are.
struct PathBatch {
  int off, total;        // this lane's first path, all paths
  int in0, nin, out0;    // v's in-list (start, length) and out-row start
};

__device__ __forceinline__ PathBatch path_batch(const CensusArgs& a, const InEdge* L, int i0, int n) {
  const int lane = lane_id();
  PathBatch p{0, 0, 0, 0, 0};
  int len = 0;
  if (i0 + lane < n) {
    const int v = __ldg(&L[i0 + lane].x);
    p.nin = __ldg(a.in_deg + v);
    p.in0 = __ldg(a.in_end + v) - p.nin;
    p.out0 = __ldg(a.g.row + v);
    len = p.nin + __ldg(a.g.deg + v);
  }
  int s = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL_MASK, s, o);
    if (lane >= o) s += y;
  }
  p.off = s - len;
  p.total = __shfl_sync(FULL_MASK, s, 31);
  return p;
}

// End of path f of the batch (all lanes call; f may be past the end): a vertex below u, or -1
// (u itself, a vertex above u, or a rank below `base`, which lies on no cycle).
__device__ __forceinline__ int path_end(const CensusArgs& a, const PathBatch& p, int f, int u) {
  // the last lane whose offset is at most f
  int j = 0;
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    const int o = __shfl_sync(FULL_MASK, p.off, j + h);
    j = o <= f ? j + h : j;
  }
  const int k = f - __shfl_sync(FULL_MASK, p.off, j);
  const int nin = __shfl_sync(FULL_MASK, p.nin, j);
  const int in0 = __shfl_sync(FULL_MASK, p.in0, j);
  const int out0 = __shfl_sync(FULL_MASK, p.out0, j);
  if (f >= p.total) return -1;
  const int x = k < nin ? __ldg(&a.in[in0 + k].x) : __ldg(a.g.adj + out0 + (k - nin));
  return x < u && x >= a.base ? x : -1;
}

// Vertices with at most SMALL_PATHS two-paths: a warp each, counters in a hash table of at
// least twice as many slots (linear probing, cleared per vertex). 512 paths keep 24 warps per
// SM resident; the rest goes to the list of the block kernel.
constexpr int SMALL_PATHS = 512;
constexpr int SMALL_SLOTS = 2 * SMALL_PATHS;
constexpr int SMALL_WARPS = 8;
constexpr size_t SMALL_SMEM = (size_t)SMALL_WARPS * SMALL_SLOTS * 2 * sizeof(int);

__global__ void __launch_bounds__(32 * SMALL_WARPS) census_small_kernel(const __grid_constant__ CensusArgs a) {
  extern __shared__ __align__(16) int sm[];
  const int lane = lane_id();
  int* key = sm + warp_in_block() * 2 * SMALL_SLOTS;
  unsigned* cnt = reinterpret_cast<unsigned*>(key + SMALL_SLOTS);
  unsigned long long s[3] = {0ull, 0ull, 0ull};  // cycles, diamonds, paws at the highest vertex
  // (runs of 32 on every graph left a graph of 18,700 vertices on 584 warps: 321 us)
  const int run = max(1, min(32, (a.g.n - a.base) / (4 * (int)gridDim.x * SMALL_WARPS)));
  while (true) {
    // vertices in descending rank, `run` at a time: the list of large ones starts with the hubs
    int c = 0;
    if (lane == 0) c = atomicAdd(a.ctl + 1, run);
    c = __shfl_sync(FULL_MASK, c, 0);
    if (c >= a.g.n - a.base) break;
    const int mine = a.g.n - 1 - c - lane;
    const int nd = lane < run && mine >= a.base ? __ldg(a.in_deg + mine) : 0;
    const int e0 = nd ? __ldg(a.in_end + mine) - nd : 0;
    // a vertex with one lower neighbour closes nothing: its edge keeps the triangles above it
    if (nd == 1) s[1] += choose2(a.up[__ldg(&a.in[e0].y)]);
    unsigned todo = __ballot_sync(FULL_MASK, nd >= 2);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const int u = a.g.n - 1 - c - src;
      const int I = __shfl_sync(FULL_MASK, nd, src);
      const InEdge* L = a.in + __shfl_sync(FULL_MASK, e0, src);
      int W = 0;
      for (int i = lane; i < I && W <= SMALL_PATHS; i += 32) W += min(__ldg(a.ud + __ldg(&L[i].x)), SMALL_PATHS + 1);
      W = (int)__reduce_add_sync(FULL_MASK, (unsigned)min(W, SMALL_PATHS + 1));
      if (W > SMALL_PATHS) {
        if (lane == 0) a.list[atomicAdd(a.ctl, 1)] = u;
        continue;
      }
      const int bits = 33 - __clz(max(W, 16) - 1);  // 2^bits >= 2 W slots
      const unsigned mask = (1u << bits) - 1u;
      for (int i = lane; i <= (int)mask; i += 32) {
        key[i] = -1;
        cnt[i] = 0u;
      }
      __syncwarp();
      for (int i0 = 0; i0 < I; i0 += 32) {
        const PathBatch p = path_batch(a, L, i0, I);
        for (int f0 = 0; f0 < p.total; f0 += 32) {
          const int x = path_end(a, p, f0 + lane, u);
          if (x >= 0) {
            unsigned h = ((unsigned)x * 2654435761u) >> (32 - bits);
            while (true) {
              const int k = atomicCAS(key + h, -1, x);
              if (k == -1 || k == x) break;
              h = (h + 1) & mask;
            }
            s[0] += atomicAdd(cnt + h, 1u);
          }
        }
      }
      __syncwarp();
      unsigned long long two_t = 0ull;  // each triangle with u highest is met from both edges at u
      for (int i = lane; i < I; i += 32) {
        const InEdge w = __ldg(&L[i]);
        unsigned t = 0u;
        unsigned h = ((unsigned)w.x * 2654435761u) >> (32 - bits);
        for (int k = key[h]; k != -1; k = key[h]) {
          if (k == w.x) {
            t = cnt[h];
            break;
          }
          h = (h + 1) & mask;
        }
        two_t += t;
        s[1] += choose2((unsigned long long)t + a.up[w.y]);
      }
      two_t = warp_sum_u64(two_t);
      if (lane == 0) s[2] += (two_t >> 1) * (unsigned long long)(__ldg(a.ud + u) - 2);
      __syncwarp();
    }
  }
  add_sums(s, a.sums + CENSUS_C4);
}

// Vertices with more two-paths: a block each, direct counters over the ranks [base, u) in
// windows of `span` (one window unless the graph has more vertices than the counters fit). C:
// 16-bit counters packed in pairs when every degree is below 65,536, else 32-bit.
template <typename C>
__global__ void census_large_kernel(const __grid_constant__ CensusArgs a, int span) {
  extern __shared__ __align__(16) unsigned cw[];
  __shared__ int s_item, s_batch;
  __shared__ unsigned long long s_two;
  const int lane = lane_id();
  const int n_list = *reinterpret_cast<volatile int*>(a.ctl);
  const int warps = blockDim.x >> 5;
  unsigned long long s[3] = {0ull, 0ull, 0ull};
  while (true) {
    if (threadIdx.x == 0) s_item = atomicAdd(a.ctl + 2, 1);
    __syncthreads();
    const int item = s_item;
    __syncthreads();  // everyone has read it before thread 0 takes the next
    if (item >= n_list) break;
    const int u = a.list[item];
    const int I = __ldg(a.in_deg + u);
    const InEdge* L = a.in + (__ldg(a.in_end + u) - I);
    if (threadIdx.x == 0) s_two = 0ull;  // (thread 0 itself read the last vertex's)
    for (int lo = a.base; lo < u; lo += span) {
      const int hi = min(u, lo + span);
      const int words = (int)(((size_t)(hi - lo) * sizeof(C) + 15) / 16);
      for (int i = threadIdx.x; i < words; i += blockDim.x) reinterpret_cast<uint4*>(cw)[i] = make_uint4(0u, 0u, 0u, 0u);
      if (threadIdx.x == 0) s_batch = 0;
      __syncthreads();
      // a warp takes `take` in-neighbours at a time: a vertex with few of them still occupies every
      // warp of the block, and with many the warps that met long rows take fewer
      const int take = max(1, min(32, I / (4 * warps)));
      while (true) {
        int i0 = 0;
        if (lane == 0) i0 = atomicAdd(&s_batch, take);
        i0 = __shfl_sync(FULL_MASK, i0, 0);
        if (i0 >= I) break;
        const PathBatch p = path_batch(a, L, i0, min(I, i0 + take));
        for (int f0 = 0; f0 < p.total; f0 += 128) {
          int x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) x[q] = path_end(a, p, f0 + 32 * q + lane, u);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (x[q] >= lo && x[q] < hi) {
              const int y = x[q] - lo;
              if constexpr (sizeof(C) == 2) {
                const unsigned sh = (y & 1) * 16;
                s[0] += (atomicAdd(cw + (y >> 1), 1u << sh) >> sh) & 0xffffu;
              } else {
                s[0] += atomicAdd(cw + y, 1u);
              }
            }
          }
        }
      }
      __syncthreads();
      const C* c = reinterpret_cast<const C*>(cw);
      unsigned long long two_t = 0ull;
      for (int i = threadIdx.x; i < I; i += blockDim.x) {
        const InEdge w = __ldg(&L[i]);
        // (an in-neighbour below `base` has no other neighbour: no triangle on its edge)
        if (w.x < lo || w.x >= hi) continue;
        const unsigned t = c[w.x - lo];
        two_t += t;
        s[1] += choose2((unsigned long long)t + a.up[w.y]);
      }
      two_t = warp_sum_u64(two_t);
      if (lane == 0 && two_t) atomicAdd(&s_two, two_t);
      __syncthreads();
    }
    if (threadIdx.x == 0) s[2] += (s_two >> 1) * (unsigned long long)(__ldg(a.ud + u) - 2);
  }
  add_sums(s, a.sums + CENSUS_C4);
  census_finish(a.sums, a.ctl, CENSUS_SUMS, a.out);
}

// ---------------- launcher ----------------

// Blocks of a launch: at most `full`, no more than dm_opts.threads allows.
static int census_grid(int64_t full, int block, const LaunchCtx& ctx) {
  if (ctx.threads > 0) full = std::min<int64_t>(full, (ctx.threads + block - 1) / block);
  return (int)std::max<int64_t>(1, full);
}

template <typename C>
static int launch_large(const CensusArgs& a, LaunchCtx& ctx) {
  // the counters of one window, at most LARGE_SMEM; a block of 512 threads while four fit an SM,
  // else one of 1,024 (the same warps per SM with fewer counter arrays)
  constexpr size_t LARGE_SMEM = 200 * 1024;
  const int ranks = std::max(1, a.g.n - a.base);
  const int span = (int)std::min<size_t>((size_t)ranks, LARGE_SMEM / sizeof(C));
  const size_t smem = ((size_t)span * sizeof(C) + 15) / 16 * 16;
  const int block = smem <= 50 * 1024 ? 512 : 1024;
  auto kern = census_large_kernel<C>;
  DM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LARGE_SMEM + 16));
  int occ = 0;
  DM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, block, smem));
  if (occ < 1) return fail(DM_EINVAL, "census kernel does not fit on an SM");
  kern<<<census_grid(ctx.num_sms * occ, block, ctx), block, smem, ctx.stream>>>(a, span);
  ctx.launches++;
  DM_CUDA(cudaGetLastError());
  return DM_OK;
}

int census_flat(const void* blocks, uint64_t units, const int32_t* ud, int n, unsigned long long* sums,
                unsigned long long* out, LaunchCtx& ctx) {
  // about four 16-byte units or degrees per thread, at most two full waves of threads
  const int64_t want = std::max<int64_t>(((int64_t)units + 1023) / 1024, ud ? (n + 1023) / 1024 : 1);
  const int grid = census_grid(std::min<int64_t>(ctx.num_sms * 8, want), 256, ctx);
  census_flat_kernel<<<grid, 256, 0, ctx.stream>>>(reinterpret_cast<const uint4*>(blocks), units, ud, n, sums,
                                                   reinterpret_cast<int*>(sums + CENSUS_SUMS), out);
  ctx.launches++;
  DM_CUDA(cudaGetLastError());
  return DM_OK;
}

int census_launch(const CensusLaunch& L, LaunchCtx& ctx) {
  CensusArgs a;
  a.g = L.g;
  a.ud = L.ud;
  a.blocks = reinterpret_cast<const uint4*>(L.blocks);
  a.boff = L.boff;
  a.in_end = L.in_end;
  a.in_deg = L.in_deg;
  a.in = reinterpret_cast<const InEdge*>(L.in);
  a.up = L.up;
  a.sums = L.sums;
  a.ctl = reinterpret_cast<int*>(L.sums + CENSUS_SUMS);
  a.out = L.out;
  a.list = L.list;
  a.order = L.order;
  a.n_wide = L.n_wide;
  a.base = L.base;
  const int grid = census_grid(std::min<int64_t>(ctx.num_sms * 8, ((int64_t)a.g.n * 8 + 255) / 256), 256, ctx);
  census_rows_kernel<<<grid, 256, 0, ctx.stream>>>(a);
  ctx.launches++;
  DM_CUDA(cudaGetLastError());
  DM_CUDA(cudaFuncSetAttribute(census_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALL_SMEM));
  const int small = census_grid(std::min(ctx.num_sms * 3, (a.g.n - a.base + SMALL_WARPS - 1) / SMALL_WARPS),
                                32 * SMALL_WARPS, ctx);
  census_small_kernel<<<small, 32 * SMALL_WARPS, SMALL_SMEM, ctx.stream>>>(a);
  ctx.launches++;
  DM_CUDA(cudaGetLastError());
  return L.wide_counters ? launch_large<unsigned>(a, ctx) : launch_large<unsigned short>(a, ctx);
}

// Class counts of the census (indices of census_class).
void census_classes(int k, const uint64_t* s, uint64_t* c) {
  if (k == 3) {
    c[0] = s[FLAT_WEDGE] - 3 * s[FLAT_TRI];
    c[1] = s[FLAT_TRI];
    return;
  }
  const uint64_t T = s[CENSUS_TRI];
  const uint64_t k4 = s[CENSUS_K4];
  const uint64_t dia = s[CENSUS_DIA] - 6 * k4;
  const uint64_t cyc = s[CENSUS_C4] - dia - 3 * k4;
  const uint64_t paw = s[CENSUS_PAW] + s[CENSUS_PAW_TOP] - 4 * dia - 12 * k4;
  const uint64_t path = s[CENSUS_EDGE] - 3 * T - 2 * paw - 4 * cyc - 6 * dia - 12 * k4;
  c[0] = path;
  c[1] = s[CENSUS_STAR] - paw - 2 * dia - 4 * k4;
  c[2] = paw;
  c[3] = cyc;
  c[4] = dia;
  c[5] = k4;
}

// The dictionary's class of each connected type (k = 3: wedge, triangle; k = 4: path, star, paw,
// cycle, diamond, clique), from the edge count and largest degree of every connected quick code.
// False when the table gives codes of one type different classes (a hand-made file): only the
// enumeration, which looks up the code of each subgraph as it meets it, reproduces that.
bool census_class(const dm_dictionary* d, int32_t* cls) {
  const int k = d->k, types = k == 3 ? 2 : 6;
  for (int t = 0; t < types; ++t) cls[t] = -1;
  for (int64_t q = 0; q < d->n_quicks; ++q) {
    int deg[4] = {1, 1, 0, 0};
    int edges = 1;
    for (int p = 2; p < k; ++p)
      for (int j = 0; j < p; ++j)
        if ((q >> ((p - 2) * (p + 1) / 2 + j)) & 1) {
          ++deg[p];
          ++deg[j];
          ++edges;
        }
    int lo = deg[0], hi = deg[0];
    for (int p = 1; p < k; ++p) {
      lo = std::min(lo, deg[p]);
      hi = std::max(hi, deg[p]);
    }
    if (lo == 0 || edges < k - 1) continue;  // not connected
    int t;
    if (k == 3) t = edges - 2;
    else if (edges == 3) t = hi == 3 ? 1 : 0;
    else if (edges == 4) t = hi == 3 ? 2 : 3;
    else t = edges - 1;
    if (cls[t] < 0) cls[t] = d->quick_to_class[q];
    else if (cls[t] != d->quick_to_class[q]) return false;
  }
  return true;
}

}  // namespace dmb
