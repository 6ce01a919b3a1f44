// Motif counting kernel for sm_100a: connected induced k-vertex subgraphs (k = 3..7) per
// canonical class, one persistent launch over all roots. The enumeration itself (semantics,
// extension sets, bulk leaf counting, virtual warps, donation) is motif_run_task in
// motif.cuh; this file holds the single-graph kernel and its launcher.
#include <algorithm>
#include <climits>
#include <string>

#include "motif.cuh"

namespace dmb {

constexpr int MOTIF_WARPS = 8;

struct MotifArgs {
  MotifCtx c;                  // graph, LB, dictionary, arena layout
  const int32_t* roots;
  int n_roots;
  int n_classes;
  unsigned long long* hist;    // n_classes
  int2* arena;                 // per warp: 32/W group arenas of c.arena_stride int2
  uint32_t* bits;              // per warp: 32/W groups x motif_bit_stride(k) bitmaps of c.bit_words (k >= 4)
  const int32_t* parts;        // optional per-root-entry part word (p | P << 16)
  int hist_smem;               // block-level class counters in shared memory (else straight to hist)
  int bits_smem;               // the bitmaps live in shared memory (zeroed at launch), not in `bits`
};

// Shared-memory budget of one block's vertex bitmaps (for 32 lanes, graphs of up to 13,800 vertices for
// k <= 5, 9,200 above); larger graphs keep them in global memory. Three blocks per SM fit beside them for
// k = 5 with 32 lanes; k = 6 from 50 KB of bitmaps on, k = 7 and narrower groups (whose state takes 28
// to 95 KB of a block) run with two, which is still faster than bitmaps in global memory: k = 7,
// random graph of 8,000 / 10,000, 32 lanes 1.61 ms with two blocks, 1.80 with three and global ones;
// k = 6, 9,000 / 16,000 1.18 and 1.24; k = 6, 2,000 / 6,000, 8 lanes 4.98 and 5.86.
constexpr size_t MOTIF_SMEM_BITS_MAX = 54 * 1024;

// Blocks per SM the registers are sized for: three for k >= 5 (80 registers; with four, 64 registers
// and 120 bytes of spills per thread, k = 5 took 3.79 ms instead of 3.53 on a Chung-Lu graph of 3,000
// vertices and 0.72 instead of 0.58 on a random graph of 2,000, k = 6 there 4.24 instead of 4.19),
// four for k = 4, whose shorter chains want the warps (5.5 ms, 5.8 with three, on a Chung-Lu
// graph of 18,700 vertices).
__host__ __device__ constexpr int motif_min_blocks(int K) { return K >= 5 ? 3 : 4; }

template <int K, int W>
__global__ void __launch_bounds__(32 * MOTIF_WARPS, motif_min_blocks(K)) motif_kernel(const __grid_constant__ MotifArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* bhist = reinterpret_cast<unsigned long long*>(smem);
  const int n_bhist = a.hist_smem ? a.n_classes : 0;
  unsigned char* wbase = smem + sizeof(unsigned long long) * ((n_bhist + 1) & ~1);
  const int lane = lane_id();
  const int wib = warp_in_block();
  MotifShared* ws = reinterpret_cast<MotifShared*>(wbase + motif_warp_smem<K, W>() * wib);
  const MotifCtx& c = a.c;
  const size_t warp_bit_words = (size_t)c.bit_words * motif_bit_stride(K) * (32 / W);
  uint32_t* sbits = reinterpret_cast<uint32_t*>(wbase + motif_warp_smem<K, W>() * MOTIF_WARPS);
  for (int cl = threadIdx.x; cl < n_bhist; cl += blockDim.x) bhist[cl] = 0;
  motif_zero_sweeps<K, W>(ws);
  if (a.bits_smem)
    for (size_t i = threadIdx.x; i < warp_bit_words * MOTIF_WARPS; i += blockDim.x) sbits[i] = 0u;
  __syncthreads();
  const size_t gw = (size_t)blockIdx.x * MOTIF_WARPS + wib;
  const int total_warps = gridDim.x * MOTIF_WARPS;
  int2* warp_arena = a.arena + gw * (size_t)c.arena_stride * (32 / W);
  uint32_t* warp_bits = a.bits_smem ? sbits + wib * warp_bit_words
                                    : (a.bits ? a.bits + gw * warp_bit_words : nullptr);
  unsigned long long ntasks = 0, nodes = 0;
  while (true) {
    int first = 0, count = 0, b = 0, e = -1, ok = 0, level = 0;
    int path[QPATH];
    for (int j = 0; j < QPATH; ++j) path[j] = 0;
    bool donated = false;
    if (lane == 0) ok = lb_next(c.lb, a.n_roots, total_warps, first, count, b, e, donated, level, path) ? 1 : 0;
    ok = __shfl_sync(FULL_MASK, ok, 0);
    if (!ok) break;
    first = __shfl_sync(FULL_MASK, first, 0);
    count = __shfl_sync(FULL_MASK, count, 0);
    b = __shfl_sync(FULL_MASK, b, 0);
    e = __shfl_sync(FULL_MASK, e, 0);
    level = __shfl_sync(FULL_MASK, level, 0);
    for (int j = 0; j < K - 3 && j < QPATH; ++j) path[j] = __shfl_sync(FULL_MASK, path[j], 0);
    donated = __shfl_sync(FULL_MASK, donated ? 1 : 0, 0) != 0;
    // a donated DFS prefix names a level that this k has
    if (level < 0 || level > K - 3) {
      if (lane == 0) {
        set_err(c.lb.ctr, ERR_BAD_TASK);
        lb_done(c.lb, count);
      }
      break;
    }
    for (int ti = 0; ti < count; ++ti) {
      const int v0 = donated ? first : __ldg(a.roots + first + ti);
      int bb = b, ee = e;
      if (!donated && a.parts) part_bounds(__ldg(a.parts + first + ti), bb, ee);
      ++ntasks;
      // block-level class counters, added to the global ones at exit
      motif_run_task<K, W>(c, ClassHist{a.hist_smem ? reinterpret_cast<unsigned*>(bhist) : nullptr, a.hist}, ws, warp_arena, warp_bits, v0, bb, ee, level, path, nodes);
    }
    if (lane == 0) lb_done(c.lb, count);
  }
  // every lane of a group counted the group's nodes: keep the leaders' counts
  nodes = warp_sum_u64((lane & (W - 1)) == 0 ? nodes : 0ull);
  if (lane == 0) {
    atomicAdd(&c.lb.ctr->tasks, ntasks);
    atomicAdd(&c.lb.ctr->nodes, nodes);
  }
  __syncthreads();
  for (int cl = threadIdx.x; cl < n_bhist; cl += blockDim.x)
    if (bhist[cl]) atomicAdd(a.hist + cl, bhist[cl]);
}

size_t motif_warp_bit_words(int k, int bit_words, int vwarp) {
  const int w = (vwarp == 8 || vwarp == 16) ? vwarp : 32;
  return k < 4 ? 0 : (size_t)bit_words * motif_bit_stride(k) * (size_t)(32 / w);
}

size_t motif_arena_stride(int k, int maxdeg, int vwarp) {
  const int w = (vwarp == 8 || vwarp == 16) ? vwarp : 32;
  return motif_group_stride(k, maxdeg) * (size_t)(32 / w);
}

// Launch shape of one kernel: blocks that the device holds at once (within dm_opts.threads), dynamic shared
// memory, and whether the bitmaps and the block's class counters are part of it (a table of any number of
// classes is counted: one that leaves no room for the warps' state adds to global memory).
struct MotifShape {
  int grid = 0;
  size_t smem = 0;
  bool bits_smem = false;
  bool hist_smem = true;
};

template <int K, int W>
static int motif_shape(int n_classes, int bit_words, const LaunchCtx& ctx, MotifShape* s) {
  const int block = 32 * MOTIF_WARPS;
  const size_t bits_bytes = (size_t)bit_words * motif_bit_stride(K) * (32 / W) * sizeof(uint32_t) * MOTIF_WARPS;
  constexpr size_t SMEM_MAX = 227 * 1024, state = motif_warp_smem<K, W>() * MOTIF_WARPS;
  const size_t hist = sizeof(unsigned long long) * (((size_t)n_classes + 1) & ~(size_t)1);
  s->hist_smem = hist + state <= SMEM_MAX;
  s->smem = (s->hist_smem ? hist : 0) + state;
  s->bits_smem = K >= 4 && bits_bytes <= MOTIF_SMEM_BITS_MAX && s->smem + bits_bytes <= SMEM_MAX;
  if (s->bits_smem) s->smem += bits_bytes;
  static LaunchCache cache;
  int occ = 0;
  DM_CUDA(cached_occupancy(cache, motif_kernel<K, W>, ctx.device, block, s->smem, &occ));
  if (occ < 1) return fail(DM_EINVAL, "motif kernel does not fit on an SM");
  s->grid = ctx.num_sms * occ;
  if (ctx.threads > 0) s->grid = std::max(1, std::min(s->grid, (ctx.threads + block - 1) / block));
  return DM_OK;
}

template <int K, int W>
static int launch_motif(MotifArgs a, LaunchCtx& ctx, int* grid_out) {
  MotifShape s;
  int rc = motif_shape<K, W>(a.n_classes, a.c.bit_words, ctx, &s);
  if (rc) return rc;
  a.bits_smem = s.bits_smem ? 1 : 0;
  a.hist_smem = s.hist_smem ? 1 : 0;
  int grid = s.grid;
  if (grid * MOTIF_WARPS > ctx.arena_warps) grid = std::max(1, ctx.arena_warps / MOTIF_WARPS);
  const int warps = grid * MOTIF_WARPS;
  a.c.lb.hungry_trigger = ctx.threshold >= 100 ? 0 : std::max(1, (ctx.threshold * warps + 99) / 100);
  motif_kernel<K, W><<<grid, 32 * MOTIF_WARPS, s.smem, ctx.stream>>>(a);
  ctx.launches++;
  *grid_out = grid;
  DM_CUDA(cudaGetLastError());
  return DM_OK;
}

template <int K>
static int warps_motif(int vwarp, int n_classes, int bit_words, const LaunchCtx& ctx, int* warps, size_t* warp_bits) {
  MotifShape s;
  const int rc = vwarp == 8    ? motif_shape<K, 8>(n_classes, bit_words, ctx, &s)
                 : vwarp == 16 ? motif_shape<K, 16>(n_classes, bit_words, ctx, &s)
                               : motif_shape<K, 32>(n_classes, bit_words, ctx, &s);
  *warps = s.grid * MOTIF_WARPS;
  *warp_bits = s.bits_smem ? 0 : sizeof(uint32_t) * motif_warp_bit_words(K, bit_words, vwarp);
  return rc;
}

int motif_warps(int k, int vwarp, int n_classes, int bit_words, const LaunchCtx& ctx, int* warps, size_t* warp_bits) {
  switch (k) {
    case 3: return warps_motif<3>(vwarp, n_classes, bit_words, ctx, warps, warp_bits);
    case 4: return warps_motif<4>(vwarp, n_classes, bit_words, ctx, warps, warp_bits);
    case 5: return warps_motif<5>(vwarp, n_classes, bit_words, ctx, warps, warp_bits);
    case 6: return warps_motif<6>(vwarp, n_classes, bit_words, ctx, warps, warp_bits);
    case 7: return warps_motif<7>(vwarp, n_classes, bit_words, ctx, warps, warp_bits);
    default: return fail(DM_EINVAL, "motif k must be in [3, 7]");
  }
}

template <int K>
static int launch_motif_w(const MotifArgs& a, int vwarp, LaunchCtx& ctx, int* grid) {
  switch (vwarp) {
    case 8: return launch_motif<K, 8>(a, ctx, grid);
    case 16: return launch_motif<K, 16>(a, ctx, grid);
    default: return launch_motif<K, 32>(a, ctx, grid);
  }
}

int motif_launch(const MotifLaunch& L, LaunchCtx& ctx, int* grid) {
  MotifArgs a;
  a.c.g = L.g;
  a.c.lb = LBArgs{L.ctr, reinterpret_cast<QHeader*>(L.queue),
                  reinterpret_cast<QSlot*>(reinterpret_cast<char*>(L.queue) + sizeof(QHeader) * L.nq), L.qcap, 0,
                  L.max_donations, (long long)ctx.donate_after_us * 1000ll, (long long)ctx.timeout_ms * 1000000ll,
                  ctx.test_stall, 4, L.nq};
  a.c.q2c = L.q2c;
  a.c.sym = L.sym;
  a.c.maxdeg = L.maxdeg;
  a.c.arena_stride = (int)motif_group_stride(L.k, L.maxdeg);
  a.c.per_root = L.per_root;
  a.c.bit_base = 0;
  a.c.bit_words = L.bit_words;
  a.bits = L.bits;
  a.roots = L.roots;
  a.n_roots = L.n_roots;
  a.n_classes = L.n_classes;
  a.hist = L.hist;
  a.arena = reinterpret_cast<int2*>(L.arena);
  a.parts = L.parts;
  a.bits_smem = a.hist_smem = 0;
  const int w = (L.vwarp == 8 || L.vwarp == 16) ? L.vwarp : 32;
  switch (L.k) {
    case 3: return launch_motif_w<3>(a, w, ctx, grid);
    case 4: return launch_motif_w<4>(a, w, ctx, grid);
    case 5: return launch_motif_w<5>(a, w, ctx, grid);
    case 6: return launch_motif_w<6>(a, w, ctx, grid);
    case 7: return launch_motif_w<7>(a, w, ctx, grid);
    default: return fail(DM_EINVAL, "motif k must be in [3, 7]");
  }
}

}  // namespace dmb
