// Internal launch interfaces between the C ABI (engine.cu) and the kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>
#include <vector>

#include "dm_internal.hpp"

namespace dmb {

// Per-call device counters and load-balancer state. One instance lives in device memory
// for each call; the host initialises it (pending = number of root tasks). Words that
// busy and hungry warps hit concurrently sit on separate 128-byte lines.
struct alignas(128) DevCounters {
  int cursor;                    // root cursor
  int pad0[31];
  int pending;                   // roots + donated tasks not finished yet
  int pad1[31];
  int hungry;                    // warps waiting for work
  int pad2[31];
  unsigned long long progress;   // work finished (batched), watched by waiting warps
  unsigned long long pad3[15];
  int queued;                    // donated tasks in the queue
  int pad4[31];
  unsigned long long count;      // clique total
  unsigned long long nodes;      // DFS nodes expanded
  unsigned long long tasks;      // tasks executed (roots + donated ranges)
  unsigned long long donations;  // donated ranges
  unsigned long long idle_polls; // polls of the donation queue by hungry warps
  unsigned long long hungry_ns;  // time warps spent waiting for work, summed over warps
  unsigned long long max_task_ns;  // longest single task
  unsigned long long prefix_donations;  // donated DFS prefixes (a level >= 1 extension set)
  unsigned long long count_k[16];  // fused counts: cliques of every size up to k
  int max_task_root;             // its root (best effort under races)
  int test_gate;                 // never written by the library (failure-path tests)
  int err;                       // first error code raised by a kernel (0 = none)
  int blocks_done;               // self-clearing launches: blocks that have added their sums
};

constexpr int ERR_ARENA_OVERFLOW = 1;
constexpr int ERR_TIMEOUT = 2;
constexpr int ERR_BAD_TASK = 3;

// Status of a call whose kernel raised device error word `err` (non-zero): a bounded wait
// that gave up is DM_ETIMEOUT, an exceeded capacity bound DM_EOVERFLOW, and a task the
// kernel could not place (its own bookkeeping disagreeing with the graph) DM_EINTERNAL.
inline int kernel_status(int err) {
  return err == ERR_TIMEOUT ? DM_ETIMEOUT : (err == ERR_ARENA_OVERFLOW ? DM_EOVERFLOW : DM_EINTERNAL);
}

struct GraphView {
  const int32_t* row;   // padded row starts
  const int32_t* deg;
  const int32_t* adj;
  int32_t n;
};

struct LaunchCtx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 148;
  int launches = 0;
  int timeout_ms = 30000;
  int threads = 0;       // requested total threads (reference argv[3]); 0 = persistent default
  int block = 0;         // requested block size (reference argv[4]); 0 = kernel default
  int vwarp = 0;
  int threshold = 0;     // donation trigger (hungry-warp percentage); >= 100 = off
  int donations_per_warp = 16;
  int arena_warps = 0;   // warps the list arena has room for
  int donate_after_us = 20;  // a task donates only after running this long
  int test_stall = 0;        // DM_TEST_STALL_AT_EXIT
};

// Clique index (clique_cached.cuh): the local adjacency bitmap of every root r of the DAG
// with 2 <= d = |N+(r)| <= 256, as d rows of ceil(d/64) u64 words, the block starting on a
// 16-byte boundary (offset in 16-byte units; INDEX_NONE for roots without a block).
constexpr uint32_t INDEX_NONE = 0xffffffffu;
constexpr int INDEX_MAX_DEGREE = 256;
constexpr int INDEX_MAX_K = 8;  // larger k rebuild the bitmaps per launch

inline uint32_t index_block_units_host(int d) {
  const int nw = (d + 63) >> 6;
  return (uint32_t)((d * nw + 1) >> 1);
}

// One entry of a counting launch's task list on the index: root (rank space), out-degree,
// block offset (16-byte units, or INDEX_NONE) and scheduler part word (p | P << 16, 0 = whole).
struct RootDesc {
  int32_t root;
  int32_t d;
  uint32_t off;
  int32_t part;
};

// Scheduler part words: p | P << 16 (part p of P; 0 = the whole root), plus PART_EAGER when
// the learned scheduler predicts the task to be heavy, so that it donates without waiting
// for the minimum task age.
constexpr int PART_EAGER = 1 << 30;

// The learned schedule on the device (predictor.cu): inputs, scratch and outputs.
struct SchedIO {
  const float* feat = nullptr;       // n x 6 base features by original id
  float* params = nullptr;           // MLP parameters on the device
  bool params_current = false;       // params already hold this predictor's version
  int* h_hdr = nullptr;              // pinned: the schedule's task count and error flag
  const int32_t* roots = nullptr;    // n_in input entries
  const int32_t* orig = nullptr;     // rank -> original id (cliques), else null
  int n_in = 0, k = 0, warps = 1, cap = 0;
  void* scratch = nullptr;           // learned_schedule_scratch_bytes(n_in)
  int32_t* out_roots = nullptr;      // cap
  int32_t* out_parts = nullptr;      // cap
  RootDesc* out_desc = nullptr;      // cap or null
  const int32_t* odeg = nullptr;     // rank-space out-degrees (out_desc)
  const uint32_t* boff = nullptr;    // index block offsets (out_desc), or null
};
int learned_schedule_device(const void* predictor, const SchedIO& io, LaunchCtx& ctx, int* n_out);
size_t learned_schedule_scratch_bytes(int n_in);
inline int learned_schedule_cap(int n_in, int warps) { return n_in + 4 * warps + 64; }
int predictor_num_params();

// Clique engine (clique.cu).
struct CliqueLaunch {
  GraphView g;                   // degree-ordered DAG in rank space
  int k = 0;
  const int32_t* roots = nullptr;  // ordered root ranks
  int n_roots = 0;
  DevCounters* ctr = nullptr;
  void* queue = nullptr;         // donation queue: nq headers + nq * qcap slots (lb.cuh)
  int qcap = 0;                  // slots per shard
  int nq = 1;                    // shards
  int max_donations = 16;        // per task
  int32_t* arena = nullptr;      // list path: (32 / list_vwarp) x k x arena_dcap ints per warp
  int arena_dcap = 0;
  int list_vwarp = 32;           // list path: lanes per group (8, 16 or 32)
  int list_threshold = 256;
  int nwmax = 1;
  unsigned long long* per_root = nullptr;
  const int32_t* parts = nullptr;   // per root entry: p | P << 16 (0 = whole root)
  // counting on the clique index (clique_cached_*), else the per-launch bitmap build
  const RootDesc* desc = nullptr;   // task list (n_roots entries)
  const void* blocks = nullptr;     // the index (16-byte units)
  const uint32_t* boff = nullptr;   // block offset per root
  DevCounters* out = nullptr;       // page-locked host copy of the counters, written by the kernel
  DevCounters* next = nullptr;      // the next launch's counters, zeroed by the kernel
  int static_chunk = 1;             // warp w starts with entries [w * static_chunk, +static_chunk)
  int n_static = 0;                 // entries dealt statically; the root cursor starts here
  bool tma = true;                  // stage blocks by bulk asynchronous copies (else 16-byte loads)
  bool multi = false;               // fused: count every clique size up to k (count_k)
};
int clique_launch(const CliqueLaunch& L, LaunchCtx& ctx, int* grid);
int clique_max_warps(int num_sms);
// Grid of the index-counting kernel for this launch (occupancy, requested threads, arena).
int clique_cached_grid(const CliqueLaunch& L, LaunchCtx& ctx, int* grid);
// Counting on the index with that grid (L.static_chunk / L.n_static set for it).
int clique_cached_launch(const CliqueLaunch& L, LaunchCtx& ctx, int grid);
// Builds the index blocks of roots[0..n) (rank space, 2 <= out-degree <= 64 * m).
int clique_index_build(const GraphView& g, const int32_t* roots, int n, void* blocks, const uint32_t* boff, int m,
                       LaunchCtx& ctx);

// Pattern-aware queries q4..q13 (near_clique.cu): (n-2)-cliques and their common neighbours.
struct NearLaunch {
  GraphView dag;                   // rank space
  const int32_t* in_end = nullptr; // in-lists (census_in_lists)
  const int32_t* in_deg = nullptr;
  const void* in = nullptr;
  const int32_t* roots = nullptr;  // by descending out-degree
  const void* steps = nullptr;     // NearStep[n_steps]
  int n_steps = 0;
  int n_items = 0;                 // out-edges of the roots
  int c = 2;                       // clique size n - 2
  DevCounters* ctr = nullptr;      // self-clearing
  DevCounters* out = nullptr;      // page-locked host copy, written by the kernel
  DevCounters* next = nullptr;     // the next launch's counters, zeroed by the kernel
  int32_t* arena = nullptr;        // arena_ints per warp, or null
  size_t arena_ints = 0;
  int list_cap = 0;
  int max_claim = 1;               // larger claims than the guided ones, up to these (<= 32)
  // q_4 by triangles (else null): a counter per padded DAG entry, the first pair of out-neighbours of
  // each run of the whole order (roots, steps), and the shard's roots (null: all). n_items then
  // is the number of root tasks.
  unsigned* tri = nullptr;
  size_t tri_words = 0;
  const long long* pair_step = nullptr;
  long long n_pairs = 0;
  const int32_t* shard = nullptr;
  int shard_roots = 0;
};
// A run of roots of equal out-degree: its first item (out-edge), first root, out-degree.
struct NearStep {
  int32_t item, root, deg, pad;
};
int near_clique_launch(const NearLaunch& L, LaunchCtx& ctx, int* grid);
size_t near_clique_rows(int d, int deg);  // arena ints (beyond the list) for a root's edges

// Whole-graph census of the connected 3- and 4-vertex classes (census.cu).
constexpr int CENSUS_SUMS = 8;
// sums and cursors of a call: zero at launch, and zeroed again by the call's last block
constexpr size_t CENSUS_BYTES = (CENSUS_SUMS + 2) * sizeof(unsigned long long);
// k = 3, and triangles alone (ud null): sums 0 (triangles) and 1 (wedges) into out, page-locked
// host memory, from the clique index of `units` 16-byte units and the degrees.
int census_flat(const void* blocks, uint64_t units, const int32_t* ud, int n, unsigned long long* sums,
                unsigned long long* out, LaunchCtx& ctx);
struct CensusLaunch {              // k = 4
  GraphView g;                     // degree-ordered DAG in rank space
  const void* blocks = nullptr;    // clique index: a block for every root with 2 or more out-neighbours
  const uint32_t* boff = nullptr;
  const int32_t* ud = nullptr;     // undirected degree by rank
  const int32_t* order = nullptr;  // ranks by descending out-degree; n_wide of them with 32 or more
  int n_wide = 0;
  int base = 0;                    // ranks below it have degree 0 or 1
  bool wide_counters = false;      // a degree of 65,536 or more: 32-bit path counters
  // in-lists (census_in_lists), edge array (one word per padded DAG entry) and vertex list
  const int32_t* in_end = nullptr;
  const int32_t* in_deg = nullptr;
  const void* in = nullptr;
  uint32_t* up = nullptr;
  int* list = nullptr;
  unsigned long long* sums = nullptr;  // CENSUS_BYTES
  unsigned long long* out = nullptr;   // page-locked host memory: CENSUS_SUMS
};
int census_launch(const CensusLaunch& L, LaunchCtx& ctx);
// In-lists of the DAG: n end offsets, n lengths, 8 bytes per edge, and one scratch int.
int census_in_lists(const GraphView& g, int32_t* in_end, int32_t* in_deg, void* in, int* pool, LaunchCtx& ctx);
// Class of each connected type in the dictionary (false: the table is not constant on a type),
// and the types' counts from the sums.
bool census_class(const dm_dictionary* d, int32_t* cls);
void census_classes(int k, const uint64_t* sums, uint64_t* counts);

// Motif engine (motif.cu).
struct MotifLaunch {
  GraphView g;                   // undirected CSR, original ids
  int k = 0;
  const int32_t* roots = nullptr;
  int n_roots = 0;
  DevCounters* ctr = nullptr;
  void* queue = nullptr;
  int qcap = 0;
  int nq = 1;
  int max_donations = 16;
  const int32_t* q2c = nullptr;
  int sym = 0;                   // dm_dictionary::sym
  int n_classes = 0;
  unsigned long long* hist = nullptr;
  void* arena = nullptr;
  int maxdeg = 0;
  unsigned long long* per_root = nullptr;
  const int32_t* parts = nullptr;
  int vwarp = 32;                // virtual-warp width: 8, 16 or 32
  uint32_t* bits = nullptr;      // k >= 4, per warp: motif_warp_bit_words zeroed words
  int bit_words = 0;
};
// 32-bit words of one membership bitmap over n vertices.
inline int motif_bit_words(int n) { return (n + 31) / 32 + 1; }
int motif_launch(const MotifLaunch& L, LaunchCtx& ctx, int* grid);
size_t motif_warp_bit_words(int k, int bit_words, int vwarp);  // words of vertex bitmaps per warp
// Warps that a launch keeps on the device at once, and the bytes of bitmaps each needs in global memory.
int motif_warps(int k, int vwarp, int n_classes, int bit_words, const LaunchCtx& ctx, int* warps, size_t* warp_bits);
size_t motif_arena_stride(int k, int maxdeg, int vwarp);  // int2 slots per warp

const char* cuda_err_str(cudaError_t e);

// Launch configuration of one kernel, settled once per device: the dynamic shared-memory
// attribute is set and the resident blocks per SM are queried on the first launch only, so
// a call spends no driver time on them afterwards.
constexpr int LAUNCH_CACHE_DEVICES = 64;
struct LaunchCache {
  int smem[LAUNCH_CACHE_DEVICES] = {};
  int occ[LAUNCH_CACHE_DEVICES] = {};
};
template <typename Kern>
inline cudaError_t cached_occupancy(LaunchCache& c, Kern kern, int device, int block, size_t smem, int* occ) {
  if (device >= 0 && device < LAUNCH_CACHE_DEVICES && c.occ[device] > 0 && c.smem[device] == (int)smem) {
    *occ = c.occ[device];
    return cudaSuccess;
  }
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, block, smem);
  if (e == cudaSuccess && device >= 0 && device < LAUNCH_CACHE_DEVICES) {
    c.smem[device] = (int)smem;
    c.occ[device] = *occ;
  }
  return e;
}

// Host helpers shared by the entry points (engine.cu).
int select_device(const dm_opts* o, LaunchCtx& ctx);   // device, stream and options -> ctx
int check_opts(const dm_opts* o);
// Device buffers from the library's per-device pool (current device; safe from any thread). A
// buffer is given back only once nothing on the device uses it any more.
cudaError_t gbuf_alloc(void** p, size_t bytes);
// cudaMalloc that releases the pooled buffers and tries again when the device has no room (no error is
// left behind), and the bytes such allocations can have: free ones and pooled ones.
cudaError_t device_alloc(void** p, size_t bytes);
cudaError_t device_room(size_t* bytes);
void gbuf_free(void* p, int dev);
// Transfers of pageable host memory through pooled page-locked buffers (engine.cu), on `st`.
struct Staging {
  void* buf[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};  // the last copy from or into the buffer
  cudaEvent_t beg[2] = {nullptr, nullptr}, end[2] = {nullptr, nullptr};  // its times, where it is timed
  bool busy[2] = {false, false};
  bool pinned = true;
};
class Stager {
 public:
  Stager(int device, cudaStream_t st);
  ~Stager();
  Stager(const Stager&) = delete;
  Stager& operator=(const Stager&) = delete;
  // The source may change as soon as the call returns; the destination is written in stream order.
  cudaError_t upload(void* dst, const void* src, size_t bytes);
  // fill(buf, n) writes up to n bytes and returns how many (fewer end the upload); *got: the total. These
  // copies are timed: copy_ms() is their device time, once the stream has been waited for.
  cudaError_t upload(void* dst, size_t bytes, const std::function<size_t(void*, size_t)>& fill, size_t* got);
  // The destination is complete when the call returns.
  cudaError_t download(void* dst, const void* src, size_t bytes);
  float copy_ms();

 private:
  cudaError_t wait(int i);
  cudaError_t sent(int i);
  int dev_;
  cudaStream_t st_;
  Staging s_;
  int next_ = 0;
  bool timed_[2] = {false, false};
  float ms_ = 0.f;
  cudaError_t err_ = cudaSuccess;
};
int queue_init_launch(void* queue, int nq, int cap, cudaStream_t st);  // empty donation queue
constexpr int QUEUE_SHARDS = 64;        // donation-queue shards of a workspace
constexpr int QUEUE_SHARD_SLOTS = 2048; // slots per shard

}  // namespace dmb

#define DM_CUDA(call)                                                              \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) {                                                       \
      cudaGetLastError(); /* (else the next call's launch check would find it) */  \
      return ::dmb::fail(DM_ECUDA, std::string(#call " failed: ") + cudaGetErrorString(e_)); \
    }                                                                              \
  } while (0)
