// Host-side state shared by the grid and probabilistic-map entry points.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <string>

#include "bonxai_gb300.h"
#include "bxg_device.cuh"
#include "bxg_mark.cuh"

namespace bxg {

// A growable device buffer.
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  // Test hook (bxg_debug_alloc_limit): this host thread's larger requests fail as they do on
  // a device without memory.
  static inline thread_local size_t limit = SIZE_MAX;
  static cudaError_t alloc(void** q, size_t bytes) {
    *q = nullptr;
    return bytes <= limit ? cudaMalloc(q, bytes) : cudaErrorMemoryAllocation;
  }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    size_t want = cap ? cap : 4096;
    while (want < bytes) want *= 2;
    return ensure_exact(want);
  }
  // Like ensure, but not rounded up.
  cudaError_t ensure_exact(size_t bytes) {
    if (bytes <= cap) return cudaSuccess;
    release();
    const cudaError_t e = alloc(&p, bytes);
    if (e == cudaSuccess) cap = bytes;
    return e;
  }
  // Like ensure, but keeps the first `keep` bytes of the old content.
  cudaError_t ensure_keep(size_t bytes, size_t keep, cudaStream_t s) {
    if (bytes <= cap) return cudaSuccess;
    size_t want = cap ? cap : 4096;
    while (want < bytes) want *= 2;
    void* np = nullptr;
    cudaError_t e = alloc(&np, want);
    if (e != cudaSuccess) return e;
    if (p && keep) {
      e = cudaMemcpyAsync(np, p, keep < cap ? keep : cap, cudaMemcpyDeviceToDevice, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) {
        cudaFree(np);
        return e;
      }
    }
    if (p) cudaFree(p);
    p = np;
    cap = want;
    return cudaSuccess;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
  DevBuf() = default;
  DevBuf(const DevBuf&) = default;
  DevBuf& operator=(const DevBuf&) = default;
  ~DevBuf() { release(); }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// One map: pools, counters, stream, scratch and error text.
struct MapCore {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  uint32_t flags = 0;
  double res = 0, inv_res = 0;
  DMap dm{};
  size_t budget = 0;
  size_t init_inners = 0, init_leaves = 0;  // pool sizes at creation
  float load_factor = 0.5f;
  uint32_t rays_per_warp = 0, block_size = 0, ray_unroll = 0;
  // bumped whenever leaf slots may be released (clear, releaseUnusedMemory):
  // caches of coordinate -> slot built before are stale after it
  uint64_t leaf_gen = 0;
  // ray kernel launch shape: block size and one resident wave of blocks
  int ray_wave_bs[2] = {0, 0};
  uint32_t ray_wave_blocks[2] = {0, 0};

  // pools
  DevBuf buckets, ichild, imask, lmask, ldata, lkey, lfree, ctr;
  uint32_t* h_ctr = nullptr;  // pinned mirror of ctr

  // scratch
  DevBuf s_in, s_in2, s_out, s_out2, s_dedup, s_dedup2, s_ep, s_cast, s_tmp;
  // 16-byte units of s_dedup known to be empty, from 0 (the ray phase clears
  // the table the last endpoint phase used, so the next one needs no memset)
  uint32_t dedup_clean = 0;
  uint32_t dedup_used = 0;  // 16-byte units that the last endpoint phase used
  DevBuf s_dir;             // leaf directory of the ray kernel (bxg_scan.cuh)

  std::string err;
  uint64_t launches = 0;
  int sm_count = 0;

  ~MapCore();
};

// Pointer kind: the ordinal of the GPU whose memory p is in, kPtrManaged for
// managed memory (usable in place on any device), kPtrHost otherwise.
constexpr int kPtrHost = -1;
constexpr int kPtrManaged = -2;
int ptr_device(const void* p);
bool is_device_ptr(const void* p);

int set_error(MapCore* m, int status, const std::string& msg);
int cuda_fail(MapCore* m, cudaError_t e, const char* what);

// Lifecycle and pools (bxg_core.cu).
int core_init(MapCore* m, double res, int ib, int lb, size_t esz, const bxg_config* cfg);
int core_clear(MapCore* m);
// clear(CLEAR_MEMORY) that also gives the node pools' memory back: the pools
// shrink to their sizes at creation (bonxai.hpp:678-684).
int core_release_pools(MapCore* m);
// Reads the counters back (synchronising the stream) and converts device error
// bits into a status; clears them and repairs overshooting allocation counters.
int core_sync(MapCore* m, uint32_t* err_bits_out = nullptr);
// Grows pools ahead of need (after a sync).
int core_maintain(MapCore* m);
// Grows what the error bits say ran out; returns BXG_OK if a retry may succeed.
int core_grow_for(MapCore* m, uint32_t err_bits);
size_t core_mem_usage(const MapCore* m);
int core_dump(MapCore* m, int32_t* out_xyz, void* out_values, size_t cap, size_t* n_out,
              int filter, int32_t thr);
int core_active_cells(MapCore* m, size_t* out);
int core_node_counts(MapCore* m, size_t* roots, size_t* leaves);

// Staging of caller arrays that may live on the host.
// Returns a device pointer holding `bytes` of `src` (copied if host memory).
int stage_in(MapCore* m, DevBuf& buf, const void* src, size_t bytes, const void** dev);
// Returns a device pointer to write `bytes` into; after the kernels call
// stage_out_finish to copy it to `dst` when dst is host memory.
int stage_out(MapCore* m, DevBuf& buf, void* dst, size_t bytes, void** dev);
int stage_out_finish(MapCore* m, void* dst, const void* dev, size_t bytes);

inline unsigned long long* stats_of(const MapCore* m) {
  return reinterpret_cast<unsigned long long*>(m->ctr.as<uint32_t>() + C_STATS);
}

#define BXG_CUDA(m, call)                                  \
  do {                                                     \
    cudaError_t e_ = (call);                               \
    if (e_ != cudaSuccess) return cuda_fail((m), e_, #call); \
  } while (0)

#define BXG_LAUNCHED(m)                                        \
  do {                                                         \
    (m)->launches++;                                           \
    cudaError_t e_ = cudaGetLastError();                       \
    if (e_ != cudaSuccess) return cuda_fail((m), e_, "launch"); \
  } while (0)

// Launches a kernel that begins with after_previous() (bxg_device.cuh): it is set up before
// the stream's previous kernel has ended and its caches are flushed (programmatic dependent
// launch). For the kernels that follow one another in a call: a scan of 2k points 91 ->
// 79 us, a room scan 104 -> 92, a depth frame 143 -> 140, LiDAR 130 -> 124, a grid batch of
// 300k points 57 -> 55. None of them lets
// the next one start while it runs (griddepcontrol.launch_dependents): the waiting blocks
// take slots of blocks that work (LiDAR 135 us, room 119). In the batched tick, whose
// kernels are nodes of a graph, it changes nothing (8 maps: 222 us, 221).
template <class... P, class... A>
void launch_after(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t stream,
                  A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.stream = stream;
  c.attrs = &attr;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

// Shared kernels (bxg_core.cu).
void launch_dedup_clear(MapCore* m, uint4* tab, uint32_t cap);
// Inserts the non-empty buckets of old_b[0..old_cap) into the table of M.
void launch_rehash(MapCore* m, const uint4* old_b, uint32_t old_cap, const DMap& M);
// Runs a batch that creates topology, retrying once pools have grown.
template <class F>
int run_with_growth(MapCore* m, F&& body) {
  for (int attempt = 0; attempt < 12; attempt++) {
    int st = body();
    if (st) return st;
    uint32_t err = 0;
    st = core_sync(m, &err);
    if (st == BXG_OK) return core_maintain(m);
    if (!(err & (ERR_POOL_INNER | ERR_POOL_LEAF | ERR_HASH_FULL)) ||
        (err & (ERR_WAIT | ERR_RAY_TOO_LONG | ERR_SCRATCH)))
      return st;
    const int g = core_grow_for(m, err);
    if (g) return g;
  }
  return set_error(m, BXG_ERR_OUT_OF_POOL, "pools could not grow enough");
}

// Entries of the endpoint dedup table of a scan of n points: a power of two, at least 2 n
// and up to 16 n in small scans. A thread probes with one CAS after the other, about 1 us
// each, and a small scan waits for the longest of the chains, while a large one has many
// points per cell and pays for clearing its table. With entries of 16 bytes (dedup_key: now
// 8 in most scans), endpoints at 2, 4, 8, 16 entries per
// point: 2k points 10.2, 6.2, 5.3, 4.9 us; 60k room 11.6, 8.9, 8.3, 7.7 us with 17.4, 17.3,
// 17.6, 19.6 us for k_mark, which clears it; 131k LiDAR 9.1, 7.6, 7.2, 7.2 with 24.9, 25.9,
// 26.3, 27.6; 64 maps of 10-500 k points 264, 250, 248, 245 us with 55, 110, 219, 440 us to
// clear. At 8.0 and 8.4, 65 and 66, 130 and 133 k points, the two sides of each line, the
// kernels of a LiDAR, room or depth scan take about 5 % longer at most with the factor used than
// with the best of 2, 4, 8, 16 (with 2 everywhere 16 %). The grid batches' tables are sized by
// the same rule. From 2^30 points it is 2^31
// entries, more than there are points in the largest batch (2^31 - 2).
inline uint32_t dedup_entries(uint64_t n) {
  const uint64_t per = n <= (1u << 13) ? 16 : n <= (1u << 16) ? 8 : n <= (1u << 17) ? 4 : 2;
  uint32_t p = 64;
  while (p < per * n && p < (1u << 31)) p <<= 1;
  return p;
}

// Text of the last failed create call on this host thread.
void set_create_error(const std::string& msg);
const MapCore* core_of_handle(const void* handle);

}  // namespace bxg

// A ProbabilisticMap handle: a map core plus the scan state of
// probabilistic_map.hpp:127-134.
struct bxg_pmap_s {
  bxg::MapCore core;
  bxg_pmap_options opt{};
  int update_count = 1;      // _update_count (probabilistic_map.hpp:129)
  uint64_t cast_ub = 0;      // upper bound of queued rays on the device
  uint64_t last_stats[8] = {0};
  float last_times[4] = {0};
  float last_query_ms = 0;       // device time of the last lookup kernel (BXG_FLAG_TIMING)
  uint32_t last_new_leaves = 0;  // leaves created by the last scan (pool headroom)
  double dir_reach = 0;          // cells of the coming ray phase lie within this range
  // the leaf directory kept across scans: its cube (leaf coordinates of the
  // corner, side), epoch (1..15) and the leaf generation it was built at
  int dir_x0 = 0, dir_y0 = 0, dir_z0 = 0;
  uint32_t dir_side = 0;
  uint32_t dir_epoch = 0;
  uint64_t dir_gen = 0;
  bool dir_live = false;
  // the ray phase's cube bitmap (bxg_mark.cuh): all zero between scans, sized for
  // cube_blocks leaf blocks; root bits of the marked cells; and, of the per-map
  // path, the rays' segments and the rays that leave the cube
  bxg::DevBuf cube_bits;
  size_t cube_blocks = 0;
  bxg::DevBuf cube_roots, ray_segs, ray_tails;
  // the cube that the winners of the ray list knew (no bits: none, the list holds rays of
  // addHitPoint/addMissPoint batches), whose segments are in ray_segs and long rays in
  // ray_tails; and the origin cell that it and dir_reach are of
  bxg::ScanCube list_cube{};
  int list_origin[3] = {0, 0, 0};
  cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  ~bxg_pmap_s() {
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
  }
};

namespace bxg {
// The cube of a scan's ray phase from origin cell (ox, oy, oz) whose rays end
// within `reach` (world units) of the origin; with `reach` infinite or above the
// size limit, Q->open is set and the cube holds the rays' first Q->kin
// cells. *ok = false when the scan cannot use one (other node sizes, non-finite
// points kept, single pass asked for, no memory for it) or is faster without. rays: room for their
// segments (0: none). Buffers grow here (cudaMalloc, zeroed).
int scan_cube(bxg_pmap_s* pm, int ox, int oy, int oz, double reach, uint64_t rays, ScanCube* Q,
              bool* ok);
// The bitmap of an open cube, 147 MB, is memory that such a scan can do without (its rays are
// walked on the tree then). It counts against the map's budget, behind the pools: it is
// made, and held, while both fit.
constexpr size_t kOpenCubeBlocks =
    size_t(4 * (2 * kOpenCubeHalf + 1)) * (4 * (2 * kOpenCubeHalf + 1)) * (4 * (2 * kOpenCubeHalf + 1));
constexpr size_t kOpenCubeBytes = kOpenCubeBlocks * 64;
// A scan of this reach takes an open cube.
bool open_reach(const MapCore* m, double reach);
// Bytes of an open cube's bitmap that the map holds.
size_t open_cube_held(const bxg_pmap_s* pm);
void drop_open_cube(bxg_pmap_s* pm);
// Sets up the ray walk's leaf directory of a scan (bxg_pmap.cu).
int leaf_dir_for_scan(bxg_pmap_s* pm, int ox, int oy, int oz, LeafDir* D, size_t max_words);
// Completes a scan whose endpoints were listed (and possibly applied) by a
// batched tick but whose map ran out of pool: grows the pools and re-runs the
// idempotent endpoint completion and ray phases on the map's own stream.
int pmap_complete_scan(bxg_pmap_s* pm, const int4* d_cast, const uint32_t* d_count,
                       uint32_t cap, int ox, int oy, int oz, int32_t u);
// bxg_batch_insert_f32, with the points of scan s either at xyz + 3 offsets[s] or, with
// parts, in host memory at parts[s]. New bitmaps of open cubes take at most cube_room bytes.
int batch_insert(bxg_batch b, const bxg_pmap* maps, size_t n_scans, const float* xyz,
                 const float* const* parts, const uint64_t* offsets, const float* origins,
                 const double* max_ranges, uint64_t* ray_cells, size_t cube_room);
// Grows the map's pools so that the next scan has at least `leaves` free leaf
// slots and the root hash stays under its load factor.
int core_reserve(MapCore* m, size_t leaves, size_t inners);
}  // namespace bxg
