// ProbabilisticMap on the GPU: insertPointCloud / addHitPoint / addMissPoint /
// updateFreeCells / isOccupied / getOccupiedVoxels, bit-exact with
// bonxai_map/include/bonxai_map/probabilistic_map.hpp and
// bonxai_map/src/probabilistic_map.cpp.
//
// Why a scan parallelises without changing its result: see bxg_scan.cuh.
//
// Kernels per scan (all on the handle's stream):
//   k_endpoints   fp64 endpoint of each point, exactly as hpp:147-156 rounds
//                 it; lowest index per endpoint cell via a scratch hash table.
//   k_winners     the lowest-index point of each cell reads the pre-scan word;
//                 unless update_id == u it applies its hit/miss and appends
//                 {cell, hit/miss} to the ray list (and counts the ray length
//                 for the ray-cell total).
//   k_apply       only after a pool ran out: completes the listed endpoints.
//   k_mark        the ray phase's first part: every listed ray's cells set
//                 their bits in the scan's cube bitmap (bxg_mark.cuh).
//   k_apply_rays  per marked leaf, get-or-create the leaf and apply the miss
//                 update to its marked cells.
//   k_tail        only when rays may be longer than the cube (no range limit):
//                 walks the rest of those that are.
//   k_rays        the single-pass form of the ray phase, for rays queued by
//                 addHitPoint/addMissPoint batches and for maps that keep
//                 non-finite points or ask for it: a group of W lanes walks one
//                 ray, W consecutive cells per step, creating leaves on the way
//                 and applying the miss update.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "bxg_internal.h"
#include "bxg_mark.cuh"
#include "bxg_scan.cuh"

namespace bxg {

// Endpoint of each point; lowest index per endpoint cell in the scratch table.
// zero: bit 0 -- the scan's statistics start at zero; bit 1 -- the ray list
// starts empty (no rays queued by earlier addHitPoint/addMissPoint batches).
// Done by the first kernel of a scan instead of memsets.
// bit 2 -- the ray phase's root bits and segment count start at zero.
enum : int { ZERO_STATS = 1, ZERO_CAST = 2, ZERO_RAYS = 4 };
__device__ __forceinline__ void zero_scan_stats(const DMap& M, int zero,
                                                uint32_t* roots = nullptr,
                                                uint32_t root_words = 0) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < root_words;
       t += gridDim.x * blockDim.x)
    roots[t] = 0u;
  if (blockIdx.x != 0) return;
  if ((zero & ZERO_RAYS) && threadIdx.x == 33) M.ctr[C_SEGS] = M.ctr[C_TAILS] = 0u;
  if ((zero & ZERO_STATS) && threadIdx.x < S_COUNT)
    reinterpret_cast<unsigned long long*>(M.ctr + C_STATS)[threadIdx.x] = 0ull;
  if ((zero & ZERO_CAST) && threadIdx.x == 32) M.ctr[C_CAST] = 0u;
}

template <typename PT>
__global__ void k_endpoints(const __grid_constant__ DMap M, const uint8_t* __restrict__ pts, size_t stride, uint32_t n,
                            double fx, double fy, double fz, double max_range, double mr2,
                            double inv_res, int keep_nonfinite, int4* __restrict__ ep,
                            uint4* tab, uint32_t tmask, int zero_stats, EpFast F,
                            uint32_t* roots, uint32_t root_words, DedupKey K) {
  zero_scan_stats(M, zero_stats, roots, root_words);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  int4 e = make_int4(0, 0, 0, EP_SKIP);
  if (i < n) {
    const PT* p = reinterpret_cast<const PT*>(pts + size_t(i) * stride);
    e = compute_endpoint<PT>(p, fx, fy, fz, max_range, mr2, inv_res, keep_nonfinite != 0, &F);
  }
  endpoint_enter(M, e, i, tab, tmask, K);
  if (i < n) ep[i] = e;
}

// A sensor-frame cloud with its sensor-to-world transform (row-major 3x4),
// the ingest of bonxai_ros/src/bonxai_server.cpp:147-171 fused into the
// endpoint kernel: points with a non-finite coordinate are dropped (:147-154),
// the rest are transformed in float (:166-168), then handled as k_endpoints
// does. A dropped point keeps its index, so the lowest-index rule gives the
// same winners as the host's compaction. Transform order per axis, in float
// without contraction: ((m[r][0]*x + m[r][1]*y) + m[r][2]*z) + m[r][3].
struct Xf {
  float m[12];
};

__device__ __forceinline__ float xf_row(const Xf& t, int r, float x, float y, float z) {
  return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(t.m[4 * r], x), __fmul_rn(t.m[4 * r + 1], y)),
                             __fmul_rn(t.m[4 * r + 2], z)),
                   t.m[4 * r + 3]);
}

__global__ void k_endpoints_sensor(const __grid_constant__ DMap M, const uint8_t* __restrict__ pts, size_t stride,
                                   uint32_t n, Xf xf, double fx, double fy, double fz,
                                   double max_range, double mr2, double inv_res,
                                   int4* __restrict__ ep, uint4* tab, uint32_t tmask,
                                   int zero_stats, EpFast F, uint32_t* roots,
                                   uint32_t root_words, DedupKey K) {
  zero_scan_stats(M, zero_stats, roots, root_words);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* p = reinterpret_cast<const float*>(pts + size_t(i) * stride);
  const float x = p[0], y = p[1], z = p[2];
  if (!(isfinite(x) && isfinite(y) && isfinite(z))) {
    ep[i] = make_int4(0, 0, 0, EP_SKIP);
    return;
  }
  const float w[3] = {xf_row(xf, 0, x, y, z), xf_row(xf, 1, x, y, z), xf_row(xf, 2, x, y, z)};
  const int4 e = compute_endpoint<float>(w, fx, fy, fz, max_range, mr2, inv_res, true, &F);
  ep[i] = e;
  if (e.w != EP_SKIP) dedup_min_insert(tab, tmask, e.x, e.y, e.z, i, M, K);
}

// addHitPoint / addMissPoint batches: double points with a given kind, or a
// per-point kind (0 hit, 1 miss) when kinds != nullptr.
__global__ void k_endpoints_kind(const __grid_constant__ DMap M, const double* __restrict__ pts, uint32_t n, int kind,
                                 const uint8_t* __restrict__ kinds, double inv_res,
                                 int4* __restrict__ ep, uint4* tab, uint32_t tmask, int zero) {
  zero_scan_stats(M, zero);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (kinds) kind = kinds[i] ? EP_MISS : EP_HIT;
  const int cx = __double2int_rd(__dmul_rn(pts[3 * i + 0], inv_res));
  const int cy = __double2int_rd(__dmul_rn(pts[3 * i + 1], inv_res));
  const int cz = __double2int_rd(__dmul_rn(pts[3 * i + 2], inv_res));
  ep[i] = make_int4(cx, cy, cz, kind);
  dedup_min_insert(tab, tmask, cx, cy, cz, i, M, DedupKey{});
}

// The lowest-index point of each endpoint cell (winners_block).
__global__ void __launch_bounds__(256) k_winners(const __grid_constant__ DMap M, int4* ep, uint32_t n,
                          uint4* tab, uint32_t tmask, int ox, int oy, int oz, int32_t u, Opts o,
                          int4* cast, uint32_t cast_cap, const __grid_constant__ ScanCube Q) {
  __shared__ WinnersShared S;
  after_previous();
  winners_block(M, ep, n, blockIdx.x * blockDim.x + threadIdx.x, tab, tmask, ox, oy, oz, u, o,
                cast, cast_cap, Q, S);
}

// Completes listed endpoints after a pool ran out: creates each cell and
// applies its hit or miss (probabilistic_map.cpp:35-41,49-54). Idempotent --
// a cell already at u is left alone -- so it may run over the whole list.
__global__ void k_apply(const __grid_constant__ DMap M, const int4* __restrict__ cast, uint32_t cast_cap, int32_t u,
                        Opts o) {
  const uint32_t n = min(ld_volatile(M.ctr + C_CAST), cast_cap);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int4 e = cast[k];
    const uint32_t lf = leaf_of(M, e.x, e.y, e.z, true);
    if (lf == kNone) continue;
    const uint32_t ci = leaf_index(M, e.x, e.y, e.z);
    cell_mark_on(M, lf, ci);
    int32_t* cp = reinterpret_cast<int32_t*>(M.ldata) + size_t(lf) * M.lsize + ci;
    const int32_t w = *cp;
    if (cell_id(w) != u) {
      const int32_t p = cell_prob(w);
      const int32_t np = e.w == EP_HIT ? min(wrap_add(p, o.hit), o.cmax)
                                       : max(wrap_add(p, o.miss), o.cmin);
      *cp = cell_pack(np, u);
    }
  }
}

// Ray phase: one group of W lanes per listed ray (walk_ray, or walk_ray2 with
// two cells per lane per step when U == 2).
// Also clears tab[0, tab_n), the endpoint dedup table of the scan, so that
// the next scan's endpoint phase starts from an empty table without a memset.
template <int W, int U>
__global__ void __launch_bounds__(U == 2 ? 256 : 1024, U == 2 ? 3 : 1) k_rays(const __grid_constant__ DMap M, const int4* __restrict__ cast,
                                                 uint32_t cast_cap, int ox, int oy, int oz,
                                                 int32_t u, int32_t miss, int32_t cmin,
                                                 uint4* __restrict__ tab, uint32_t tab_n,
                                                 LeafDir D) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < tab_n; t += gridDim.x * blockDim.x)
    tab[t] = make_uint4(kNone, kNone, kNone, kNone);
  const uint32_t n_cast = min(ld_volatile(M.ctr + C_CAST), cast_cap);
  const unsigned lane = threadIdx.x & 31;
  const unsigned sl = lane & (W - 1);
  const unsigned gbase = lane & ~(W - 1);
  const unsigned gmask = (W == 32) ? 0xffffffffu : (((1u << W) - 1u) << gbase);
  const uint32_t gid = (blockIdx.x * blockDim.x + threadIdx.x) / W;
  const uint32_t ngroups = (gridDim.x * blockDim.x) / W;
  uint32_t visited = 0, updated = 0;
  for (uint32_t r = gid; r < n_cast; r += ngroups) {
    if (U == 2)
      walk_ray2<W>(M, cast[r], ox, oy, oz, u, miss, cmin, sl, gbase, gmask, visited, updated);
    else
      walk_ray<W, true>(M, cast[r], ox, oy, oz, u, miss, cmin, sl, gbase, gmask, visited,
                        updated, D.words ? &D : nullptr);
  }
  visited = __reduce_add_sync(0xffffffffu, visited);
  updated = __reduce_add_sync(0xffffffffu, updated);
  if (lane == 0 && visited) {
    unsigned long long* st = reinterpret_cast<unsigned long long*>(M.ctr + C_STATS);
    atomicAdd(st + S_VISITED, static_cast<unsigned long long>(visited));
    atomicAdd(st + S_UPDATED, static_cast<unsigned long long>(updated));
  }
}

// Mark phase (mark_scan). Also clears tab[0, tab_n), the scan's endpoint dedup
// table, for the next scan.
__global__ void __launch_bounds__(kMarkThreads, kMarkBlocksPerSM) k_mark(
    const __grid_constant__ DMap M, const __grid_constant__ ScanCube Q,
    int4* cast, uint32_t cast_cap, int ox, int oy, int oz, uint4* tab, uint32_t tab_n) {
  __shared__ MarkShared S;
  after_previous();
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < tab_n; t += gridDim.x * blockDim.x)
    tab[t] = make_uint4(kNone, kNone, kNone, kNone);
  const uint32_t n_cast = min(ld_volatile(M.ctr + C_CAST), cast_cap);
  const uint32_t n_segs = ld_volatile(M.ctr + C_SEGS);
  uint32_t visited = 0;
  // The first blocks take the near cells, two rays per thread (one in a small scan): each
  // of them ORs its whole neighbourhood into the bitmap at its end, but a thread's rays
  // are walked one after the other (room scan, 40 k rays: one ray 19.0 us, two 17.5, four
  // 22.8; depth, 70 k: 63.0, 59.4, 59.0). On both sides of the line, mark and apply with one
  // ray and two: LiDAR, 4.7 k rays 24.5, 26.6, 14 k 31.4, 32.7, 29 k 42.3, 42.0; room at 2 cm
  // 8.6 k 32.5, 34.8, 18 k 36.8, 38.2, 35 k 48.8, 45.8; depth 8.2 k 25.9, 27.0, 16 k 29.0,
  // 28.7: one is a little faster up to about 20 k, also above the line.
  // The segments start at the blocks after them: no block of a small scan has both (2k points:
  // 9.5 us, 14.5 with both in the first blocks). A block takes 256 segments side by side:
  // warps that take them 32 by 32 in turn over the grid share fewer words (2k points 13.1 us
  // against 8.5, LiDAR 28.4 against 24.1).
  const uint32_t per = n_cast > 8192u ? 2 * kMarkThreads : kMarkThreads;
  const uint32_t near_blocks = min((n_cast + per - 1u) / per, gridDim.x);
  const uint32_t v = (blockIdx.x + gridDim.x - near_blocks) % gridDim.x;
  mark_scan(M, Q, cast, blockIdx.x < near_blocks ? blockIdx.x * kMarkThreads : n_cast, n_cast,
            v * kMarkThreads + (threadIdx.x & ~31u), Q.segs ? n_segs : 0u,
            near_blocks * kMarkThreads, gridDim.x * kMarkThreads, ox, oy, oz, S, visited);
  visited = __reduce_add_sync(0xffffffffu, visited);
  if ((threadIdx.x & 31) == 0 && visited)
    atomicAdd(reinterpret_cast<unsigned long long*>(M.ctr + C_STATS) + S_VISITED,
              static_cast<unsigned long long>(visited));
}

// Apply phase (apply_scan).
__global__ void __launch_bounds__(256, 4) k_apply_rays(const __grid_constant__ DMap M,
                                                    const __grid_constant__ ScanCube Q, int32_t u,
                                                    int32_t miss, int32_t cmin) {
  __shared__ uint32_t pre[kRootFlagWords], sums[kApplyWarps];
  __shared__ ApplyShared S;
  after_previous();
  const uint32_t n_roots = apply_roots(Q, pre, sums);
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t updated = 0;
  apply_scan(M, Q, n_roots, pre, gw, (gridDim.x * blockDim.x) >> 5, u, miss, cmin,
             S.rows[threadIdx.x >> 5], updated);
  updated = __reduce_add_sync(0xffffffffu, updated);
  if ((threadIdx.x & 31) == 0 && updated)
    atomicAdd(reinterpret_cast<unsigned long long*>(M.ctr + C_STATS) + S_UPDATED,
              static_cast<unsigned long long>(updated));
}

// The parts of the scan's rays that the cube does not hold (tail_rays).
__global__ void __launch_bounds__(256) k_tail(const __grid_constant__ DMap M,
                                              const __grid_constant__ ScanCube Q,
                                              int4* cast, uint32_t cast_cap, int ox, int oy,
                                              int oz, int32_t u, int32_t miss, int32_t cmin) {
  after_previous();
  uint32_t visited = 0, updated = 0;
  tail_rays(M, Q, cast, cast_cap, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
            (gridDim.x * blockDim.x) >> 5, ox, oy, oz, u, miss, cmin, visited, updated);
  tail_count(M, visited, updated);
}

// isOccupied / isUnknown / isFree (probabilistic_map.cpp:56-75).
__global__ void k_query(const __grid_constant__ DMap M, const int32_t* __restrict__ xyz, uint32_t n, int mode,
                        int32_t thr, uint8_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
  const uint32_t lf = leaf_of(M, x, y, z, false);
  bool have = false;
  int32_t p = 0;
  if (lf != kNone) {
    // The cell word first: an on cell of a ProbabilisticMap has update_id in
    // 1..3 (a nonzero word), an off cell holds zero, so only a zero word
    // needs the mask bit (it may be an on cell written through the grid).
    const uint32_t ci = leaf_index(M, x, y, z);
    const int32_t w = reinterpret_cast<const int32_t*>(M.ldata)[size_t(lf) * M.lsize + ci];
    have = w != 0 || cell_is_on(M, lf, ci);
    p = cell_prob(w);
  }
  uint8_t r;
  if (mode == 0)
    r = have && p > thr;
  else if (mode == 1)
    r = have ? p == thr : 1;
  else
    r = have && p < thr;
  out[i] = r;
}

// ComputeRay for a batch of rays (probabilistic_map.hpp:13-19), thread per ray.
__global__ void k_compute_rays(const int32_t* __restrict__ o, const int32_t* __restrict__ e,
                               uint32_t n, uint32_t* __restrict__ len,
                               const unsigned long long* __restrict__ off,
                               int32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int ox = o[3 * i], oy = o[3 * i + 1], oz = o[3 * i + 2];
  const int dx = e[3 * i] - ox, dy = e[3 * i + 1] - oy, dz = e[3 * i + 2] - oz;
  const uint32_t ax = abs(dx), ay = abs(dy), az = abs(dz);
  const uint32_t m = max(ax, max(ay, az));
  if (len) len[i] = m;
  if (!out || m == 0 || m >= kMaxRayCells) return;
  const uint32_t two_m = 2u * m;
  const float rtm = __frcp_rn(static_cast<float>(two_m));
  AxisStep X, Y, Z;
  axis_init(X, ax, m, two_m, rtm, 0, 1);
  axis_init(Y, ay, m, two_m, rtm, 0, 1);
  axis_init(Z, az, m, two_m, rtm, 0, 1);
  int32_t* dst = out + 3 * off[i];
  for (uint32_t k = 0; k < m; k++) {
    dst[3 * k + 0] = ox + (dx < 0 ? -int(X.n) : int(X.n));
    dst[3 * k + 1] = oy + (dy < 0 ? -int(Y.n) : int(Y.n));
    dst[3 * k + 2] = oz + (dz < 0 ? -int(Z.n) : int(Z.n));
    axis_advance(X, two_m);
    axis_advance(Y, two_m);
    axis_advance(Z, two_m);
  }
}

}  // namespace bxg

using namespace bxg;

namespace {

Opts opts_of(const bxg_pmap_s* pm) {
  return Opts{pm->opt.prob_miss_log, pm->opt.prob_hit_log, pm->opt.clamp_min_log,
              pm->opt.clamp_max_log};
}

// logods(p) = int32_t(1e6 * log(p / (1.0 - p))) (probabilistic_map.hpp:34-36).
int32_t logods(float p) {
  return static_cast<int32_t>(1e6 * std::log(p / (1.0 - p)));
}

void record(bxg_pmap_s* pm, int k) {
  if ((pm->core.flags & BXG_FLAG_TIMING) && pm->ev[k]) cudaEventRecord(pm->ev[k], pm->core.stream);
}

int reset_scan_stats(MapCore* m) {
  BXG_CUDA(m, cudaMemsetAsync(m->ctr.as<uint32_t>() + C_STATS, 0, S_COUNT * 8, m->stream));
  return BXG_OK;
}

// Endpoint phase for n staged points (k_endpoints or k_endpoints_kind), then
// the winners that join the ray list, then the endpoint updates.
template <class Launch>
int endpoint_phase(bxg_pmap_s* pm, uint32_t n, int ox, int oy, int oz, const ScanCube& cube,
                   Launch&& launch_ep) {
  MapCore* m = &pm->core;
  const uint32_t tcap = dedup_entries(n);
  BXG_CUDA(m, m->s_ep.ensure(size_t(n) * 16));
  const void* old_tab = m->s_dedup.p;
  const uint32_t tab_n = dedup_key(cube).packed ? tcap / 2 : tcap;  // 16-byte units
  BXG_CUDA(m, m->s_dedup.ensure(size_t(tab_n) * 16));
  if (m->s_dedup.p != old_tab) m->dedup_clean = 0;
  // the ray list persists across add-batches until updateFreeCells
  const uint64_t need = pm->cast_ub + n;
  BXG_CUDA(m, m->s_cast.ensure_keep(need * 16, pm->cast_ub * 16, m->stream));
  if (m->dedup_clean < tab_n) launch_dedup_clear(m, m->s_dedup.as<uint4>(), tab_n);
  m->dedup_clean = 0;
  m->dedup_used = std::max(m->dedup_used, tab_n);
  const unsigned blocks = (n + 255) / 256;
  launch_ep(blocks, m->s_ep.as<int4>(), m->s_dedup.as<uint4>(), tcap - 1);
  BXG_LAUNCHED(m);
  record(pm, 1);
  launch_after(k_winners, blocks, 256, m->stream, m->dm, m->s_ep.as<int4>(), n,
               m->s_dedup.as<uint4>(), tcap - 1, ox, oy, oz, pm->update_count, opts_of(pm),
               m->s_cast.as<int4>(), uint32_t(m->s_cast.cap / 16), cube);
  BXG_LAUNCHED(m);
  record(pm, 2);
  pm->cast_ub = need;
  pm->list_cube = cube;
  return BXG_OK;
}

int launch_apply(bxg_pmap_s* pm) {
  MapCore* m = &pm->core;
  const unsigned blocks =
      unsigned(std::min<uint64_t>((pm->cast_ub + 255) / 256, uint64_t(m->sm_count) * 8));
  if (blocks) {
    k_apply<<<std::max(blocks, 1u), 256, 0, m->stream>>>(
        m->dm, m->s_cast.as<int4>(), uint32_t(m->s_cast.cap / 16), pm->update_count,
        opts_of(pm));
    BXG_LAUNCHED(m);
  }
  return BXG_OK;
}

}  // namespace

namespace bxg {
// The leaf directory for a scan from (ox, oy, oz) whose ray cells lie within
// pm->dir_reach of the origin: a cube of words over leaf coordinates, each
// (epoch << 28) | leaf slot. The cube and its words are kept across scans: a
// scan reuses them while its own cube of leaves lies inside and no leaf slot
// was released since they were written (MapCore::leaf_gen). Otherwise a new
// cube, centred on this origin with a margin so that a moving sensor keeps it
// for several scans, takes the next epoch. The whole buffer is cleared when
// the 4-bit epoch wraps, so a word of another epoch is always empty. *D stays
// empty (the walk probes the root hash for every leaf run) when the cube would
// exceed max_words words, when there is no memory for it, or leaf slots do not fit in 28 bits.
int leaf_dir_for_scan(bxg_pmap_s* pm, int ox, int oy, int oz, LeafDir* D, size_t max_words) {
  MapCore* m = &pm->core;
  *D = LeafDir{};
  if (!(pm->dir_reach > 0) || m->dm.lcap >= (1u << 28)) return BXG_OK;
  const double cells = std::ceil(pm->dir_reach * m->inv_res) + 2;
  const double halfd = std::ceil(cells / double(1 << m->dm.lb)) + 1;
  if (!(halfd < 128)) return BXG_OK;
  const int half = int(halfd);
  const int cx = ox >> m->dm.lb, cy = oy >> m->dm.lb, cz = oz >> m->dm.lb;
  const int side_now = int(pm->dir_side);
  auto inside = [&](int c, int lo) { return c - half >= lo && c + half < lo + side_now; };
  const bool reuse = pm->dir_live && pm->dir_gen == m->leaf_gen && inside(cx, pm->dir_x0) &&
                     inside(cy, pm->dir_y0) && inside(cz, pm->dir_z0);
  if (!reuse) {
    auto words_of = [](int h) { return size_t(2 * h + 1) * (2 * h + 1) * (2 * h + 1); };
    int h = half + std::max(2, half / 4);
    if (words_of(h) > max_words) h = half;
    if (words_of(h) > max_words) return BXG_OK;
    const size_t words = words_of(h);
    if (m->s_dir.cap < words * 4) {
      pm->dir_live = false;
      const cudaError_t e = m->s_dir.ensure(words * 4);
      if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return BXG_OK;
      }
      BXG_CUDA(m, e);
      BXG_CUDA(m, cudaMemsetAsync(m->s_dir.p, 0, m->s_dir.cap, m->stream));
      pm->dir_epoch = 0;
    }
    if (++pm->dir_epoch == 16) {  // the epoch wraps: clear every word ever written
      BXG_CUDA(m, cudaMemsetAsync(m->s_dir.p, 0, m->s_dir.cap, m->stream));
      pm->dir_epoch = 1;
    }
    pm->dir_x0 = cx - h;
    pm->dir_y0 = cy - h;
    pm->dir_z0 = cz - h;
    pm->dir_side = uint32_t(2 * h + 1);
    pm->dir_gen = m->leaf_gen;
    pm->dir_live = true;
  }
  D->words = m->s_dir.as<uint32_t>();
  D->side = pm->dir_side;
  D->x0 = pm->dir_x0;
  D->y0 = pm->dir_y0;
  D->z0 = pm->dir_z0;
  D->epoch = pm->dir_epoch;
  return BXG_OK;
}
}  // namespace bxg

namespace bxg {
constexpr uint64_t kOpenRays = 65536;
constexpr double kOpenCells = 1024.0;
// Ray ends lie within this many cells of the origin cell (the floor of the origin and of
// the end each move a cell by less than one).
static double reach_cells(const MapCore* m, double reach) {
  return std::ceil(reach * m->inv_res) + 2.0;
}
bool open_reach(const MapCore* m, double reach) {
  return !(reach_cells(m, reach) <= 32.0 * kMaxCubeHalf);
}
size_t open_cube_held(const bxg_pmap_s* pm) {
  return pm->cube_bits.cap == kOpenCubeBytes ? kOpenCubeBytes : 0;
}
void drop_open_cube(bxg_pmap_s* pm) {
  if (!open_cube_held(pm)) return;
  pm->cube_bits.release();
  pm->cube_blocks = 0;
  pm->list_cube = ScanCube{};
}

int scan_cube(bxg_pmap_s* pm, int ox, int oy, int oz, double reach, uint64_t rays, ScanCube* Q,
              bool* ok) {
  MapCore* m = &pm->core;
  *ok = false;
  *Q = ScanCube{};
  if (m->dm.lb != 3 || m->dm.ib != 2 || m->dm.esz != 4 ||
      (m->flags & (BXG_FLAG_KEEP_NONFINITE | BXG_FLAG_RAYS_SINGLE_PASS)) || !(reach > 0))
    return BXG_OK;
  int h = kOpenCubeHalf;
  if (open_reach(m, reach)) {
    // With a range just above the largest cube, every ray without a return leaves the cube by
    // little, and the tree is faster up to some ten thousand points (us, on the tree and
    // with the cube: LiDAR, 800 cells at 0.2 m, 2 k points 82, 102, 8 k 97, 119, 30 k 170, 178,
    // 131 k 235, 195; room, 1000 cells at 5 mm, 2 k 108, 212, 30 k 392, 499). Beyond, few rays
    // are that long (LiDAR, 1200 cells at 0.05 m, 2 k 123, 115, 8 k 169, 139; 2000 cells 8 k
    // 290, 163; no limit, returns to 100 m, 2 k 139, 80).
    if (rays && rays < kOpenRays && reach_cells(m, reach) <= kOpenCells) {
      *Q = ScanCube{};
      return BXG_OK;
    }
    Q->open = 1;
    if (core_mem_usage(m) + kOpenCubeBytes > m->budget) {
      drop_open_cube(pm);
      *Q = ScanCube{};
      return BXG_OK;
    }
  } else {
    h = std::max(1, (int(reach_cells(m, reach)) + 31) / 32);
  }
  Q->SR = uint32_t(2 * h + 1);
  Q->S = 4 * Q->SR;
  // cells k <= 32 h of a ray lie within h roots of the origin's
  Q->kin = uint32_t(32 * h + 1);
  const size_t blocks = size_t(Q->S) * Q->S * Q->S;
  // Without memory for one of the buffers the rays are walked on the tree.
  auto grow = [&](DevBuf& b, size_t bytes, bool exact, bool* got) -> int {
    const cudaError_t e = exact ? b.ensure_exact(bytes) : b.ensure(bytes);
    *got = e == cudaSuccess;
    if (e != cudaSuccess && e != cudaErrorMemoryAllocation) BXG_CUDA(m, e);
    if (!*got) {
      cudaGetLastError();
      *Q = ScanCube{};
    }
    return BXG_OK;
  };
  bool got = true;
  if (blocks > pm->cube_blocks) {
    pm->cube_blocks = 0;
    int st = grow(pm->cube_bits, blocks * 64, Q->open != 0, &got);
    if (!st && got) st = grow(pm->cube_roots, kRootFlagWords * 4, false, &got);
    if (st || !got) return st;
    BXG_CUDA(m, cudaMemsetAsync(pm->cube_bits.p, 0, pm->cube_bits.cap, m->stream));
    BXG_CUDA(m, cudaMemsetAsync(pm->cube_roots.p, 0, pm->cube_roots.cap, m->stream));
    pm->cube_blocks = blocks;
    // the batched tick uses the buffers from another stream
    BXG_CUDA(m, cudaStreamSynchronize(m->stream));
  }
  // 2 GB at most. (LiDAR, 17 M points at 0.05 m, rays of up to 602 cells: 0.64 ms; rays walked
  // whole, a thread each: 0.92.)
  const uint64_t segs = rays * max_segments(*Q);
  if (rays && rays <= kMaxSegRays && segs <= (1u << 29)) {
    const int st = grow(pm->ray_segs, segs * 4, false, &got);
    if (st || !got) return st;
    Q->segs = pm->ray_segs.as<uint32_t>();
  }
  if (rays && Q->open) {
    const int st = grow(pm->ray_tails, rays * 4, false, &got);
    if (st || !got) return st;
    Q->tails = pm->ray_tails.as<uint32_t>();
  }
  Q->bits = pm->cube_bits.as<uint32_t>();
  Q->roots = pm->cube_roots.as<uint32_t>();
  Q->x0 = ((ox >> 5) - h) * 32;
  Q->y0 = ((oy >> 5) - h) * 32;
  Q->z0 = ((oz >> 5) - h) * 32;
  *ok = true;
  return BXG_OK;
}
}  // namespace bxg

namespace {

using RayKernel = void (*)(DMap, const int4*, uint32_t, int, int, int, int32_t, int32_t, int32_t,
                           uint4*, uint32_t, LeafDir);

RayKernel ray_kernel(uint32_t rpw, bool u2) {
  if (rpw == 4) return u2 ? k_rays<8, 2> : k_rays<8, 1>;
  if (rpw == 2) return u2 ? k_rays<16, 2> : k_rays<16, 1>;
  return u2 ? k_rays<32, 2> : k_rays<32, 1>;
}

// Launch shape of the ray kernel: one resident wave (SM count x blocks per
// SM), each warp walking every (grid warps)-th ray of the list. Blocks of 1024
// threads (one per SM) let 32 warps walk 32 neighbouring rays of the list at
// once, which share cells and leaves in the SM's L1; scans with fewer ray
// slots than two such waves (the point count bounds the ray count) launch
// 256-thread blocks instead, so that their few rays still reach every SM
// (LiDAR scans: 256 threads faster at 4 k points, 1024 from 16 k points).
// U = 2 kernels hold 80 registers and launch 256 threads.
int launch_rays(bxg_pmap_s* pm, int ox, int oy, int oz) {
  MapCore* m = &pm->core;
  if (!pm->cast_ub) return BXG_OK;
  // rays left by a scan that failed, now cast from another origin: how far they reach, and
  // where they would be cut into segments, is not known
  const int* lo = pm->list_origin;
  if (lo[0] != ox || lo[1] != oy || lo[2] != oz) {
    pm->list_cube = ScanCube{};
    pm->dir_reach = 0.0;
  }
  {
    // two-phase form: mark the rays' cells, then apply per leaf. Rays queued by
    // addHitPoint/addMissPoint batches have no segments and are walked on the tree (100 k of
    // 60-400 cells, with the batch that queues them: 590 us; 1425 marked, a thread per ray)
    const ScanCube& Q = pm->list_cube;
    if (Q.bits) {
      const Opts o = opts_of(pm);
      const uint32_t ccap = uint32_t(m->s_cast.cap / 16);
      const uint32_t tab_n = m->dedup_used;
      // one resident wave, and no more blocks than have a ray or segment per thread
      const uint64_t pieces = pm->cast_ub * (1 + (Q.kin - 1) / kSegCells);
      const unsigned mblocks = unsigned(
          std::min<uint64_t>(uint64_t(m->sm_count) * kMarkBlocksPerSM,
                             (pieces + kMarkThreads - 1) / kMarkThreads));
      launch_after(k_mark, mblocks, kMarkThreads, m->stream, m->dm, Q, m->s_cast.as<int4>(), ccap,
                   ox, oy, oz, m->s_dedup.as<uint4>(), tab_n);
      BXG_LAUNCHED(m);
      // the marked roots are at most those of the cube, or of the rays' pieces
      const uint64_t rows = 16 * std::min<uint64_t>(uint64_t(Q.SR) * Q.SR * Q.SR, 8 * pieces);
      const unsigned ablocks =
          unsigned(std::min<uint64_t>(uint64_t(m->sm_count) * 12, (rows + 7) / 8));
      launch_after(k_apply_rays, ablocks, 256, m->stream, m->dm, Q, pm->update_count, o.miss,
                   o.cmin);
      BXG_LAUNCHED(m);
      if (Q.open) {
        const unsigned tblocks = unsigned(std::min<uint64_t>(
            uint64_t(m->sm_count) * 8, (pm->cast_ub * kTailPieces + 7) / 8));
        launch_after(k_tail, tblocks, 256, m->stream, m->dm, Q, m->s_cast.as<int4>(), ccap, ox,
                     oy, oz, pm->update_count, o.miss, o.cmin);
        BXG_LAUNCHED(m);
      }
      m->dedup_clean = std::max(m->dedup_clean, tab_n);
      m->dedup_used = 0;
      return BXG_OK;
    }
  }
  const uint32_t rpw = m->rays_per_warp ? m->rays_per_warp : 1;
  const bool u2 = m->ray_unroll == 2;
  const int bs_max = u2 ? 256 : 1024;
  const bool wide = pm->cast_ub >= uint64_t(2) * m->sm_count * 32 * rpw;
  const int bs = m->block_size ? std::min(bs_max, std::max(64, int(m->block_size) & ~31))
                               : (wide ? bs_max : 256);
  const RayKernel kern = ray_kernel(rpw, u2);
  const int wi = bs == 1024 ? 1 : 0;  // cached residency of the two default shapes
  if (m->ray_wave_bs[wi] != bs) {
    int per_sm = 0;
    BXG_CUDA(m, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                    &per_sm, reinterpret_cast<const void*>(kern), bs, 0));
    m->ray_wave_blocks[wi] = uint32_t(std::max(per_sm, 1)) * uint32_t(m->sm_count);
    m->ray_wave_bs[wi] = bs;
  }
  const uint64_t groups_per_block = uint64_t(bs) / (32 / rpw);
  uint64_t blocks = (pm->cast_ub + groups_per_block - 1) / groups_per_block;
  blocks = std::min<uint64_t>(blocks, m->ray_wave_blocks[wi]);
  if (!blocks) return BXG_OK;
  const Opts o = opts_of(pm);
  const uint32_t ccap = uint32_t(m->s_cast.cap / 16);
  const dim3 g{unsigned(blocks)}, b{unsigned(bs)};
  const uint32_t tab_n = m->dedup_used;
  LeafDir dir{};
  int st = leaf_dir_for_scan(pm, ox, oy, oz, &dir, size_t(1) << 24);
  if (st) return st;
  kern<<<g, b, 0, m->stream>>>(m->dm, m->s_cast.as<int4>(), ccap, ox, oy, oz, pm->update_count,
                               o.miss, o.cmin, m->s_dedup.as<uint4>(), tab_n, dir);
  BXG_LAUNCHED(m);
  m->dedup_clean = std::max(m->dedup_clean, tab_n);
  m->dedup_used = 0;
  return BXG_OK;
}

// Applies the queued endpoints (if not yet applied) and casts the rays,
// growing pools and retrying on exhaustion; then ends the scan.
int finish_scan(bxg_pmap_s* pm, int ox, int oy, int oz, bool cast_rays, uint64_t* ray_cells,
                bool include_points) {
  MapCore* m = &pm->core;
  int st = BXG_OK;
  for (int attempt = 0; attempt < 12; attempt++) {
    if (attempt) {
      // a retry walks every ray again (recount the visits) but updates only
      // the cells the failed attempt could not reach: the updated-cell count
      // adds up over the attempts
      unsigned long long* s = stats_of(m);
      BXG_CUDA(m, cudaMemsetAsync(s + S_VISITED, 0, 8, m->stream));
    }
    if (attempt) {  // the winners applied the endpoints; complete them after growth
      st = launch_apply(pm);
      if (st) return st;
    }
    record(pm, 3);
    if (cast_rays) {
      st = launch_rays(pm, ox, oy, oz);
      if (st) return st;
    }
    record(pm, 4);
    uint32_t err = 0;
    st = core_sync(m, &err);
    if (st == BXG_OK) break;
    if (!(err & (ERR_POOL_INNER | ERR_POOL_LEAF | ERR_HASH_FULL)) ||
        (err & (ERR_WAIT | ERR_RAY_TOO_LONG | ERR_SCRATCH)))
      return st;
    const int g = core_grow_for(m, err);
    if (g) return g;
  }
  if (st) return st;
  const unsigned long long* hs = reinterpret_cast<const unsigned long long*>(m->h_ctr + C_STATS);
  pm->last_stats[0] = hs[S_POINTS];
  pm->last_stats[1] = pm->cast_ub ? m->h_ctr[C_CAST] : 0;
  pm->last_stats[2] = hs[S_VISITED];
  pm->last_stats[3] = hs[S_UPDATED];
  pm->last_stats[4] = m->h_ctr[C_LEAF];
  pm->last_stats[5] = m->launches;
  if (ray_cells) *ray_cells = (include_points ? hs[S_POINTS] : 0) + hs[S_RAY_LEN];
  if (m->flags & BXG_FLAG_TIMING) {
    for (int k = 0; k < 4; k++) {
      float ms = 0;  // a phase that never ran has no event yet
      if (pm->ev[k] && pm->ev[k + 1] &&
          cudaEventElapsedTime(&ms, pm->ev[k], pm->ev[k + 1]) != cudaSuccess) {
        cudaGetLastError();
        ms = 0;
      }
      pm->last_times[k] = ms;
    }
  }
  if (cast_rays) {
    // end of scan: empty the ray list (the next scan's first kernel zeroes
    // the device count), advance the counter (cpp:301-310)
    pm->cast_ub = 0;
    pm->dir_reach = 0.0;
    if (++pm->update_count == 4) pm->update_count = 1;
  }
  return core_maintain(m);
}

// Σ Chebyshev length from origin cell o of the rays queued by addHitPoint /
// addMissPoint batches (their add-time lengths were measured from (0,0,0)):
// read back and summed on the host; this path is not the streaming one.
int queued_ray_cells(bxg_pmap_s* pm, const int* o, uint64_t* len) {
  MapCore* m = &pm->core;
  *len = 0;
  if (!pm->cast_ub) return BXG_OK;
  int st = core_sync(m);
  if (st) return st;
  const uint32_t n_cast = m->h_ctr[C_CAST];
  if (!n_cast) return BXG_OK;
  std::vector<int4> h(n_cast);
  BXG_CUDA(m, cudaMemcpy(h.data(), m->s_cast.p, size_t(n_cast) * 16, cudaMemcpyDeviceToHost));
  for (const int4& e : h) {
    const int64_t dx = std::llabs(int64_t(e.x) - o[0]), dy = std::llabs(int64_t(e.y) - o[1]),
                  dz = std::llabs(int64_t(e.z) - o[2]);
    *len += uint64_t(std::max(dx, std::max(dy, dz)));
  }
  return BXG_OK;
}

int origin_coord(const MapCore* m, double x, double y, double z, int* c) {
  c[0] = static_cast<int>(std::floor(x * m->inv_res));
  c[1] = static_cast<int>(std::floor(y * m->inv_res));
  c[2] = static_cast<int>(std::floor(z * m->inv_res));
  return BXG_OK;
}

template <typename PT>
int insert_impl(bxg_pmap m_, const PT* xyz, size_t stride, size_t n, const PT* origin,
                double max_range, uint64_t* ray_cells, bool sync, const Xf* xf = nullptr) {
  if (!m_) return BXG_ERR_INVALID_ARG;
  bxg_pmap_s* pm = m_;
  MapCore* m = &pm->core;
  if (!origin || (n && !xyz) || n >= 0x7FFFFFFFu)
    return set_error(m, BXG_ERR_INVALID_ARG, "null input or batch too large");
  if (!stride) stride = 3 * sizeof(PT);
  cudaSetDevice(m->device);
  // from = ConvertPoint<Vector3d>(origin): the origin widened to double.
  const double fx = static_cast<double>(origin[0]), fy = static_cast<double>(origin[1]),
               fz = static_cast<double>(origin[2]);
  int o[3];
  origin_coord(m, fx, fy, fz, o);
  // rays queued by earlier addHitPoint/addMissPoint batches are cast by this
  // scan too (updateFreeCells, probabilistic_map.hpp:159): count their cells
  uint64_t queued = 0;
  if (ray_cells && pm->cast_ub) {
    const int qs = queued_ray_cells(pm, o, &queued);
    if (qs) return qs;
  }
  // Headroom for this scan's new leaves (twice the last scan's, at least a
  // quarter of the points), so that the scan rarely has to grow and re-run.
  const uint32_t leaves_before = m->h_ctr[C_LEAF];
  int st = core_reserve(m, std::max<size_t>({size_t(2) * pm->last_new_leaves, n / 4, 1024}),
                        std::max<size_t>(n / 64, 256));
  if (st) return st;
  record(pm, 0);  // the scan's device time starts here
  if (!n) {  // otherwise the endpoint kernel zeroes the statistics
    st = reset_scan_stats(m);
    if (st) return st;
  }
  if (n) {
    const void* dpts = nullptr;
    st = stage_in(m, m->s_in, xyz, stride * (n - 1) + 3 * sizeof(PT), &dpts);
    if (st) return st;
    const double mr2 = max_range * max_range;
    const int keep = (m->flags & BXG_FLAG_KEEP_NONFINITE) ? 1 : 0;
    // rays of this scan end within max_range of the origin (hits are closer);
    // rays queued by earlier add batches may not: no directory then
    pm->dir_reach = pm->cast_ub == 0 ? max_range : 0.0;
    std::copy(o, o + 3, pm->list_origin);
    // the winners cut the rays of a scan that starts its list into segments
    ScanCube cube{};
    if (pm->cast_ub == 0) {
      bool ok = false;
      st = scan_cube(pm, o[0], o[1], o[2], max_range, n, &cube, &ok);
      if (st) return st;
    }
    const uint32_t root_words = cube.roots ? cube_root_words(cube) : 0;
    const int zero = ZERO_STATS | ZERO_RAYS | (pm->cast_ub == 0 ? ZERO_CAST : 0);
    const DedupKey key = dedup_key(cube);
    EpFast fast = make_ep_fast(fx, fy, fz, max_range, m->inv_res);
    if (sizeof(PT) != 4) fast.on = 0;
    st = endpoint_phase(pm, uint32_t(n), o[0], o[1], o[2], cube,
                        [&](unsigned blocks, int4* ep, uint4* tab, uint32_t tmask) {
                          if (xf)
                            k_endpoints_sensor<<<blocks, 256, 0, m->stream>>>(
                                m->dm, static_cast<const uint8_t*>(dpts), stride, uint32_t(n),
                                *xf, fx, fy, fz, max_range, mr2, m->inv_res, ep, tab, tmask, zero,
                                fast, cube.roots, root_words, key);
                          else
                            k_endpoints<PT><<<blocks, 256, 0, m->stream>>>(
                                m->dm, static_cast<const uint8_t*>(dpts), stride, uint32_t(n), fx,
                                fy, fz, max_range, mr2, m->inv_res, keep, ep, tab, tmask, zero,
                                fast, cube.roots, root_words, key);
                        });
    if (st) return st;
  }
  if (!sync) {
    // asynchronous form: no retry; pools must have room (see core_maintain)
    st = launch_rays(pm, o[0], o[1], o[2]);
    if (st) return st;
    BXG_CUDA(m, cudaMemsetAsync(m->ctr.as<uint32_t>() + C_CAST, 0, 4, m->stream));
    pm->cast_ub = 0;
    if (++pm->update_count == 4) pm->update_count = 1;
    return BXG_OK;
  }
  st = finish_scan(pm, o[0], o[1], o[2], true, ray_cells, true);
  if (!st) {
    pm->last_new_leaves = m->h_ctr[C_LEAF] > leaves_before ? m->h_ctr[C_LEAF] - leaves_before : 0;
    if (ray_cells) *ray_cells += queued;
  }
  return st;
}

int add_points(bxg_pmap m_, const double* xyz, size_t n, int kind,
               const uint8_t* kinds = nullptr) {
  if (!m_) return BXG_ERR_INVALID_ARG;
  bxg_pmap_s* pm = m_;
  MapCore* m = &pm->core;
  if (!n) return BXG_OK;
  if (!xyz || n >= 0x7FFFFFFFu) return set_error(m, BXG_ERR_INVALID_ARG, "null input");
  cudaSetDevice(m->device);
  record(pm, 0);
  // rays queued here may end anywhere: the coming ray phase has no bound
  pm->dir_reach = 0.0;
  // the first batch after a scan starts the statistics and the ray list
  const int zero = pm->cast_ub == 0 ? (ZERO_STATS | ZERO_CAST) : 0;
  const void* dpts = nullptr;
  const void* dkinds = nullptr;
  int st = stage_in(m, m->s_in, xyz, n * 24, &dpts);
  if (st) return st;
  if (kinds) {
    st = stage_in(m, m->s_in2, kinds, n, &dkinds);
    if (st) return st;
  }
  st = endpoint_phase(pm, uint32_t(n), 0, 0, 0, ScanCube{},
                      [&](unsigned blocks, int4* ep, uint4* tab, uint32_t tmask) {
                        k_endpoints_kind<<<blocks, 256, 0, m->stream>>>(
                            m->dm, static_cast<const double*>(dpts), uint32_t(n), kind,
                            static_cast<const uint8_t*>(dkinds), m->inv_res, ep, tab, tmask,
                            zero);
                      });
  if (st) return st;
  // apply now so that queries see the endpoint updates, as in the reference
  return finish_scan(pm, 0, 0, 0, false, nullptr, false);
}

// The occupied-voxel export of bonxai_server.cpp:217-243 as one compaction:
// each occupied cell (probability_log > thr, probabilistic_map.cpp:108-116)
// becomes its corner position coordToPos(c) = double(c) * res
// (bonxai.hpp:413-417), kept when min_z <= z <= max_z, narrowed to float
// xyz (the PCLPoint the node publishes). Order is unspecified, as the
// reference's unordered_map order is. (A ProbabilisticMap's leaves are 8^3.)
//
// A lane looks at rows of 8 cells (one mask byte, one 32-byte sector, one z): two of each of
// its warp's kExportLeaves leaves, all their mask bytes loaded at once; only the
// words of on cells in rows of the band are read, and the block takes its output range
// with one atomic. Bound by the latency of mask, then cells. 82 k leaves with 26 k occupied
// cells: 29 us (134 us with a thread per mask word, up to 64 cells one after the other).
constexpr int kExportLeaves = 2;  // per warp (1: the same; 4: 33 us, 8: 38 us)
__global__ void __launch_bounds__(256) k_export_occupied(const __grid_constant__ DMap M, uint32_t n_leaves, float* __restrict__ out, size_t cap,
                                  unsigned long long* __restrict__ counter, int32_t thr,
                                  double res, double min_z, double max_z) {
  __shared__ uint32_t s_cnt[8];
  __shared__ unsigned long long s_base;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t leaf0 = (blockIdx.x * 8u + warp) * kExportLeaves;
  const uint8_t* mask = reinterpret_cast<const uint8_t*>(M.lmask);
  int4 key[kExportLeaves];
  uint32_t on[kExportLeaves][2];
#pragma unroll
  for (int l = 0; l < kExportLeaves; ++l) {
    key[l] = make_int4(0, 0, 0, -1);
    on[l][0] = on[l][1] = 0u;
    if (leaf0 + l < n_leaves) {
      key[l] = M.lkey[leaf0 + l];
      on[l][0] = mask[size_t(leaf0 + l) * 64u + lane];
      on[l][1] = mask[size_t(leaf0 + l) * 64u + 32u + lane];
    }
  }
  // occupied cells of the rows: eight bits each
  uint32_t cnt = 0;
#pragma unroll
  for (int l = 0; l < kExportLeaves; ++l)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double pz = __dmul_rn(double(key[l].z | int((lane >> 3) + 4 * h)), res);
      uint32_t w = key[l].w != -1 && pz >= min_z && pz <= max_z ? on[l][h] : 0u;
      if (w) {
        const int4* c = reinterpret_cast<const int4*>(M.ldata) + size_t(leaf0 + l) * 128u +
                        2u * (lane + 32u * h);
        int4 v[2];
        if (w & 0xFu) v[0] = c[0];
        if (w & 0xF0u) v[1] = c[1];
        const int32_t* x = reinterpret_cast<const int32_t*>(v);
#pragma unroll
        for (int b = 0; b < 8; ++b)
          if (((w >> b) & 1u) && !(cell_prob(x[b]) > thr)) w &= ~(1u << b);
      }
      on[l][h] = w;
      cnt += __popc(w);
    }
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= static_cast<unsigned>(o)) incl += v;
  }
  if (lane == 31) s_cnt[warp] = incl;
  __syncthreads();
  uint32_t before = incl - cnt, total = 0;
#pragma unroll
  for (unsigned w = 0; w < 8; ++w) {
    if (w < warp) before += s_cnt[w];
    total += s_cnt[w];
  }
  if (!total) return;
  if (threadIdx.x == 0) s_base = atomicAdd(counter, static_cast<unsigned long long>(total));
  __syncthreads();
  unsigned long long pos = s_base + before;
#pragma unroll
  for (int l = 0; l < kExportLeaves; ++l)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      for (uint32_t w = on[l][h]; w; w &= w - 1u) {
        const int b = __ffs(static_cast<int>(w)) - 1;
        if (pos < cap) {
          out[3 * pos + 0] = float(__dmul_rn(double(key[l].x | b), res));
          out[3 * pos + 1] = float(__dmul_rn(double(key[l].y | int(lane & 7u)), res));
          out[3 * pos + 2] = float(__dmul_rn(double(key[l].z | int((lane >> 3) + 4 * h)), res));
        }
        pos++;
      }
}

int export_occupied(bxg_pmap m_, float* out_xyz, size_t cap, size_t* n_out, double min_z,
                    double max_z) {
  MapCore* m = &m_->core;
  int st = core_sync(m);
  if (st) return st;
  const uint32_t n_leaves = m->h_ctr[C_LEAF];
  void* dout = nullptr;
  if (cap && out_xyz) {
    st = stage_out(m, m->s_out, out_xyz, cap * 12, &dout);
    if (st) return st;
  }
  BXG_CUDA(m, m->s_tmp.ensure(8));
  BXG_CUDA(m, cudaMemsetAsync(m->s_tmp.p, 0, 8, m->stream));
  const size_t wcap = dout ? cap : 0;
  if (n_leaves) {
    k_export_occupied<<<(n_leaves + 8 * kExportLeaves - 1) / (8 * kExportLeaves), 256, 0,
                        m->stream>>>(
        m->dm, n_leaves, static_cast<float*>(dout), wcap, m->s_tmp.as<unsigned long long>(),
        m_->opt.occupancy_threshold_log, m->res, min_z, max_z);
    BXG_LAUNCHED(m);
  }
  unsigned long long n = 0;
  BXG_CUDA(m, cudaMemcpyAsync(&n, m->s_tmp.p, 8, cudaMemcpyDeviceToHost, m->stream));
  BXG_CUDA(m, cudaStreamSynchronize(m->stream));
  if (dout) {
    st = stage_out_finish(m, out_xyz, dout, std::min<size_t>(size_t(n), wcap) * 12);
    if (st) return st;
  }
  if (n_out) *n_out = size_t(n);
  if (size_t(n) > cap) return set_error(m, BXG_ERR_CAPACITY, "output buffer too small");
  return BXG_OK;
}

int query(bxg_pmap m_, const int32_t* xyz, size_t n, uint8_t* out, int mode) {
  if (!m_) return BXG_ERR_INVALID_ARG;
  MapCore* m = &m_->core;
  if (!n) return BXG_OK;
  if (!xyz || !out || n >= 0x7FFFFFFFu) return set_error(m, BXG_ERR_INVALID_ARG, "null pointer");
  cudaSetDevice(m->device);
  const void* dxyz = nullptr;
  void* dout = nullptr;
  int st = stage_in(m, m->s_in, xyz, n * 12, &dxyz);
  if (st) return st;
  st = stage_out(m, m->s_out, out, n, &dout);
  if (st) return st;
  record(m_, 0);
  k_query<<<unsigned((n + 255) / 256), 256, 0, m->stream>>>(
      m->dm, static_cast<const int32_t*>(dxyz), uint32_t(n), mode,
      m_->opt.occupancy_threshold_log, static_cast<uint8_t*>(dout));
  BXG_LAUNCHED(m);
  record(m_, 1);
  st = stage_out_finish(m, out, dout, n);
  if (st) return st;
  BXG_CUDA(m, cudaStreamSynchronize(m->stream));
  if ((m->flags & BXG_FLAG_TIMING) && m_->ev[0] && m_->ev[1])
    cudaEventElapsedTime(&m_->last_query_ms, m_->ev[0], m_->ev[1]);
  return BXG_OK;
}

}  // namespace

namespace bxg {
int pmap_complete_scan(bxg_pmap_s* pm, const int4* d_cast, const uint32_t* d_count, uint32_t cap,
                       int ox, int oy, int oz, int32_t u) {
  MapCore* m = &pm->core;
  cudaSetDevice(m->device);
  const Opts o = opts_of(pm);
  uint32_t err = 0;
  int st = core_sync(m, &err);  // reads and clears what the tick left
  if (st && (!(err & (ERR_POOL_INNER | ERR_POOL_LEAF | ERR_HASH_FULL)) ||
              (err & (ERR_WAIT | ERR_RAY_TOO_LONG | ERR_SCRATCH))))
    return st;
  if (d_count != m->ctr.as<uint32_t>() + C_CAST)
    BXG_CUDA(m, cudaMemcpyAsync(m->ctr.as<uint32_t>() + C_CAST, d_count, 4,
                                cudaMemcpyDeviceToDevice, m->stream));
  for (int attempt = 0; attempt < 12 && err; attempt++) {
    st = core_grow_for(m, err);
    if (st) return st;
    const unsigned ablocks = unsigned(std::min<uint64_t>((cap + 255) / 256, uint64_t(m->sm_count) * 8));
    k_apply<<<std::max(ablocks, 1u), 256, 0, m->stream>>>(m->dm, d_cast, cap, u, o);
    BXG_LAUNCHED(m);
    const unsigned rblocks = unsigned(std::min<uint64_t>((cap + 7) / 8, uint64_t(m->sm_count) * 8));
    k_rays<32, 1><<<std::max(rblocks, 1u), 256, 0, m->stream>>>(m->dm, d_cast, cap, ox, oy, oz,
                                                               u, o.miss, o.cmin, nullptr, 0,
                                                               LeafDir{});
    BXG_LAUNCHED(m);
    st = core_sync(m, &err);
    if (st && (!(err & (ERR_POOL_INNER | ERR_POOL_LEAF | ERR_HASH_FULL)) ||
              (err & (ERR_WAIT | ERR_RAY_TOO_LONG | ERR_SCRATCH))))
    return st;
  }
  BXG_CUDA(m, cudaMemsetAsync(m->ctr.as<uint32_t>() + C_CAST, 0, 4, m->stream));
  BXG_CUDA(m, cudaStreamSynchronize(m->stream));
  if (err) return set_error(m, BXG_ERR_OUT_OF_POOL, "pools could not grow enough");
  return BXG_OK;
}

const MapCore* core_of_handle(const void* handle) {
  // Both handle types hold their MapCore as first member.
  return reinterpret_cast<const MapCore*>(handle);
}
}  // namespace bxg

extern "C" {

int bxg_pmap_create(bxg_pmap* out, double resolution, const bxg_config* cfg) {
  if (!out) return BXG_ERR_INVALID_ARG;
  *out = nullptr;
  bxg_pmap pm = new bxg_pmap_s();
  // ProbabilisticMap's grid is VoxelGrid<CellT>(resolution) with default bits.
  int st = core_init(&pm->core, resolution, 2, 3, 4, cfg);
  if (st) {
    set_create_error(pm->core.err);
    delete pm;
    return st;
  }
  pm->opt.prob_miss_log = logods(0.4f);
  pm->opt.prob_hit_log = logods(0.7f);
  pm->opt.clamp_min_log = logods(0.12f);
  pm->opt.clamp_max_log = logods(0.97f);
  pm->opt.occupancy_threshold_log = logods(0.5f);
  if (pm->core.flags & BXG_FLAG_TIMING)
    for (auto& e : pm->ev) cudaEventCreate(&e);
  *out = pm;
  return BXG_OK;
}

int bxg_pmap_destroy(bxg_pmap m) {
  delete m;
  return BXG_OK;
}

int bxg_pmap_get_options(bxg_pmap m, bxg_pmap_options* out) {
  if (!m || !out) return BXG_ERR_INVALID_ARG;
  *out = m->opt;
  return BXG_OK;
}

int bxg_pmap_set_options(bxg_pmap m, const bxg_pmap_options* opt) {
  if (!m || !opt) return BXG_ERR_INVALID_ARG;
  m->opt = *opt;
  return BXG_OK;
}

int bxg_pmap_insert_point_cloud_f32(bxg_pmap m, const float* xyz, size_t stride, size_t n,
                                    const float origin[3], double max_range,
                                    uint64_t* ray_cells) {
  return insert_impl(m, xyz, stride, n, origin, max_range, ray_cells, true);
}

int bxg_pmap_insert_point_cloud_f64(bxg_pmap m, const double* xyz, size_t stride, size_t n,
                                    const double origin[3], double max_range,
                                    uint64_t* ray_cells) {
  return insert_impl(m, xyz, stride, n, origin, max_range, ray_cells, true);
}

int bxg_pmap_insert_point_cloud_f32_async(bxg_pmap m, const float* xyz, size_t stride,
                                          size_t n, const float origin[3], double max_range) {
  return insert_impl(m, xyz, stride, n, origin, max_range, nullptr, false);
}

int bxg_pmap_insert_sensor_cloud_f32(bxg_pmap m, const float* xyz, size_t stride, size_t n,
                                     const float sensor_to_world[12], double max_range,
                                     uint64_t* ray_cells) {
  if (!m || !sensor_to_world) return BXG_ERR_INVALID_ARG;
  Xf xf;
  std::memcpy(xf.m, sensor_to_world, sizeof(xf.m));
  // origin = the transform's translation (bonxai_server.cpp:171-173); a
  // negative max_range means no limit (:174-179)
  const float origin[3] = {xf.m[3], xf.m[7], xf.m[11]};
  if (max_range < 0) max_range = HUGE_VAL;
  return insert_impl(m, xyz, stride, n, origin, max_range, ray_cells, true, &xf);
}

int bxg_pmap_export_occupied_f32(bxg_pmap m, float* out_xyz, size_t cap, size_t* n_out,
                                 double min_z, double max_z) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  return export_occupied(m, out_xyz, cap, n_out, min_z, max_z);
}

int bxg_pmap_add_hit_points(bxg_pmap m, const double* xyz, size_t n) {
  return add_points(m, xyz, n, EP_HIT);
}

int bxg_pmap_add_miss_points(bxg_pmap m, const double* xyz, size_t n) {
  return add_points(m, xyz, n, EP_MISS);
}

int bxg_pmap_add_points(bxg_pmap m, const double* xyz, const uint8_t* kinds, size_t n) {
  if (n && !kinds) return BXG_ERR_INVALID_ARG;
  return add_points(m, xyz, n, EP_HIT, kinds);
}

bxg_grid bxg_pmap_grid(bxg_pmap m) {
  // Both handle types hold their MapCore first and the grid entry points use
  // only that, so the map itself serves as its VoxelGrid<CellT>.
  return reinterpret_cast<bxg_grid>(m);
}

int bxg_pmap_update_free_cells(bxg_pmap pm, const double origin[3], uint64_t* ray_cells) {
  if (!pm || !origin) return BXG_ERR_INVALID_ARG;
  MapCore* m = &pm->core;
  cudaSetDevice(m->device);
  int o[3];
  origin_coord(m, origin[0], origin[1], origin[2], o);
  uint64_t len = 0;
  if (ray_cells) {
    const int st = queued_ray_cells(pm, o, &len);
    if (st) return st;
  }
  const int st = finish_scan(pm, o[0], o[1], o[2], true, nullptr, false);
  if (st) return st;
  if (ray_cells) *ray_cells = len;
  return BXG_OK;
}

int bxg_pmap_is_occupied(bxg_pmap m, const int32_t* xyz, size_t n, uint8_t* out) {
  return query(m, xyz, n, out, 0);
}
int bxg_pmap_is_unknown(bxg_pmap m, const int32_t* xyz, size_t n, uint8_t* out) {
  return query(m, xyz, n, out, 1);
}
int bxg_pmap_is_free(bxg_pmap m, const int32_t* xyz, size_t n, uint8_t* out) {
  return query(m, xyz, n, out, 2);
}

int bxg_pmap_get_occupied(bxg_pmap m, int32_t* out_xyz, size_t cap, size_t* n_out) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  return core_dump(&m->core, out_xyz, nullptr, cap, n_out, 1, m->opt.occupancy_threshold_log);
}

int bxg_pmap_get_free(bxg_pmap m, int32_t* out_xyz, size_t cap, size_t* n_out) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  return core_dump(&m->core, out_xyz, nullptr, cap, n_out, 2, m->opt.occupancy_threshold_log);
}

int bxg_pmap_dump(bxg_pmap m, int32_t* out_xyz, int32_t* out_cells, size_t cap, size_t* n_out) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  return core_dump(&m->core, out_xyz, out_cells, cap, n_out, 0, 0);
}

int bxg_pmap_active_cells(bxg_pmap m, size_t* out) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  return core_active_cells(&m->core, out);
}

int bxg_pmap_node_counts(bxg_pmap m, size_t* roots, size_t* leaves) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  return core_node_counts(&m->core, roots, leaves);
}

int bxg_pmap_mem_usage(bxg_pmap m, size_t* out) {
  if (!m || !out) return BXG_ERR_INVALID_ARG;
  *out = core_mem_usage(&m->core);
  return BXG_OK;
}

int bxg_pmap_update_count(bxg_pmap m, int* out) {
  if (!m || !out) return BXG_ERR_INVALID_ARG;
  *out = m->update_count;
  return BXG_OK;
}

int bxg_pmap_clear(bxg_pmap m) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  m->cast_ub = 0;
  return core_clear(&m->core);
}

int bxg_pmap_synchronize(bxg_pmap m) {
  if (!m) return BXG_ERR_INVALID_ARG;
  cudaSetDevice(m->core.device);
  int st = core_sync(&m->core);
  if (st) return st;
  return core_maintain(&m->core);
}

int bxg_pmap_last_stats(bxg_pmap m, uint64_t out[8]) {
  if (!m || !out) return BXG_ERR_INVALID_ARG;
  std::memcpy(out, m->last_stats, sizeof(m->last_stats));
  return BXG_OK;
}

int bxg_pmap_last_query_ms(bxg_pmap m, float* ms) {
  if (!m || !ms) return BXG_ERR_INVALID_ARG;
  *ms = m->last_query_ms;
  return BXG_OK;
}

int bxg_pmap_kernel_times(bxg_pmap m, float out[4]) {
  if (!m || !out) return BXG_ERR_INVALID_ARG;
  std::memcpy(out, m->last_times, sizeof(m->last_times));
  return BXG_OK;
}

void* bxg_pmap_stream(bxg_pmap m) { return m ? static_cast<void*>(m->core.stream) : nullptr; }

int bxg_compute_rays(const int32_t* origin_xyz, const int32_t* end_xyz, size_t n,
                     uint32_t* out_len, const uint64_t* offsets, int32_t* out_xyz) {
  if (!n) return BXG_OK;
  if (!origin_xyz || !end_xyz || n >= 0x7FFFFFFFu) return BXG_ERR_INVALID_ARG;
  if (out_xyz && !offsets) return BXG_ERR_INVALID_ARG;
  MapCore tmp;
  tmp.device = -1;
  cudaGetDevice(&tmp.device);
  cudaStream_t s = nullptr;
  BXG_CUDA(&tmp, cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  tmp.stream = s;
  tmp.own_stream = true;
  const void *dO = nullptr, *dE = nullptr, *dOff = nullptr;
  void *dLen = nullptr, *dOut = nullptr;
  int st = stage_in(&tmp, tmp.s_in, origin_xyz, n * 12, &dO);
  if (!st) st = stage_in(&tmp, tmp.s_in2, end_xyz, n * 12, &dE);
  if (!st) st = stage_out(&tmp, tmp.s_out, out_len, n * 4, &dLen);
  size_t total = 0;
  if (!st && out_xyz) {
    // total cells = offsets[n-1] + length of the last ray
    uint64_t last_off = 0;
    if (is_device_ptr(offsets))
      cudaMemcpy(&last_off, offsets + (n - 1), 8, cudaMemcpyDeviceToHost);
    else
      last_off = offsets[n - 1];
    int32_t lo[3], le[3];
    if (is_device_ptr(origin_xyz)) {
      cudaMemcpy(lo, origin_xyz + 3 * (n - 1), 12, cudaMemcpyDeviceToHost);
      cudaMemcpy(le, end_xyz + 3 * (n - 1), 12, cudaMemcpyDeviceToHost);
    } else {
      std::memcpy(lo, origin_xyz + 3 * (n - 1), 12);
      std::memcpy(le, end_xyz + 3 * (n - 1), 12);
    }
    const uint64_t ml = std::max({std::llabs(int64_t(le[0]) - lo[0]),
                                  std::llabs(int64_t(le[1]) - lo[1]),
                                  std::llabs(int64_t(le[2]) - lo[2])});
    total = size_t(last_off + ml);
    st = stage_in(&tmp, tmp.s_ep, offsets, n * 8, &dOff);
    if (!st) st = stage_out(&tmp, tmp.s_out2, out_xyz, total * 12, &dOut);
  }
  if (st) return st;
  k_compute_rays<<<unsigned((n + 255) / 256), 256, 0, s>>>(
      static_cast<const int32_t*>(dO), static_cast<const int32_t*>(dE), uint32_t(n),
      static_cast<uint32_t*>(dLen), static_cast<const unsigned long long*>(dOff),
      static_cast<int32_t*>(dOut));
  BXG_LAUNCHED(&tmp);
  if (dLen) st = stage_out_finish(&tmp, out_len, dLen, n * 4);
  if (!st && dOut) st = stage_out_finish(&tmp, out_xyz, dOut, total * 12);
  if (st) return st;
  BXG_CUDA(&tmp, cudaStreamSynchronize(s));
  return BXG_OK;
}

}  // extern "C"
