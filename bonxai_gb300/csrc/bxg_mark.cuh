// Two-phase ray update of a ProbabilisticMap scan (updateFreeCells,
// probabilistic_map.cpp:77-106): first mark, then apply.
//
// The ray update is a function of each visited cell's own word (a cell whose
// update_id != u becomes {max(p + miss, clamp_min), u}; bxg_scan.cuh), so it
// only needs the SET of cells the scan's rays visit, not the visits:
//
//   mark   Rays are walked without touching the tree. Every visited cell sets
//          its bit in a per-scan bitmap over a cube around the origin, blocked
//          by leaf (one 512-bit block of 16 words per 8^3 leaf, bit =
//          getLeafIndex, x fastest), and the roots it lies in are noted.
//   apply  The leaf blocks of the noted roots are read; a marked one gets its leaf
//          (topology: once per leaf, not once per ray crossing), then the miss
//          update of the marked cells with vector loads and stores, the mask
//          bits of cells turned on, and the block cleared for the next scan.
//
// This is the two-phase insert (topology, then values) over deduplicated
// coordinates: the bitmap is the deduplication. The result equals the per-ray
// walk's bit for bit; the bitmap is scratch that is all zero between scans.
#pragma once

#include "bxg_scan.cuh"

namespace bxg {

// Fire-and-forget OR into global memory: an atomicOr on an address that the
// compiler cannot tell to be global compiles to an atomic that returns its old value, which
// the warp then waits for; this always issues the reduction form.
__device__ __forceinline__ void red_or(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
               "r"(v)
               : "memory");
}
constexpr int kApplyGroup = 8;  // lanes that look for one leaf

// Leaf slot of the leaf whose lowest cell is (lx, ly, lz), created if
// missing, for a group of kApplyGroup lanes (sl = lane in group, gmask = the
// group's lanes). The root bucket is probed cooperatively, one bucket per lane;
// a missing or pending root, a long chain or a missing leaf goes through the
// bounded-wait creation path on the group's first lane.
__device__ __forceinline__ uint32_t apply_leaf_slot(const DMap& M, int lx, int ly, int lz,
                                                    unsigned sl, unsigned gbase, unsigned gmask) {
  const int32_t rm = root_mask(M);
  const int rx = lx & rm, ry = ly & rm, rz = lz & rm;
  const uint32_t h0 = root_hash(M, rx, ry, rz);
  const uint4 bk = M.buckets[(h0 + sl) & M.hmask];
  const bool hit = key_eq(bk, rx, ry, rz);
  const bool empty = static_cast<int>(bk.x) == kEmptyKey;
  const unsigned hm = (__ballot_sync(gmask, hit) & gmask) >> gbase;
  const unsigned em = (__ballot_sync(gmask, empty) & gmask) >> gbase;
  uint32_t in = kPending;
  if (hm) {
    const int fh = __ffs(hm) - 1;
    const unsigned before = em & ((1u << fh) - 1u);
    const uint32_t v = __shfl_sync(gmask, bk.w, fh, kApplyGroup);
    if (!before && v < kPending) in = v;
  }
  uint32_t leaf = kNone;
  if (sl == 0) {
    if (in == kPending) in = root_get_or_create(M, rx, ry, rz);
    if (in != kNone) {
      const uint32_t ii = inner_index(M, lx, ly, lz);
      leaf = M.ichild[static_cast<size_t>(in) * M.isize + ii];
      if (leaf >= kPending) leaf = leaf_get_or_create(M, in, ii, lx, ly, lz);
    }
  }
  return __shfl_sync(gmask, leaf, 0, kApplyGroup);
}

// ---------------------------------------------------------------------------
// Mark: segments of cells, straight into the bitmap.
//
// The cube is aligned to roots (32 cells with the map's default bits), and a bit per
// root says that some segment may have marked cells there; the apply phase
// goes through the leaf blocks of those roots.
//
// A ray's cells k < kNearCells lie in the 7^3 leaves around the origin's, which
// every ray crosses: their bits are collected in shared memory and go to the
// bitmap once per block. The cells beyond are cut into segments of kSegCells;
// the winners kernel writes the list of segments, by number within each of its
// warps, so that the threads of a warp walk the same stretch of neighbouring
// rays. A thread collects the bits of a run of cells in one word (8 x 4 cells)
// and stores it with one OR that nothing waits for, and leaves out a cell that
// the thread before it is in at the same step. A cell's coordinates come from
// one fused multiply-add per axis:
//
//   n(k) = sign(d) floor((2 k |d| + m) / (2 m)) = sign(d) floor(k |d|/m + 1/2)
//
// and floor(fma(k, fl(d fl(1/m)), 1/2 + sign(d)/(4m))) is exactly that for k < 801
// and m <= 2047: the values (2 k |d| + m) / (2 m) are multiples of 1/(2m), so adding
// half of that keeps each 1/(4m) >= 1.22e-4 from the next integer, and the
// error (1.5 k 2^-24 of the slope, which is rounded twice, 2^-15 of the rounded sum, 2^-25 of
// the offset) stays below 1.03e-4; for d < 0 the value is 1 more than the floor of k d/m - 1/2 -
// 1/(4m), which is never an integer. (All d, m and k of the range: compared on a CPU.)
// Added to 2^23 + the origin's cell and rounded down, the float's low bits are the
// cell's coordinate: no conversion, sign or origin is left to apply, and the exponent's
// bits are a constant in the address. Longer rays divide in integers.
//
// What bounds it: instruction issue, and for clouds of one narrow direction (a
// depth frame) the ORs that meet in few words of L2. Kernel times on a GB300,
// L2 warm, against tasks of rays whose segments were found by a prefix and a
// search and walked with integer divisions (the form before): LiDAR 131k points,
// 9.3 M cells, 24 us (62); depth 307k points, 10.5 M cells, 59 us (105); room
// 60k points 18 us (30); 2k points 8.5 us (16). With the sign, the origin and the number
// of cells applied at each step (18.9 M instructions for the LiDAR scan, now 16.2 M) and
// no load ahead these were 25, 60, 18 and 9.9 us, and 64 maps in a batch 1.47 ms, now 1.33.
// Before the near cells got blocks of their
// own these were 28, 62, 20 and 14 us, of which without the far ORs 26, 39, 19
// and 13 us, and with every lane's cells ORed, neighbours' too, 36, 65, 21 us. Measured and not
// kept: rays sorted by direction and collected per block in shared memory, in
// a dense box of leaves (LiDAR 55 us, depth 60 us: scanning the box costs more
// than the ORs it saves), in a hash of leaves or behind a table (80-100 us: a
// first touch stalls the warp); a look at the word in L1 before the OR (45 us,
// 69 us: the look waits).
// ---------------------------------------------------------------------------
constexpr int kMarkThreads = 256;
constexpr int kMarkBlocksPerSM = 5;  // 48 registers; 6 (40, spilled): 3 % slower
constexpr int kNearNB = 3;                       // leaves on each side of the origin's
constexpr uint32_t kNearCells = 8 * kNearNB + 1;
constexpr uint32_t kNearW = 2 * kNearNB + 1;     // words of 8 x 4 cells: 7 x 14 x 56
constexpr uint32_t kNearWords = kNearW * 2 * kNearW * 8 * kNearW;
constexpr uint32_t kSegCells = 32;
constexpr uint32_t kSegBits = 5;                 // of a segment's number, beside its ray's
constexpr uint32_t kMaxSegRays = 1u << (32 - kSegBits);
constexpr uint32_t kMarkMaxRay = 32768;          // longer rays are walked on the tree (k_tail)
constexpr uint32_t kFmaMaxRay = 2047;
constexpr int kMaxCubeHalf = 24;                 // roots on each side: bit addresses in 32 bits
constexpr int kOpenCubeHalf = 16;                // of a scan whose rays may be of any length
static_assert((32 * kMaxCubeHalf + 1 - kNearCells + kSegCells - 1) / kSegCells <= 1u << kSegBits,
              "segments of the longest ray");
constexpr uint32_t kRootFlagWords =
    ((2 * kMaxCubeHalf + 1) * (2 * kMaxCubeHalf + 1) * (2 * kMaxCubeHalf + 1) + 31) / 32;

struct ScanCube {
  uint32_t* bits;   // S^3 leaf blocks of 16 words, x fastest; zero between scans
  uint32_t* roots;  // one bit per root (SR^3), set by the segments
  uint32_t* segs;   // segments: ray << kSegBits | number; nullptr: rays are walked whole
  uint32_t* tails;  // rays longer than kin; nullptr: there are none
  int x0, y0, z0;   // lowest cell (multiples of 32)
  uint32_t S, SR;   // leaves, roots per side
  uint32_t kin;     // cells k < kin of every ray lie in the cube
  uint32_t open;    // rays may be longer (k_tail walks the rest)
};

// The scan's dedup entries: its cells lie in the cube, of at most 49 * 32 cells a side,
// unless rays may leave it. What the table costs is its memory: 64 maps of 10-500 k points,
// whose tables of 128-bit entries are 300 MB (L2: 129 MB), clear 79 -> 39 us, endpoints 258
// -> 239, winners 262 -> 238; scans whose table lies in L2 within 2 %.
__host__ __device__ inline DedupKey dedup_key(const ScanCube& Q) {
  return DedupKey{Q.x0, Q.y0, Q.z0, Q.bits && !Q.open ? 1u : 0u};
}
__host__ __device__ inline uint32_t cube_root_words(const ScanCube& Q) {
  return (Q.SR * Q.SR * Q.SR + 31u) / 32u;
}
// Segments of the longest ray.
__host__ __device__ inline uint32_t max_segments(const ScanCube& Q) {
  return (Q.kin - kNearCells + kSegCells - 1) / kSegCells;
}
// Segments of a ray of len cells.
__device__ __forceinline__ uint32_t far_segments(const ScanCube& Q, uint32_t len) {
  const uint32_t m = min(len, Q.kin);
  return len < kMarkMaxRay && m > kNearCells ? (m - kNearCells + kSegCells - 1) / kSegCells : 0u;
}

// One thread's ray, as the marking needs it.
struct MarkRay {
  float sx, sy, sz;  // slopes d / m
  float fx, fy, fz;  // rounding offsets
  uint32_t m;        // cells to mark; 0: none
  int dx, dy, dz;
  uint32_t len;
};

__device__ __forceinline__ MarkRay mark_ray(const DMap& M, const ScanCube& Q, int4 e, int ox,
                                            int oy, int oz) {
  MarkRay r;
  r.dx = e.x - ox;
  r.dy = e.y - oy;
  r.dz = e.z - oz;
  r.len = max(static_cast<uint32_t>(abs(r.dx)),
              max(static_cast<uint32_t>(abs(r.dy)), static_cast<uint32_t>(abs(r.dz))));
  r.m = r.len < kMarkMaxRay ? min(r.len, Q.kin) : 0u;
  if (r.len >= min(kMarkMaxRay, Q.kin) && !Q.open)
    set_err(M, ERR_SCRATCH);  // outside the cube: cannot happen for scan rays
  const float inv = __frcp_rn(static_cast<float>(max(r.len, 1u)));
  r.sx = static_cast<float>(r.dx) * inv;
  r.sy = static_cast<float>(r.dy) * inv;
  r.sz = static_cast<float>(r.dz) * inv;
  r.fx = __fmaf_rn(r.dx < 0 ? -0.25f : 0.25f, inv, 0.5f);
  r.fy = __fmaf_rn(r.dy < 0 ? -0.25f : 0.25f, inv, 0.5f);
  r.fz = __fmaf_rn(r.dz < 0 ? -0.25f : 0.25f, inv, 0.5f);
  return r;
}

// The float 2^23 + n has the bits kFloatInt + n (0 <= n < 2^23).
constexpr uint32_t kFloatInt = 0x4B000000u;
__device__ __forceinline__ float float_int(int n) { return 8388608.0f + static_cast<float>(n); }
// floor of step f along an axis plus the integer that c = float_int() was made of.
__device__ __forceinline__ uint32_t step_bits(float f, float s, float off, float c) {
  return __float_as_uint(__fadd_rd(__fmaf_rn(f, s, off), c));
}

// Cell k of the ray, whose origin is the cell (qx, qy, qz).
template <bool LONG>
__device__ __forceinline__ void mark_cell(const MarkRay& r, uint32_t k, int qx, int qy, int qz,
                                          int& x, int& y, int& z) {
  if (LONG) {
    const uint32_t tm = 2u * r.len;
    auto step = [&](int d) {
      const int n = int((2u * k * uint32_t(abs(d)) + r.len) / tm);
      return d < 0 ? -n : n;
    };
    x = qx + step(r.dx);
    y = qy + step(r.dy);
    z = qz + step(r.dz);
  } else {
    const float f = static_cast<float>(k);
    x = int(step_bits(f, r.sx, r.fx, float_int(qx)) - kFloatInt);
    y = int(step_bits(f, r.sy, r.fy, float_int(qy)) - kFloatInt);
    z = int(step_bits(f, r.sz, r.fz, float_int(qz)) - kFloatInt);
  }
}

// Marks cells 0 .. n - 1 (1 <= n <= kNearCells) in the shared neighbourhood, where the
// origin is the cell (nx, ny, nz). The walk starts at cell rot: the lanes of a warp are
// apart then, where they would all OR the origin's word.
template <bool LONG>
__device__ __forceinline__ void mark_near(const MarkRay& r, uint32_t n, uint32_t rot, int nx,
                                          int ny, int nz, uint32_t* sm) {
  // the constant that the words of the steps' bits carry
  constexpr uint32_t kBias = LONG ? 0u
                                  : (kFloatInt >> 3) + kNearW * (kFloatInt >> 2) +
                                        2u * kNearW * kNearW * kFloatInt;
  const float cx = float_int(nx), cy = float_int(ny), cz = float_int(nz);
  uint32_t cur = 0, acc = 0;
  auto put = [&](uint32_t X, uint32_t Y, uint32_t Z) {
    const uint32_t w = (X >> 3) + kNearW * (Y >> 2) + 2 * kNearW * kNearW * Z;
    if (w != cur) {
      if (acc) atomicOr(sm + (cur - kBias), acc);
      acc = 0;
      cur = w;
    }
    acc |= 1u << (((X & 7u) + (Y << 3)) & 31u);
  };
  if (LONG) {
    uint32_t k = rot;
    for (uint32_t j = 0; j < n; ++j) {
      int x, y, z;
      mark_cell<true>(r, k, nx, ny, nz, x, y, z);
      put(uint32_t(x), uint32_t(y), uint32_t(z));
      k = k + 1 < n ? k + 1 : 0;
    }
  } else {
    const float last = static_cast<float>(n - 1);
    float f = static_cast<float>(rot);
    for (uint32_t j = 0; j < n; ++j) {
      put(step_bits(f, r.sx, r.fx, cx), step_bits(f, r.sy, r.fy, cy),
          step_bits(f, r.sz, r.fz, cz));
      f = f < last ? f + 1.0f : 0.0f;
    }
  }
  if (acc) atomicOr(sm + (cur - kBias), acc);
}

// Marks cells ka <= k < kb (ka < kb) of each thread's ray in the bitmap, where the origin
// is the cell (qx, qy, qz). All lanes of the warp, unless LONG.
template <bool LONG>
__device__ __forceinline__ void mark_far(const ScanCube& Q, const MarkRay& r, uint32_t ka,
                                         uint32_t kb, int qx, int qy, int qz) {
  // bit address: x + 8 y + 64 z, and for each axis the leaf's offset less the cells' own
  const uint32_t cy = 512u * Q.S - 64u, cz = 512u * Q.S * Q.S - 512u;
  auto address = [&](uint32_t x, uint32_t y, uint32_t z) {
    return x + 8u * y + 64u * z + (x >> 3) * 504u + (y >> 3) * cy + (z >> 3) * cz;
  };
  // the constant that the addresses of the steps' bits carry (a multiple of 32)
  const uint32_t bias = LONG ? 0u : 73u * kFloatInt + (kFloatInt >> 3) * (504u + cy + cz);
  uint32_t cur = 0, acc = 0;
  auto put = [&](uint32_t a) {
    if ((a ^ cur) & ~31u) {
      if (acc) red_or(Q.bits + ((cur - bias) >> 5), acc);
      acc = 0;
      cur = a;
    }
    acc |= 1u << (a & 31u);
  };
  if (LONG) {
    for (uint32_t k = ka; k < kb; ++k) {
      int x, y, z;
      mark_cell<true>(r, k, qx, qy, qz, x, y, z);
      put(address(uint32_t(x), uint32_t(y), uint32_t(z)));
    }
  } else {
    const float bx = float_int(qx), by = float_int(qy), bz = float_int(qz);
    const bool first = (threadIdx.x & 31) == 0;
    const uint32_t steps = min(__reduce_max_sync(0xffffffffu, kb - ka), kSegCells);
    // a thread whose segment is shorter than the warp's longest stays at its last cell
    const float last = static_cast<float>(kb - 1);
    float f = static_cast<float>(ka);
    for (uint32_t j = 0; j < steps; ++j) {
      const uint32_t a =
          address(step_bits(f, r.sx, r.fx, bx), step_bits(f, r.sy, r.fy, by),
                  step_bits(f, r.sz, r.fz, bz));
      const uint32_t before = __shfl_up_sync(0xffffffffu, a, 1);
      if (first || before != a) put(a);
      f = fminf(f + 1.0f, last);
    }
  }
  if (acc) red_or(Q.bits + ((cur - bias) >> 5), acc);
}

// The roots between two cells (at most 32 apart on each axis) into the block's root bits.
__device__ __forceinline__ void flag_roots(const ScanCube& Q, int ax, int ay, int az, int bx,
                                           int by, int bz, uint32_t* s_roots) {
  const int lx = min(ax, bx) >> 5, hx = max(ax, bx) >> 5, ly = min(ay, by) >> 5,
            hy = max(ay, by) >> 5, lz = min(az, bz) >> 5, hz = max(az, bz) >> 5;
  for (int z = lz; z <= hz; ++z)
    for (int y = ly; y <= hy; ++y)
      for (int x = lx; x <= hx; ++x) {
        const uint32_t i = uint32_t(x) + Q.SR * (uint32_t(y) + Q.SR * uint32_t(z));
        const uint32_t bit = 1u << (i & 31u);
        if (!(*reinterpret_cast<volatile uint32_t*>(s_roots + (i >> 5)) & bit))
          atomicOr(s_roots + (i >> 5), bit);
      }
}

struct MarkShared {
  uint32_t near[kNearWords];
  uint32_t roots[kRootFlagWords];
};

// A block's part of a scan's rays: the near cells of rays r, r + r_step, ... < r_end (r: the
// first thread's), and the segments s, s + s_step, ... < s_end of each warp's first lane (steps
// a multiple of kMarkThreads). All threads of a block of kMarkThreads. Adds the cells walked to
// `visited`.
__device__ __forceinline__ void mark_scan(const DMap& M, const ScanCube& Q,
                                          const int4* __restrict__ cast, uint32_t r,
                                          uint32_t r_end, uint32_t s, uint32_t s_end,
                                          uint32_t r_step, uint32_t s_step, int ox, int oy, int oz,
                                          MarkShared& S, uint32_t& visited) {
  const int qx = ox - Q.x0, qy = oy - Q.y0, qz = oz - Q.z0;  // the origin in the cube
  // the neighbourhood's lowest cell, from the origin
  const int wx = ((qx >> 3) - kNearNB) * 8 - qx, wy = ((qy >> 3) - kNearNB) * 8 - qy,
            wz = ((qz >> 3) - kNearNB) * 8 - qz;
  const uint32_t root_words = cube_root_words(Q);
  // a thread's next segment and its ray are loaded ahead of the one it walks; threads past
  // the end go over the last segment again
  auto segment = [&](uint32_t i) { return Q.segs[min(i + (threadIdx.x & 31), s_end - 1)]; };
  uint32_t seg = 0;
  int4 e = make_int4(0, 0, 0, 0);
  if (s < s_end) {
    seg = segment(s);
    e = cast[seg >> kSegBits];
  }
  if (r < r_end)
    for (uint32_t t = threadIdx.x; t < kNearWords; t += kMarkThreads) S.near[t] = 0u;
  for (uint32_t t = threadIdx.x; t < root_words; t += kMarkThreads) S.roots[t] = 0u;
  __syncthreads();
  for (uint32_t i = r + threadIdx.x; i < r_end; i += r_step) {
    const MarkRay q = mark_ray(M, Q, cast[i], ox, oy, oz);
    if (!q.m) continue;
    visited += q.m;
    const uint32_t n = min(q.m, kNearCells);
    const uint32_t rot = (threadIdx.x & 31) * n >> 5;
    if (q.len > kFmaMaxRay)
      mark_near<true>(q, n, rot, -wx, -wy, -wz, S.near);
    else
      mark_near<false>(q, n, rot, -wx, -wy, -wz, S.near);
    if (Q.segs) continue;
    for (uint32_t ka = kNearCells; ka < q.m; ka += kSegCells) {
      const uint32_t kb = min(ka + kSegCells, q.m);
      int ax, ay, az, bx, by, bz;
      mark_cell<true>(q, ka, qx, qy, qz, ax, ay, az);
      mark_cell<true>(q, kb - 1, qx, qy, qz, bx, by, bz);
      mark_far<true>(Q, q, ka, kb, qx, qy, qz);
      flag_roots(Q, ax, ay, az, bx, by, bz, S.roots);
    }
  }
  while (s < s_end) {
    const MarkRay q = mark_ray(M, Q, e, ox, oy, oz);
    const uint32_t ka = kNearCells + (seg & ((1u << kSegBits) - 1u)) * kSegCells;
    const uint32_t kb = min(ka + kSegCells, q.m);
    s += s_step;
    if (s < s_end) {
      seg = segment(s);
      e = cast[seg >> kSegBits];
    }
    int ax, ay, az, bx, by, bz;
    if (__any_sync(0xffffffffu, q.len > kFmaMaxRay)) {
      mark_cell<true>(q, ka, qx, qy, qz, ax, ay, az);
      mark_cell<true>(q, kb - 1, qx, qy, qz, bx, by, bz);
      mark_far<true>(Q, q, ka, kb, qx, qy, qz);
    } else {
      mark_cell<false>(q, ka, qx, qy, qz, ax, ay, az);
      mark_cell<false>(q, kb - 1, qx, qy, qz, bx, by, bz);
      mark_far<false>(Q, q, ka, kb, qx, qy, qz);
    }
    flag_roots(Q, ax, ay, az, bx, by, bz, S.roots);
  }
  __syncthreads();
  if (r < r_end) {
    const uint32_t lx = uint32_t((qx + wx) >> 3), ly = uint32_t((qy + wy) >> 3),
                   lz = uint32_t((qz + wz) >> 3);
    for (uint32_t t = threadIdx.x; t < kNearWords; t += kMarkThreads) {
      const uint32_t v = S.near[t];
      if (!v) continue;
      const uint32_t x = t % kNearW, y = t / kNearW % (2 * kNearW), z = t / (2 * kNearW * kNearW);
      const uint32_t bx = lx + x, by = ly + (y >> 1), bz = lz + (z >> 3);
      red_or(Q.bits + (bx + Q.S * (by + Q.S * bz)) * 16u + (y & 1u) + ((z & 7u) << 1), v);
      const uint32_t i = (bx >> 2) + Q.SR * ((by >> 2) + Q.SR * (bz >> 2));
      const uint32_t bit = 1u << (i & 31u);
      if (!(*reinterpret_cast<volatile uint32_t*>(S.roots + (i >> 5)) & bit))
        atomicOr(S.roots + (i >> 5), bit);
    }
    __syncthreads();
  }
  for (uint32_t t = threadIdx.x; t < root_words; t += kMarkThreads)
    if (S.roots[t]) red_or(Q.roots + t, S.roots[t]);
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Apply, a warp per row of four leaf blocks of a root.
//
// Four groups of eight lanes each read a block's bits and find (or create) its leaf;
// the rows of 8 cells (one 32-byte sector) that have marked cells go on a
// list in shared memory, and then each lane updates one listed row at a time.
//
// What bounds it: the chain bits -> root bucket -> child word -> cells -> stores, and
// DRAM sectors where few cells of a leaf are marked. LiDAR 131k points, 4.0 M
// cells in 18 k leaves: 24 us (37 with eight lanes for each leaf of a list, a
// lane 64 cells and two rounds of eight loads); 8 maps of few points, 225 k leaves
// with 29 cells each: 82 us (107 with the whole warp on one leaf's 64 rows at a
// time: most rows have no marked cell). One scan cannot fill the chip and loads two rows
// at a time, at four blocks per SM (2k points 12.1 us against 13.8, room 11.9 against
// 13.4); a tick can, and takes one at eight blocks per SM (64 maps: 1.28 ms; two at
// a time 1.34).
// ---------------------------------------------------------------------------
constexpr int kApplyWarps = 8;
struct ApplyShared {
  uint2 rows[kApplyWarps][256];  // (leaf slot * 64 + row) << 8 | cells, low word first
};

// Updates the cells c[0..3] whose bits are set in nib; returns the cells that
// were zero (to turn on), sets `changed`.
__device__ __forceinline__ uint32_t miss_run(int4& v, uint32_t nib, int32_t u, int32_t miss,
                                             int32_t cmin, bool& changed, uint32_t& updated) {
  int32_t* c = reinterpret_cast<int32_t*>(&v);
  uint32_t fresh = 0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    if (!((nib >> t) & 1u)) continue;
    const int32_t old = c[t];
    if (cell_id(old) != u) {
      c[t] = cell_pack(max(wrap_add(cell_prob(old), miss), cmin), u);
      changed = true;
      ++updated;
    }
    if (old == 0) fresh |= 1u << t;
  }
  return fresh;
}

// Blocks 4 rx .. 4 rx + 3 of the row (by, bz), in leaves of the cube. ROWS: listed rows
// that a lane loads before it updates them.
template <int ROWS>
__device__ __forceinline__ void apply_row(const DMap& M, const ScanCube& Q, uint32_t rx,
                                          uint32_t by, uint32_t bz, int32_t u, int32_t miss,
                                          int32_t cmin, uint2* list, uint32_t& updated) {
  const unsigned lane = threadIdx.x & 31, sl = lane & 7u, gbase = lane & 24u;
  const uint32_t bx = 4u * rx + (lane >> 3);
  uint2* wp = reinterpret_cast<uint2*>(Q.bits + size_t(bx + Q.S * (by + Q.S * bz)) * 16u) + sl;
  const uint2 wv = *wp;
  const unsigned any = __ballot_sync(0xffffffffu, (wv.x | wv.y) != 0u);
  if (!any) return;
  uint32_t leaf = kNone;
  if ((any >> gbase) & 0xFFu) {
    leaf = apply_leaf_slot(M, Q.x0 + 8 * int(bx), Q.y0 + 8 * int(by), Q.z0 + 8 * int(bz), sl,
                           gbase, 0xFFu << gbase);
    if (wv.x | wv.y) *wp = make_uint2(0u, 0u);
  }
  __syncwarp();
  // a lane's eight bytes are the rows 8 sl .. 8 sl + 7 of its block (none without
  // a leaf: the pool is full and the scan is re-run)
  const uint2 rows = leaf == kNone ? make_uint2(0u, 0u) : wv;
  auto marked = [](uint32_t v) { return (((v & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | v) & 0x80808080u; };
  const uint32_t mx = marked(rows.x), my = marked(rows.y);
  const uint32_t cnt = __popc(mx) + __popc(my);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= unsigned(o)) incl += v;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  uint32_t k = incl - cnt;
  const unsigned long long row0 = static_cast<unsigned long long>(leaf) * 64u + 8u * sl;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t w = h ? rows.y : rows.x;
    for (uint32_t m = h ? my : mx; m; m &= m - 1u) {
      const uint32_t j = uint32_t(__ffs(m) - 1) >> 3;
      const unsigned long long e = ((row0 + 4u * h + j) << 8) | ((w >> (8u * j)) & 0xFFu);
      list[k++] = make_uint2(uint32_t(e), uint32_t(e >> 32));
    }
  }
  __syncwarp();
  for (uint32_t i = lane; i < total; i += 32 * ROWS) {
    uint2 e[ROWS];
    int4 v[ROWS][2];
    auto row_of = [](uint2 x) { return (static_cast<unsigned long long>(x.y) << 24) | (x.x >> 8); };
#pragma unroll
    for (int p = 0; p < ROWS; ++p) {
      e[p] = i + 32 * p < total ? list[i + 32 * p] : make_uint2(0u, 0u);
      const int4* c = reinterpret_cast<const int4*>(M.ldata) + 2 * row_of(e[p]);
      if (e[p].x & 0xFu) v[p][0] = c[0];
      if (e[p].x & 0xF0u) v[p][1] = c[1];
    }
#pragma unroll
    for (int p = 0; p < ROWS; ++p) {
      const unsigned long long row = row_of(e[p]);
      const uint32_t cells = e[p].x & 0xFFu;
      int4* c = reinterpret_cast<int4*>(M.ldata) + 2 * row;
      uint32_t fresh = 0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t nib = (cells >> (4 * q)) & 0xFu;
        if (!nib) continue;
        bool changed = false;
        fresh |= miss_run(v[p][q], nib, u, miss, cmin, changed, updated) << (4 * q);
        if (changed) c[q] = v[p][q];
      }
      // the row's mask byte, in its 32-bit word
      if (fresh)
        red_or(reinterpret_cast<uint32_t*>(M.lmask) + (row >> 2), fresh << (8u * (row & 3u)));
    }
  }
  __syncwarp();
}

// The marked roots before each word of Q.roots, into pre (cube_root_words(Q) shared words);
// returns their number. All threads of the block.
__device__ __forceinline__ uint32_t apply_roots(const ScanCube& Q, uint32_t* pre,
                                                uint32_t* warp_sums) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t words = cube_root_words(Q), total_bits = Q.SR * Q.SR * Q.SR;
  const uint32_t per = (words + blockDim.x - 1) / blockDim.x, w0 = threadIdx.x * per;
  auto count = [&](uint32_t w) {
    uint32_t v = Q.roots[w];
    if (w == words - 1 && (total_bits & 31u)) v &= (1u << (total_bits & 31u)) - 1u;
    return static_cast<uint32_t>(__popc(v));
  };
  uint32_t c = 0;
  for (uint32_t w = w0; w < min(w0 + per, words); ++w) c += count(w);
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= unsigned(o)) incl += v;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  uint32_t before = incl - c, all = 0;
  for (unsigned k = 0; k < nw; ++k) {
    if (k < warp) before += warp_sums[k];
    all += warp_sums[k];
  }
  for (uint32_t w = w0; w < min(w0 + per, words); ++w) {
    pre[w] = before;
    before += count(w);
  }
  __syncthreads();
  return all;
}

// All of a scan's marked cells: warps `warp`, `warp` + n_warps, ... of 16 rows for each
// marked root.
__device__ __forceinline__ void apply_scan(const DMap& M, const ScanCube& Q, uint32_t n_roots,
                                           const uint32_t* pre, uint32_t warp, uint32_t n_warps,
                                           int32_t u, int32_t miss, int32_t cmin, uint2* list,
                                           uint32_t& updated) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t words = cube_root_words(Q);
  for (uint32_t t = warp; t < 16u * n_roots; t += n_warps) {
    const uint32_t k = t >> 4;
    uint32_t lo = 0, hi = words;  // last word with at most k roots before it
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (pre[mid] <= k) lo = mid; else hi = mid;
    }
    const uint32_t v = Q.roots[lo];  // its (k - pre[lo])-th set bit
    const uint32_t i = 32u * lo + uint32_t(__ffs(__ballot_sync(
        0xffffffffu, ((v >> lane) & 1u) && uint32_t(__popc(v & ((1u << lane) - 1u))) == k - pre[lo])) - 1);
    const uint32_t rz = i / (Q.SR * Q.SR), ry = (i - rz * Q.SR * Q.SR) / Q.SR,
                   rx = i - (rz * Q.SR + ry) * Q.SR;
    apply_row<2>(M, Q, rx, 4u * ry + (t & 3u), 4u * rz + ((t >> 2) & 3u), u, miss, cmin, list,
              updated);
  }
}

// The lowest-index point of each endpoint cell decides and applies
// (winner_apply) and, if its ray is cast, joins the ray list.
// One block-wide atomic each for the ray list, the point count and the ray
// lengths (a per-warp atomic on three shared counters serialised in L2). The block waits
// for three of them: a lane of the first warp issues each, where one thread after the other
// took 2k points 10.0 us, LiDAR 12.5, depth 13.1, room 8.0 and now 8.5, 11.3, 11.4, 7.5.
struct WinnersShared {
  uint32_t cnt[8], pts[8], seg[8], tail[8];  // per warp; then what the warps before it have
  unsigned long long len[8];
  uint32_t base[3];  // the block's first place on the lists of rays, segments, tails
};
// All threads of a block of 256, for points i of one scan (i >= n: none).
__device__ __forceinline__ void winners_block(const DMap& M, const int4* __restrict__ ep,
                                              uint32_t n, uint32_t i,
                                              const uint4* __restrict__ tab, uint32_t tmask,
                                              int ox, int oy, int oz, int32_t u, const Opts& o,
                                              int4* __restrict__ cast, uint32_t cast_cap,
                                              const ScanCube& Q, WinnersShared& S) {
  bool add = false;
  int4 e = make_int4(0, 0, 0, EP_SKIP);
  if (i < n) {
    e = ep[i];
    if (e.w == EP_HIT || e.w == EP_MISS) {
      // the root's bucket is on its way while the table's is
      const int32_t rm = root_mask(M);
      const uint32_t in = root_probe_fast(M, e.x & rm, e.y & rm, e.z & rm);
      if (dedup_lookup(tab, tmask, e.x, e.y, e.z, dedup_key(Q)) == i) add = winner_apply(M, e, in, u, o);
    }
  }
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned valid = __ballot_sync(0xffffffffu, i < n && e.w != EP_SKIP);
  const unsigned am = __ballot_sync(0xffffffffu, add);
  const uint32_t len = add ? chebyshev(ox, oy, oz, e.x, e.y, e.z) : 0u;
  const unsigned long long wlen = __reduce_add_sync(0xffffffffu, len >> 16) * 65536ull +
                                  __reduce_add_sync(0xffffffffu, len & 0xFFFFu);
  // with a cube, the ray's segments go on the scan's list of segments
  const uint32_t nseg = add && Q.segs ? far_segments(Q, len) : 0u;
  uint32_t seg = nseg;
#pragma unroll
  for (int o2 = 1; o2 < 32; o2 <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, seg, o2);
    if (lane >= unsigned(o2)) seg += v;
  }
  if (lane == 31) S.seg[wid] = seg;
  // and the rays that leave the cube on the list of those
  const unsigned tails =
      __ballot_sync(0xffffffffu, add && Q.tails && len > Q.kin);
  if (lane == 0) {
    S.cnt[wid] = __popc(am);
    S.tail[wid] = __popc(tails);
    S.pts[wid] = __popc(valid);
    S.len[wid] = wlen;
  }
  __syncthreads();
  if (wid == 0) {
    // lane w < 8: warp w's counts
    const bool w8 = lane < 8;
    uint32_t c = w8 ? S.cnt[lane] : 0u, g = w8 ? S.seg[lane] : 0u, t = w8 ? S.tail[lane] : 0u;
    const uint32_t c0 = c, g0 = g, t0 = t;
#pragma unroll
    for (int o2 = 1; o2 < 8; o2 <<= 1) {
      const uint32_t a = __shfl_up_sync(0xffffffffu, c, o2), b = __shfl_up_sync(0xffffffffu, g, o2),
                     d = __shfl_up_sync(0xffffffffu, t, o2);
      if (lane >= unsigned(o2)) {
        c += a;
        g += b;
        t += d;
      }
    }
    const uint32_t pts = __reduce_add_sync(0xffffffffu, w8 ? S.pts[lane] : 0u);
    unsigned long long tl = w8 ? S.len[lane] : 0ull;
#pragma unroll
    for (int o2 = 4; o2 > 0; o2 >>= 1) tl += __shfl_down_sync(0xffffffffu, tl, o2);
    const uint32_t tot = __shfl_sync(0xffffffffu, c, 7), segs = __shfl_sync(0xffffffffu, g, 7),
                   tails_n = __shfl_sync(0xffffffffu, t, 7);
    // a lane for each of the counters: their atomics are under way together
    if (lane < 3) {
      const uint32_t v = lane == 0 ? tot : lane == 1 ? segs : tails_n;
      S.base[lane] =
          v ? atomicAdd(M.ctr + (lane == 0 ? C_CAST : lane == 1 ? C_SEGS : C_TAILS), v) : 0u;
    }
    unsigned long long* st = reinterpret_cast<unsigned long long*>(M.ctr + C_STATS);
    if (lane == 0 && tl) atomicAdd(st + S_RAY_LEN, tl);
    if (lane == 1 && pts) atomicAdd(st + S_POINTS, static_cast<unsigned long long>(pts));
    if (w8) {
      S.cnt[lane] = c - c0;
      S.seg[lane] = g - g0;
      S.tail[lane] = t - t0;
    }
  }
  __syncthreads();
  uint32_t ray = 0;
  if (add) {
    const uint32_t k = S.base[0] + S.cnt[wid] + __popc(am & ((1u << lane) - 1));
    if (k < cast_cap)
      cast[k] = e;
    else
      set_err(M, ERR_SCRATCH);
    ray = k;
    if ((tails >> lane) & 1u)
      Q.tails[S.base[2] + S.tail[wid] + __popc(tails & ((1u << lane) - 1u))] = k;
  }
  // the warp's segments, number by number: neighbouring rays' segments lie side by side
  uint32_t at = S.base[1] + S.seg[wid];
  for (uint32_t j = 0;; ++j) {
    const unsigned has = __ballot_sync(0xffffffffu, nseg > j);
    if (!has) break;
    if (nseg > j) Q.segs[at + __popc(has & ((1u << lane) - 1u))] = (ray << kSegBits) | j;
    at += __popc(has);
  }
}

// An endpoint (e.w == EP_SKIP: none) of point i into the dedup table. Neighbouring points
// often share an endpoint cell: within a warp only the lowest lane (lowest index) of each cell
// enters the table; the others can never be the cell's lowest index and are
// marked EP_DUP. All lanes of a warp, whose points are consecutive.
__device__ __forceinline__ void endpoint_enter(const DMap& M, int4& e, uint32_t i, uint4* tab,
                                               uint32_t tmask, const DedupKey& K) {
  const unsigned vm = __ballot_sync(0xffffffffu, e.w != EP_SKIP);
  if (e.w == EP_SKIP) return;
  const unsigned same = __match_any_sync(vm, e.x) & __match_any_sync(vm, e.y) &
                        __match_any_sync(vm, e.z);
  if (same & ((1u << (threadIdx.x & 31)) - 1u))
    e.w = EP_DUP;
  else
    dedup_min_insert(tab, tmask, e.x, e.y, e.z, i, M, K);
}

// The parts of rays that the cube does not hold (cells k >= kin; all cells of a
// ray of kMarkMaxRay cells or more), walked on the tree. A warp takes a piece of a
// ray, of at least two steps of 32 cells: a walk is a chain of dependent loads, about 4 us a
// step, and the rays that go far are few (29 k points at 0.05 m with returns to 100 m, in 32
// pieces: 16 us; with eight rays per warp and pieces of 256 cells 125 us; the whole scan
// walked by k_rays 330 us, against 17 for k_mark, 25 for k_apply_rays and this). Where they
// are many a piece costs more than it gives -- finding its place divides in 64 bits, and
// most pieces of a ray that is not much longer than the cube are empty: about four pieces
// per warp then, down to whole rays (whole scans of 131 k points whose rays all have 800
// cells: 0.83 ms, 2.8 in 32 pieces, 0.98 walked by k_rays; of 30 k with a fifth of such
// rays 163 us, 234, 197; of 2 k with rays of 3000-8000 cells 365, 373, 620).
constexpr uint32_t kTailPieces = 32;
__device__ __forceinline__ void tail_rays(const DMap& M, const ScanCube& Q,
                                          const int4* __restrict__ cast, uint32_t cast_cap,
                                          uint64_t warp, uint64_t n_warps, int ox, int oy, int oz,
                                          int32_t u, int32_t miss, int32_t cmin,
                                          uint32_t& visited, uint32_t& updated) {
  const uint32_t n = min(ld_volatile(M.ctr + C_TAILS), cast_cap);
  if (!n) return;
  const unsigned lane = threadIdx.x & 31;
  const uint32_t pieces = uint32_t(max(min(4 * n_warps / n, uint64_t(kTailPieces)), uint64_t(1)));
  for (uint64_t t = warp; t < uint64_t(n) * pieces; t += n_warps) {
    const uint32_t i = uint32_t(t / pieces), j = uint32_t(t % pieces);
    const int4 e = cast[Q.tails[i]];
    const uint32_t m = chebyshev(ox, oy, oz, e.x, e.y, e.z);
    if (m >= kMaxRayCells) {
      if (lane == 0) set_err(M, ERR_RAY_TOO_LONG);
      continue;
    }
    const uint32_t from = m < kMarkMaxRay ? Q.kin : 0u;
    const uint32_t piece = max(64u, (((m - from) / pieces + 32u) & ~31u));
    if (from + j * piece < m)
      walk_ray<32>(M, e, ox, oy, oz, u, miss, cmin, lane, 0u, 0xffffffffu, visited, updated,
                   nullptr, from + j * piece, from + (j + 1) * piece);
  }
}
// A warp's counts of walked and updated cells into the scan's statistics.
__device__ __forceinline__ void tail_count(const DMap& M, uint32_t visited, uint32_t updated) {
  visited = __reduce_add_sync(0xffffffffu, visited);
  updated = __reduce_add_sync(0xffffffffu, updated);
  if ((threadIdx.x & 31) == 0 && visited) {
    unsigned long long* st = reinterpret_cast<unsigned long long*>(M.ctr + C_STATS);
    atomicAdd(st + S_VISITED, static_cast<unsigned long long>(visited));
    atomicAdd(st + S_UPDATED, static_cast<unsigned long long>(updated));
  }
}

}  // namespace bxg
