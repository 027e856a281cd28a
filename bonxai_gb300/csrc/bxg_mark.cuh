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
//          getLeafIndex, x fastest). A block takes a run of rays and cuts
//          them into segments that its threads walk (closed-form Bresenham
//          start, then the RayIterator step): the cells near the origin,
//          which every ray crosses, in a neighbourhood of leaves kept in
//          shared memory and ORed into the bitmap once per block task; the
//          rest in segments of kMarkSeg cells whose bits are ORed into the
//          bitmap one word at a time, fire-and-forget. A block's first OR
//          also sets the block's bit in a per-block "touched" bitmap.
//   list   The touched bitmap is turned into the scan's list of marked blocks
//          and cleared.
//   apply  One group of 8 lanes per listed block: a cooperative probe of the
//          root hash (8 buckets per step), the leaf get-or-create (topology:
//          once per leaf, not once per ray crossing), then the miss update of
//          the marked cells with vector loads and stores, the mask bits of
//          cells turned on, and the block cleared for the next scan.
//
// This is the two-phase insert (topology, then values) over deduplicated
// coordinates: the bitmap is the deduplication. The result equals the per-ray
// walk's bit for bit; the cube, its bits and its touched bits are scratch that
// is all zero between scans.
#pragma once

#include "bxg_scan.cuh"

namespace bxg {

constexpr uint32_t kMarkSeg = 16;  // cells of a segment beyond the neighbourhood
// Shared-memory neighbourhood of the origin: the leaves within NB of the
// origin's leaf, (2 NB + 1)^3 blocks of 16 words. NB = 3 (21.4 KiB) for the
// per-scan kernel's 1024-thread blocks, NB = 2 (7.8 KiB) in the batched tick,
// whose 256-thread blocks also hold the tick's scan table. A ray's cell k
// (k cells from the origin along the major axis) lies within Chebyshev
// distance k of the origin cell, so cells k <= 8 NB are always inside the
// neighbourhood; they form each ray's first kMarkLocalParts segments.
constexpr int kMarkNB = 3;
constexpr uint32_t kMarkLocalParts = 2;
__host__ __device__ constexpr int mark_smem_words(int nb) {
  return (2 * nb + 1) * (2 * nb + 1) * (2 * nb + 1) * 16;
}
constexpr int kMarkSmemWords = mark_smem_words(kMarkNB);
constexpr int kApplyGroup = 8;  // lanes per listed block in apply (4 blocks per warp)

// The bitmap of one scan. Block b = bx + S*(by + S*bz) covers the cells
// x0 + 8*bx .. x0 + 8*bx + 7 (likewise y, z).
//
// The touched bitmap has one bit per block at a scattered position, bit
// (b * kTouchMul) mod 2^k (2^k >= S^3; odd multiplier, so a permutation whose
// inverse multiplies by kTouchInv): with bit b, one 32-byte sector held the
// flags of 256 blocks in a row, and every ray along that row set them through
// the same sector of L2 (those ORs serialised: 100 us of a 110 us LiDAR mark).
struct RayCube {
  uint32_t* bits;     // S^3 * 16 words
  uint32_t* touched;  // (tmask + 1) bits: some bit of the block is set
  uint32_t* list;     // listed blocks
  uint32_t* count;    // entries on the list
  int x0, y0, z0;     // lowest cell of the cube (multiples of 8)
  uint32_t S;         // leaves per side
  uint32_t cap;       // list capacity (S^3)
  uint32_t tmask;     // 2^k - 1 with 2^k >= max(S^3, 32)
};

constexpr uint32_t kTouchMul = 0x9E3779B1u;
constexpr uint32_t kTouchInv = 0x0E8B2F51u;  // kTouchMul * kTouchInv == 1 mod 2^32
static_assert(kTouchMul * kTouchInv == 1u, "inverse of the touched-bit permutation");

__host__ __device__ inline uint32_t cube_touched_words(const RayCube& Q) {
  return (Q.tmask + 1u) / 32u;
}
// 2^k - 1 for the smallest 2^k >= max(S^3, 32)
__host__ __device__ inline uint32_t cube_touched_mask(uint32_t S) {
  uint32_t p = 32u;
  while (p < S * S * S) p <<= 1;
  return p - 1u;
}
__device__ __forceinline__ void touch_block(const RayCube& Q, uint32_t b) {
  const uint32_t t = (b * kTouchMul) & Q.tmask;
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(
                   __cvta_generic_to_global(Q.touched + (t >> 5))),
               "r"(1u << (t & 31))
               : "memory");
}

// Fire-and-forget ORs and AND into global memory. The pointers may reach the
// code as generic addresses (the batched tick keeps its scan table, with the
// bitmap and pool pointers, in shared memory), and an atomicOr on a generic
// address compiles to an atomic that returns its old value, which the warp
// then waits for; these always issue the reduction form.
__device__ __forceinline__ void red_or(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
               "r"(v)
               : "memory");
}
__device__ __forceinline__ void red_or64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.or.b64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
               "l"(v)
               : "memory");
}

// The rays of one block task, in shared memory, T at a time: each ray's
// offset from the origin (dx, dy, dz), its length m (cells before the end
// cell), and the first of its segments beyond the neighbourhood. Also a
// direct-mapped cache of blocks whose touched bit the block task has set: a
// hit skips the OR (most blocks are crossed by many of a task's rays).
constexpr uint32_t kTouchCache = 2048;
template <int T>
struct MarkRays {
  uint2 d[T];  // (dx, dy) and (dz, m) as 16-bit halves
  uint32_t start[T];
  uint32_t wsum[32];
  uint32_t n_far;  // segments beyond the neighbourhood, all rays of the batch
  uint32_t touched[kTouchCache];
};

// Walks cells k0 .. k1 - 1 of the ray from cube cell (qx, qy, qz) with offset
// (dx, dy, dz) and length m: the closed-form state at k0 (n_b = floor((2 k0
// d_b + m) / 2m), r_b the remainder, as in bxg_device.cuh), then
// RayIterator's step. `word` maps a cell to its word and `flush` stores a
// word's collected bits.
template <class Word, class Flush>
__device__ __forceinline__ void mark_walk(int qx, int qy, int qz, int dx, int dy, int dz,
                                          uint32_t m, uint32_t k0, uint32_t k1, Word&& word,
                                          Flush&& flush) {
  const uint32_t ax = uint32_t(abs(dx)), ay = uint32_t(abs(dy)), az = uint32_t(abs(dz));
  const uint32_t tm = 2u * m;
  const float rtm = __frcp_rn(float(tm));
  uint32_t nx, rx, ny, ry, nz, rz;
  divmod_small(2u * k0 * ax + m, tm, rtm, nx, rx);
  divmod_small(2u * k0 * ay + m, tm, rtm, ny, ry);
  divmod_small(2u * k0 * az + m, tm, rtm, nz, rz);
  const int sx = dx < 0 ? -1 : 1, sy = dy < 0 ? -1 : 1, sz = dz < 0 ? -1 : 1;
  int cx = qx + sx * int(nx), cy = qy + sy * int(ny), cz = qz + sz * int(nz);
  const uint32_t ax2 = 2u * ax, ay2 = 2u * ay, az2 = 2u * az;
  uint32_t cur = word(cx, cy, cz), acc = 0;
  for (uint32_t k = k0; k < k1; ++k) {
    const uint32_t w = word(cx, cy, cz);
    if (w != cur) {
      flush(cur, acc);
      cur = w;
      acc = 0;
    }
    acc |= 1u << (uint32_t(cx & 7) | (uint32_t(cy & 3) << 3));
    rx += ax2;
    if (rx >= tm) {
      rx -= tm;
      cx += sx;
    }
    ry += ay2;
    if (ry >= tm) {
      ry -= tm;
      cy += sy;
    }
    rz += az2;
    if (rz >= tm) {
      rz -= tm;
      cz += sz;
    }
  }
  flush(cur, acc);
}

// The block marks rays [r0, r1) of one scan from origin cell (ox, oy, oz)
// (blockDim.x == T). sm (mark_smem_words(NB) words) is zero on entry and on
// return; every thread of the block calls this with the same arguments. Adds
// the cells walked to `visited`. The cube must reach at least NB + 1 leaves
// beyond the origin's leaf on every side; a ray whose end cell lies outside
// the cube sets ERR_SCRATCH and is not walked.
template <int NB, int T>
__device__ __forceinline__ void mark_rays_block(const DMap& M, const RayCube& Q,
                                                const int4* __restrict__ cast, uint32_t r0,
                                                uint32_t r1, int ox, int oy, int oz,
                                                uint32_t* sm, MarkRays<T>& R,
                                                uint32_t& visited) {
  constexpr int NS = 2 * NB + 1;
  constexpr uint32_t kNear = 8u * NB + 1u;  // cells 0 .. kNear - 1 are in the neighbourhood
  constexpr uint32_t kPart = (kNear + kMarkLocalParts - 1) / kMarkLocalParts;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int qox = ox - Q.x0, qoy = oy - Q.y0, qoz = oz - Q.z0;  // origin, cube cells
  const int side = int(Q.S) * 8;
  // the neighbourhood's lowest cell (cube cells) and its leaf
  const int nlx = (qox >> 3) - NB, nly = (qoy >> 3) - NB, nlz = (qoz >> 3) - NB;
  const int nbx = 8 * nlx, nby = 8 * nly, nbz = 8 * nlz;
  const uint32_t S = Q.S, SS = Q.S * Q.S;
  uint32_t last_b = kNone;  // last block this thread set the touched bit of
  auto near_word = [&](int cx, int cy, int cz) -> uint32_t {
    const uint32_t ux = uint32_t(cx - nbx), uy = uint32_t(cy - nby), uz = uint32_t(cz - nbz);
    return (((uz >> 3) * NS + (uy >> 3)) * NS + (ux >> 3)) * 16u + ((uy >> 2) & 1u) +
           ((uz & 7u) << 1);
  };
  // Every ray starts at the origin, so lanes walking near segments flush the
  // same few words at once: the lanes flushing one word OR their bits
  // together and one of them issues the shared atomic (same-address shared
  // atomics are serialised).
  auto near_flush = [&](uint32_t w, uint32_t acc) {
    const unsigned grp = __match_any_sync(__activemask(), w);
    const uint32_t v = __reduce_or_sync(grp, acc);
    if (lane == unsigned(__ffs(grp) - 1)) atomicOr(sm + w, v);
  };
  auto far_word = [&](int cx, int cy, int cz) -> uint32_t {
    return ((uint32_t(cx) >> 3) + S * (uint32_t(cy) >> 3) + SS * (uint32_t(cz) >> 3)) * 16u +
           ((uint32_t(cy) >> 2) & 1u) + ((uint32_t(cz) & 7u) << 1);
  };
  auto far_flush = [&](uint32_t w, uint32_t acc) {
    red_or(Q.bits + w, acc);
    const uint32_t b = w >> 4;
    if (b != last_b) {
      last_b = b;
      uint32_t& c = R.touched[(b * kTouchMul) >> 21];
      if (c != b) {  // races between threads only repeat an OR
        c = b;
        touch_block(Q, b);
      }
    }
  };
  for (uint32_t t = threadIdx.x; t < kTouchCache; t += T) R.touched[t] = kNone;
  for (uint32_t base = r0; base < r1; base += T) {
    const uint32_t nr = min(uint32_t(T), r1 - base);
    uint32_t nfar = 0;
    if (threadIdx.x < nr) {
      const int4 e = cast[base + threadIdx.x];
      int dx = e.x - ox, dy = e.y - oy, dz = e.z - oz;
      uint32_t m = uint32_t(max(abs(dx), max(abs(dy), abs(dz))));
      if (uint32_t(e.x - Q.x0) >= uint32_t(side) || uint32_t(e.y - Q.y0) >= uint32_t(side) ||
          uint32_t(e.z - Q.z0) >= uint32_t(side)) {
        set_err(M, ERR_SCRATCH);  // outside the cube: cannot happen for scan rays
        dx = dy = dz = 0;
        m = 0;
      }
      nfar = m > kNear ? (m - kNear + kMarkSeg - 1) / kMarkSeg : 0u;
      R.d[threadIdx.x] = make_uint2((uint32_t(dx) & 0xFFFFu) | (uint32_t(dy) << 16),
                                    (uint32_t(dz) & 0xFFFFu) | (m << 16));
    }
    // exclusive prefix of the far segment counts over the batch
    uint32_t incl = nfar;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= unsigned(o)) incl += v;
    }
    if (lane == 31) R.wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const uint32_t x0 = lane < T / 32 ? R.wsum[lane] : 0u;
      uint32_t x = x0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= unsigned(o)) x += v;
      }
      if (lane < T / 32) R.wsum[lane] = x - x0;
      if (lane == 31) R.n_far = x;
    }
    __syncthreads();
    R.start[threadIdx.x] = incl - nfar + R.wsum[warp];
    __syncthreads();
    // segments: kMarkLocalParts per ray near the origin, then the far ones
    const uint32_t n_near = nr * kMarkLocalParts;
    const uint32_t total = n_near + R.n_far;
    for (uint32_t j = threadIdx.x; j < total; j += T) {
      uint32_t r, k0, k1;
      if (j < n_near) {
        r = j / kMarkLocalParts;
        k0 = (j % kMarkLocalParts) * kPart;
        k1 = min(k0 + kPart, kNear);
      } else {
        const uint32_t g = j - n_near;
        uint32_t lo = 0, hi = nr;  // last ray whose first far segment is <= g
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (R.start[mid] <= g) lo = mid; else hi = mid;
        }
        r = lo;
        k0 = kNear + (g - R.start[r]) * kMarkSeg;
        k1 = k0 + kMarkSeg;
      }
      const uint2 p = R.d[r];
      const uint32_t m = p.y >> 16;
      k1 = min(k1, m);
      if (k0 >= k1) continue;
      visited += k1 - k0;
      const int dx = int(p.x << 16) >> 16, dy = int(p.x) >> 16, dz = int(p.y << 16) >> 16;
      if (j < n_near)
        mark_walk(qox, qoy, qoz, dx, dy, dz, m, k0, k1, near_word, near_flush);
      else
        mark_walk(qox, qoy, qoz, dx, dy, dz, m, k0, k1, far_word, far_flush);
    }
    __syncthreads();
  }
  // the neighbourhood's words into the bitmap, once per block task; the first
  // non-zero word of each block (16 lanes) sets its touched bit
  for (int t0 = int(threadIdx.x & ~31u); t0 < mark_smem_words(NB); t0 += T) {
    const int t = t0 + int(lane);
    uint32_t v = 0;
    if (t < mark_smem_words(NB)) {
      v = sm[t];
      if (v) sm[t] = 0;
    }
    const unsigned nz = __ballot_sync(0xffffffffu, v != 0);
    if (!v) continue;
    const int q = t >> 4, qx = q % NS, qy = (q / NS) % NS, qz = q / (NS * NS);
    const uint32_t b = uint32_t(nlx + qx) + S * uint32_t(nly + qy) + SS * uint32_t(nlz + qz);
    red_or(Q.bits + b * 16u + (t & 15), v);
    const unsigned half = (nz >> (lane & 16u)) & 0xFFFFu;
    if ((lane & 15u) == unsigned(__ffs(half) - 1)) touch_block(Q, b);
  }
  __syncthreads();
}

// Moves the blocks whose touched bits are set in words [32 c, 32 c + 32) of
// the touched bitmap onto the scan's list and clears those words (one warp,
// all lanes).
__device__ __forceinline__ void list_touched(const DMap& M, const RayCube& Q, uint32_t c) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t nw = cube_touched_words(Q);
  const uint32_t wi = c * 32u + lane;
  uint32_t w = 0;
  if (wi < nw) {
    w = Q.touched[wi];
    if (w) Q.touched[wi] = 0;
  }
  const uint32_t cnt = __popc(w);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= unsigned(o)) incl += v;
  }
  const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
  if (!tot) return;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(Q.count, tot);
  uint32_t k = __shfl_sync(0xffffffffu, base, 0) + incl - cnt;
  while (w) {
    const uint32_t bit = uint32_t(__ffs(w) - 1);
    w &= w - 1u;
    if (k < Q.cap)
      Q.list[k] = ((wi * 32u + bit) * kTouchInv) & Q.tmask;
    else
      set_err(M, ERR_SCRATCH);
    ++k;
  }
}


// Leaf slot of the leaf whose lowest cell is (lx, ly, lz), created if
// missing, for a group of kApplyGroup lanes (sl = lane in group, gmask = the
// group's lanes). With a leaf directory D (bxg_scan.cuh), a current word there
// gives the slot in one load; otherwise the root bucket is probed
// cooperatively, one bucket per lane, and a missing or pending root, a long
// chain or a missing leaf goes through the bounded-wait creation path on the
// group's first lane; the slot found is then written to the directory.
__device__ __forceinline__ uint32_t apply_leaf_slot(const DMap& M, int lx, int ly, int lz,
                                                    unsigned sl, unsigned gbase, unsigned gmask,
                                                    const LeafDir* D) {
  uint32_t* dw = nullptr;
  if (D) {
    const uint32_t qx = static_cast<uint32_t>((lx >> 3) - D->x0),
                   qy = static_cast<uint32_t>((ly >> 3) - D->y0),
                   qz = static_cast<uint32_t>((lz >> 3) - D->z0);
    if (qx < D->side && qy < D->side && qz < D->side) {
      dw = D->words + (static_cast<size_t>(qx) * D->side + qy) * D->side + qz;
      const uint32_t w = *dw;
      if ((w >> 28) == D->epoch) return w & 0x0FFFFFFFu;
    }
  }
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
    if (dw && leaf != kNone) *dw = (D->epoch << 28) | leaf;
  }
  return __shfl_sync(gmask, leaf, 0, kApplyGroup);
}

// Applies the ray update to listed block b and clears it (8 lanes; lane sl
// owns bitmap words 2 sl and 2 sl + 1, i.e. the 64 cells 64 sl .. 64 sl + 63
// of the 8^3 leaf, which are mask word sl). The block's bits are
// cleared even when the leaf cannot be had (pool full, error set): the bitmap
// is clean after every apply, and a scan that is re-run after the pools grew
// marks its rays again.
__device__ __forceinline__ void apply_block(const DMap& M, const RayCube& Q, uint32_t b,
                                            int32_t u, int32_t miss, int32_t cmin, unsigned sl,
                                            unsigned gbase, unsigned gmask, uint32_t& updated,
                                            const LeafDir* D = nullptr) {
  const uint32_t SS = Q.S * Q.S;
  const uint32_t bz = b / SS, rem = b - bz * SS, by = rem / Q.S, bx = rem - by * Q.S;
  const int lx = Q.x0 + 8 * int(bx), ly = Q.y0 + 8 * int(by), lz = Q.z0 + 8 * int(bz);
  uint2* wp = reinterpret_cast<uint2*>(Q.bits + size_t(b) * 16u) + sl;
  const uint2 wv = *wp;
  const uint32_t leaf = apply_leaf_slot(M, lx, ly, lz, sl, gbase, gmask, D);
  if ((wv.x | wv.y) == 0u) return;
  *wp = make_uint2(0u, 0u);
  if (leaf == kNone) return;
  int4* cells = reinterpret_cast<int4*>(reinterpret_cast<int32_t*>(M.ldata) +
                                        static_cast<size_t>(leaf) * 512u + 64u * sl);
  unsigned long long fresh = 0;  // cells whose word was zero: turn their mask bits on
  // Per bitmap word, the marked 16-byte runs are all loaded before any is
  // stored: interleaved, each store kept the next load from issuing (the
  // compiler cannot tell the runs apart), one round trip per run.
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t w = h ? wv.y : wv.x;
    if (!w) continue;
    int4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if ((w >> (4 * j)) & 0xFu) v[j] = cells[8 * h + j];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t nib = (w >> (4 * j)) & 0xFu;
      if (!nib) continue;
      int32_t* c = reinterpret_cast<int32_t*>(&v[j]);
      bool changed = false;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (!((nib >> t) & 1u)) continue;
        const int32_t old = c[t];
        if (cell_id(old) != u) {
          c[t] = cell_pack(max(wrap_add(cell_prob(old), miss), cmin), u);
          changed = true;
          ++updated;
        }
        if (old == 0) fresh |= 1ull << (32 * h + 4 * j + t);
      }
      if (changed) cells[8 * h + j] = v[j];
    }
  }
  if (fresh) red_or64(M.lmask + static_cast<size_t>(leaf) * M.lwords + sl, fresh);
}

// ---------------------------------------------------------------------------
// The per-scan form: segments of cells, marked straight into the bitmap.
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
//   n(k) = floor((2 k d + m) / (2 m)) = floor(k d/m + 1/2)
//
// and floor(fma(k, fl(d/m), 1/2 + 1/(4m))) is exactly that for k < 801 and
// m <= 2047: the values (2 k d + m) / (2 m) are multiples of 1/(2m), so adding
// half of that keeps each 1/(4m) >= 1.2e-4 from the next integer, and the
// error (k 2^-25 of the slope, 2^-15 of the rounded sum, 2^-25 of the offset)
// stays below 5.5e-5. Longer rays divide in integers.
//
// What bounds it: instruction issue, and for clouds of one narrow direction (a
// depth frame) the ORs that meet in few words of L2. Kernel times on a GB300,
// L2 warm, against tasks of rays whose segments were found by a prefix and a
// search and walked with integer divisions (the form before): LiDAR 131k points,
// 9.3 M cells, 28 us (62); depth 307k points, 10.5 M cells, 62 us (105); room
// 60k points 20 us (30). Of that, without the far ORs: 26, 39 and 19 us; with
// every lane's cells ORed, neighbours' too: 36, 65 and 21 us. Measured and not
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
constexpr uint32_t kMarkMaxRay = 32768;          // longer rays are walked on the tree (k_tail)
constexpr uint32_t kFmaMaxRay = 2047;
constexpr int kMaxCubeHalf = 24;                 // roots on each side: bit addresses in 32 bits
constexpr int kOpenCubeHalf = 16;                // of a scan whose rays may be of any length
constexpr uint32_t kRootFlagWords =
    ((2 * kMaxCubeHalf + 1) * (2 * kMaxCubeHalf + 1) * (2 * kMaxCubeHalf + 1) + 31) / 32;

struct ScanCube {
  uint32_t* bits;   // S^3 leaf blocks of 16 words, x fastest; zero between scans
  uint32_t* roots;  // one bit per root (SR^3), set by the segments
  uint32_t* segs;   // segments: ray << 8 | number; nullptr: rays are walked whole
  uint32_t* tails;  // rays longer than kin; nullptr: not listed
  int x0, y0, z0;   // lowest cell (multiples of 32)
  uint32_t S, SR;   // leaves, roots per side
  uint32_t kin;     // cells k < kin of every ray lie in the cube
  uint32_t open;    // rays may be longer (k_tail walks the rest)
};

__host__ __device__ inline uint32_t cube_root_words(const ScanCube& Q) {
  return (Q.SR * Q.SR * Q.SR + 31u) / 32u;
}
// Segments of a ray of len cells.
__device__ __forceinline__ uint32_t far_segments(const ScanCube& Q, uint32_t len) {
  const uint32_t m = min(len, Q.kin);
  return len < kMarkMaxRay && m > kNearCells ? (m - kNearCells + kSegCells - 1) / kSegCells : 0u;
}

// One thread's ray, as the marking needs it.
struct MarkRay {
  float sx, sy, sz, off;  // slopes |d| / m and the rounding offset
  int gx, gy, gz;         // signs
  uint32_t m;             // cells to mark; 0: none
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
  const float fm = static_cast<float>(max(r.len, 1u));
  r.sx = __fdiv_rn(static_cast<float>(abs(r.dx)), fm);
  r.sy = __fdiv_rn(static_cast<float>(abs(r.dy)), fm);
  r.sz = __fdiv_rn(static_cast<float>(abs(r.dz)), fm);
  r.off = 0.5f + __fdiv_rn(0.25f, fm);
  r.gx = r.dx < 0 ? -1 : 1;
  r.gy = r.dy < 0 ? -1 : 1;
  r.gz = r.dz < 0 ? -1 : 1;
  return r;
}

// Cell k of the ray, relative to its origin cell.
template <bool LONG>
__device__ __forceinline__ void mark_cell(const MarkRay& r, uint32_t k, int& x, int& y, int& z) {
  if (LONG) {
    const uint32_t tm = 2u * r.len;
    x = int((2u * k * uint32_t(abs(r.dx)) + r.len) / tm) * r.gx;
    y = int((2u * k * uint32_t(abs(r.dy)) + r.len) / tm) * r.gy;
    z = int((2u * k * uint32_t(abs(r.dz)) + r.len) / tm) * r.gz;
  } else {
    const float f = static_cast<float>(k);
    x = int(__float_as_uint(__fadd_rd(__fmaf_rn(f, r.sx, r.off), 8388608.0f)) - 0x4B000000u) * r.gx;
    y = int(__float_as_uint(__fadd_rd(__fmaf_rn(f, r.sy, r.off), 8388608.0f)) - 0x4B000000u) * r.gy;
    z = int(__float_as_uint(__fadd_rd(__fmaf_rn(f, r.sz, r.off), 8388608.0f)) - 0x4B000000u) * r.gz;
  }
}

// Marks cells 0 .. n - 1 (n <= kNearCells) in the shared neighbourhood, whose
// lowest cell is (wx, wy, wz) from the origin. The walk starts at cell rot: the
// lanes of a warp are apart then, where they would all OR the origin's word.
template <bool LONG>
__device__ __forceinline__ void mark_near(const MarkRay& r, uint32_t n, uint32_t rot, int wx,
                                          int wy, int wz, uint32_t* sm) {
  uint32_t cur = 0, acc = 0, k = rot;
  for (uint32_t j = 0; j < n; ++j) {
    int x, y, z;
    mark_cell<LONG>(r, k, x, y, z);
    const uint32_t X = uint32_t(x - wx), Y = uint32_t(y - wy), Z = uint32_t(z - wz);
    const uint32_t w = (X >> 3) + kNearW * ((Y >> 2) + 2 * kNearW * Z);
    if (w != cur) {
      if (acc) atomicOr(sm + cur, acc);
      acc = 0;
      cur = w;
    }
    acc |= 1u << ((X & 7u) | ((Y & 3u) << 3));
    k = k + 1 < n ? k + 1 : 0;
  }
  if (acc) atomicOr(sm + cur, acc);
}

// Marks cells ka <= k < kb of each thread's ray in the bitmap (ka >= kb: none);
// (qx, qy, qz): the origin in the cube. All lanes of the warp, unless LONG.
template <bool LONG>
__device__ __forceinline__ void mark_far(const ScanCube& Q, const MarkRay& r, uint32_t ka,
                                         uint32_t kb, int qx, int qy, int qz) {
  // bit address: x + 8 y + 64 z, and for each axis the leaf's offset less the cells' own
  const uint32_t cy = 512u * Q.S - 64u, cz = 512u * Q.S * Q.S - 512u;
  auto address = [&](uint32_t x, uint32_t y, uint32_t z) {
    return x + 8u * y + 64u * z + (x >> 3) * 504u + (y >> 3) * cy + (z >> 3) * cz;
  };
  uint32_t cur = 0, acc = 0;
  auto put = [&](uint32_t a) {
    if ((a ^ cur) & ~31u) {
      if (acc) red_or(Q.bits + (cur >> 5), acc);
      acc = 0;
      cur = a;
    }
    acc |= 1u << (a & 31u);
  };
  if (LONG) {
    for (uint32_t k = ka; k < kb; ++k) {
      int x, y, z;
      mark_cell<true>(r, k, x, y, z);
      put(address(uint32_t(qx + x), uint32_t(qy + y), uint32_t(qz + z)));
    }
  } else {
    // 2^23 + n as a float has the bits 0x4B000000 + n
    const uint32_t px = uint32_t(qx) - 0x4B000000u * uint32_t(r.gx),
                   py = uint32_t(qy) - 0x4B000000u * uint32_t(r.gy),
                   pz = uint32_t(qz) - 0x4B000000u * uint32_t(r.gz);
    const bool first = (threadIdx.x & 31) == 0;
    const uint32_t steps = __reduce_max_sync(0xffffffffu, kb > ka ? kb - ka : 0u);
    const float fe = static_cast<float>(kb);
    float f = static_cast<float>(ka);
    for (uint32_t j = 0; j < steps; ++j, f += 1.0f) {
      const uint32_t ix = __float_as_uint(__fadd_rd(__fmaf_rn(f, r.sx, r.off), 8388608.0f)),
                     iy = __float_as_uint(__fadd_rd(__fmaf_rn(f, r.sy, r.off), 8388608.0f)),
                     iz = __float_as_uint(__fadd_rd(__fmaf_rn(f, r.sz, r.off), 8388608.0f));
      const uint32_t a = address(px + ix * uint32_t(r.gx), py + iy * uint32_t(r.gy),
                                 pz + iz * uint32_t(r.gz));
      const bool act = f < fe;
      const uint32_t before = __shfl_up_sync(0xffffffffu, act ? a : kNone, 1);
      if (act && (first || before != a)) put(a);
    }
  }
  if (acc) red_or(Q.bits + (cur >> 5), acc);
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

// Block `block` of n_blocks marks its part of a scan's rays: the near cells of
// some rays, and some segments. All threads of a block of kMarkThreads. Adds
// the cells walked to `visited`.
__device__ __forceinline__ void mark_scan(const DMap& M, const ScanCube& Q,
                                          const int4* __restrict__ cast, uint32_t n_cast,
                                          uint32_t n_segs, uint32_t block, uint32_t n_blocks,
                                          int ox, int oy, int oz, MarkShared& S,
                                          uint32_t& visited) {
  const int qx = ox - Q.x0, qy = oy - Q.y0, qz = oz - Q.z0;  // the origin in the cube
  // the neighbourhood's lowest cell, from the origin
  const int wx = ((qx >> 3) - kNearNB) * 8 - qx, wy = ((qy >> 3) - kNearNB) * 8 - qy,
            wz = ((qz >> 3) - kNearNB) * 8 - qz;
  const uint32_t root_words = cube_root_words(Q);
  for (uint32_t t = threadIdx.x; t < kNearWords; t += kMarkThreads) S.near[t] = 0u;
  for (uint32_t t = threadIdx.x; t < root_words; t += kMarkThreads) S.roots[t] = 0u;
  __syncthreads();
  const uint32_t tid = block * kMarkThreads + threadIdx.x, nt = n_blocks * kMarkThreads;
  for (uint32_t i = tid; i < n_cast; i += nt) {
    const MarkRay r = mark_ray(M, Q, cast[i], ox, oy, oz);
    if (!r.m) continue;
    visited += r.m;
    const uint32_t n = min(r.m, kNearCells);
    const uint32_t rot = (threadIdx.x & 31) * n >> 5;
    if (r.len > kFmaMaxRay)
      mark_near<true>(r, n, rot, wx, wy, wz, S.near);
    else
      mark_near<false>(r, n, rot, wx, wy, wz, S.near);
  }
  if (Q.segs) {
    for (uint32_t i0 = tid & ~31u; i0 < n_segs; i0 += nt) {
      const uint32_t i = i0 + (threadIdx.x & 31);
      const uint32_t s = i < n_segs ? Q.segs[i] : 0u;
      const MarkRay r = mark_ray(M, Q, cast[s >> 8], ox, oy, oz);
      const uint32_t ka = kNearCells + (s & 255u) * kSegCells;
      const uint32_t kb = i < n_segs ? min(ka + kSegCells, r.m) : 0u;
      int ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;
      if (__any_sync(0xffffffffu, r.len > kFmaMaxRay)) {
        if (kb) {
          mark_cell<true>(r, ka, ax, ay, az);
          mark_cell<true>(r, kb - 1, bx, by, bz);
          mark_far<true>(Q, r, ka, kb, qx, qy, qz);
        }
      } else {
        mark_cell<false>(r, ka, ax, ay, az);
        mark_cell<false>(r, kb - 1, bx, by, bz);
        mark_far<false>(Q, r, ka, kb, qx, qy, qz);
      }
      if (kb) flag_roots(Q, qx + ax, qy + ay, qz + az, qx + bx, qy + by, qz + bz, S.roots);
    }
  } else {
    for (uint32_t i = tid; i < n_cast; i += nt) {
      const MarkRay r = mark_ray(M, Q, cast[i], ox, oy, oz);
      for (uint32_t ka = kNearCells; ka < r.m; ka += kSegCells) {
        const uint32_t kb = min(ka + kSegCells, r.m);
        int ax, ay, az, bx, by, bz;
        mark_cell<true>(r, ka, ax, ay, az);
        mark_cell<true>(r, kb - 1, bx, by, bz);
        mark_far<true>(Q, r, ka, kb, qx, qy, qz);
        flag_roots(Q, qx + ax, qy + ay, qz + az, qx + bx, qy + by, qz + bz, S.roots);
      }
    }
  }
  __syncthreads();
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
  for (uint32_t t = threadIdx.x; t < root_words; t += kMarkThreads)
    if (S.roots[t]) red_or(Q.roots + t, S.roots[t]);
}

// ---------------------------------------------------------------------------
// Apply, a warp per row of four leaf blocks of a root.
//
// Four groups of eight lanes each read a block's bits and find (or create) its leaf;
// then the whole warp updates one block after the other, each lane the cells of two
// rows of 8 cells (one 32-byte sector each).
//
// What bounds it: the chain bits -> root bucket -> child word -> cells -> stores, and
// instruction issue. LiDAR 131k points, 4.0 M cells in 18 k leaves: 24 us against 37
// with eight lanes for each leaf of a list (a lane had 64 cells, two
// rounds of eight loads). Two blocks at a time (80 registers) or fewer than six
// blocks of threads per SM: 26 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t row_bits(uint2 wv, unsigned src, unsigned lane) {
  const uint32_t a = __shfl_sync(0xffffffffu, wv.x, src), b = __shfl_sync(0xffffffffu, wv.y, src);
  return ((lane & 4u ? b : a) >> (8u * (lane & 3u))) & 0xFFu;
}

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

// Blocks 4 rx .. 4 rx + 3 of the row (by, bz), in leaves of the cube.
__device__ __forceinline__ void apply_row(const DMap& M, const ScanCube& Q, uint32_t rx,
                                          uint32_t by, uint32_t bz, int32_t u, int32_t miss,
                                          int32_t cmin, uint32_t& updated) {
  const unsigned lane = threadIdx.x & 31, sl = lane & 7u, gbase = lane & 24u;
  const uint32_t bx = 4u * rx + (lane >> 3);
  uint2* wp = reinterpret_cast<uint2*>(Q.bits + size_t(bx + Q.S * (by + Q.S * bz)) * 16u) + sl;
  const uint2 wv = *wp;
  const unsigned any = __ballot_sync(0xffffffffu, (wv.x | wv.y) != 0u);
  if (!any) return;
  uint32_t leaf = kNone;
  if ((any >> gbase) & 0xFFu) {
    leaf = apply_leaf_slot(M, Q.x0 + 8 * int(bx), Q.y0 + 8 * int(by), Q.z0 + 8 * int(bz), sl,
                           gbase, 0xFFu << gbase, nullptr);
    if (wv.x | wv.y) *wp = make_uint2(0u, 0u);
  }
  __syncwarp();
#pragma unroll 1
  for (unsigned g = 0; g < 4; ++g) {
    const uint32_t lf = __shfl_sync(0xffffffffu, leaf, 8 * g);
    if (lf == kNone) continue;  // no marked cell, or no leaf (pool full: the scan is re-run)
    uint32_t row[2] = {row_bits(wv, 8 * g + (lane >> 3), lane),
                       row_bits(wv, 8 * g + 4 + (lane >> 3), lane)};
    int4* c = reinterpret_cast<int4*>(M.ldata) + size_t(lf) * 128u + 2 * lane;
    int4 v[2][2];  // rows lane and lane + 32
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (row[h] & 0xFu) v[h][0] = c[64 * h];
      if (row[h] & 0xF0u) v[h][1] = c[64 * h + 1];
    }
    uint32_t* mw = reinterpret_cast<uint32_t*>(M.lmask) + size_t(lf) * 16u + (lane >> 2);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!row[h]) continue;
      uint32_t fresh = 0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t nib = (row[h] >> (4 * q)) & 0xFu;
        if (!nib) continue;
        bool changed = false;
        fresh |= miss_run(v[h][q], nib, u, miss, cmin, changed, updated) << (4 * q);
        if (changed) c[64 * h + q] = v[h][q];
      }
      if (fresh) red_or(mw + 8 * h, fresh << (8u * (lane & 3u)));
    }
  }
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
                                           int32_t u, int32_t miss, int32_t cmin,
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
    apply_row(M, Q, rx, 4u * ry + (t & 3u), 4u * rz + ((t >> 2) & 3u), u, miss, cmin, updated);
  }
}

}  // namespace bxg
