// Serialize and Deserialize in the reference's format (serialization.hpp:77-199):
//   "Bonxai::VoxelGrid<type,inner_bits,leaf_bits>(resolution)\n"
//   uint32 root count; per root: int32 x, y, z; inner mask words; per inner
//   bit set (ascending): leaf mask words, then each on cell's value
//   (ascending cell index).
// Roots are written in ascending (x, y, z) order (the reference writes them in
// its unordered_map's order; any order deserializes to the same grid).
//
// Saving: one kernel lists the roots with the bytes each takes; the host sorts
// them and adds up their places; a second kernel writes the file's body, 64 MB at a time, a
// block per root and a warp per leaf, and only that is copied to the host (twice copying the node
// pools to the host, writing the file there, and setting its cells as one batch of coordinates took
// 33 ms for a map of 2.4 M cells, a 12 MB file, saved and loaded; now 2.3 ms, of which the kernels are 83 us
// and the rest the copies of the file). Loading: the host goes
// through the masks to find the leaves, without touching the values, and a
// kernel puts each leaf in, a warp per leaf.
#include <algorithm>
#include <array>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <unordered_set>
#include <vector>

#include "bxg_internal.h"

namespace bxg {
namespace {

// Bytes of the body that are on the device at a time (a root may have more).
constexpr unsigned long long kFilePiece = 64ull << 20;

// A root of the file: its key, inner slot, body bytes, and the place of its body.
struct FileRoot {
  int32_t x, y, z;
  uint32_t inner, bytes, pad;
  unsigned long long at;
};
// A leaf of the file: its lowest cell and the place of its mask.
struct FileLeaf {
  int32_t x, y, z, pad;
  unsigned long long at;
};

__device__ __forceinline__ uint32_t leaf_count(const DMap& M, uint32_t leaf) {
  uint32_t c = 0;
  for (int w = 0; w < M.lwords; ++w)
    c += __popcll(M.lmask[static_cast<size_t>(leaf) * M.lwords + w]);
  return c;
}

// A warp per bucket of the root table: the roots that have a leaf, and their bytes.
__global__ void __launch_bounds__(256) k_file_roots(const __grid_constant__ DMap M,
                                                    FileRoot* __restrict__ out,
                                                    unsigned long long* __restrict__ count) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i <= M.hmask; i += nw) {
    const uint4 b = M.buckets[i];
    if (static_cast<int>(b.x) == kEmptyKey || b.w >= kPending) continue;
    uint32_t leaves = 0, cells = 0;
    for (int c = int(lane); c < M.isize; c += 32) {
      if (!((M.imask[static_cast<size_t>(b.w) * M.iwords + (c >> 6)] >> (c & 63)) & 1ull)) continue;
      ++leaves;
      if (M.esz) cells += leaf_count(M, M.ichild[static_cast<size_t>(b.w) * M.isize + c]);
    }
    leaves = __reduce_add_sync(0xffffffffu, leaves);
    cells = __reduce_add_sync(0xffffffffu, cells);
    if (lane != 0 || !leaves) continue;  // a root whose leaves were all released
    FileRoot r;
    r.x = static_cast<int32_t>(b.x);
    r.y = static_cast<int32_t>(b.y);
    r.z = static_cast<int32_t>(b.z);
    r.inner = b.w;
    r.bytes = 12u + 8u * M.iwords + leaves * 8u * M.lwords + cells * M.esz;
    r.pad = 0;
    r.at = 0;
    out[atomicAdd(count, 1ull)] = r;
  }
}

// Bytes at a place of the body: it is a multiple of four for values of four and
// eight bytes, any for smaller ones.
template <int ESZ>
__device__ __forceinline__ void put_word(uint8_t* p, unsigned long long v) {
  if (ESZ == 0 || ESZ >= 4) {
    reinterpret_cast<uint32_t*>(p)[0] = static_cast<uint32_t>(v);
    reinterpret_cast<uint32_t*>(p)[1] = static_cast<uint32_t>(v >> 32);
  } else {
    for (int k = 0; k < 8; ++k) p[k] = static_cast<uint8_t>(v >> (8 * k));
  }
}
template <int ESZ>
__device__ __forceinline__ unsigned long long get_word(const uint8_t* p) {
  if (ESZ == 0 || ESZ >= 4) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
    return w[0] | (static_cast<unsigned long long>(w[1]) << 32);
  }
  unsigned long long v = 0;
  for (int k = 0; k < 8; ++k) v |= static_cast<unsigned long long>(p[k]) << (8 * k);
  return v;
}
template <int ESZ>
__device__ __forceinline__ void copy_value(uint8_t* dst, const uint8_t* src) {
  if (ESZ >= 4) {
    for (int k = 0; k < ESZ / 4; ++k)
      reinterpret_cast<uint32_t*>(dst)[k] = reinterpret_cast<const uint32_t*>(src)[k];
  } else {
    for (int k = 0; k < ESZ; ++k) dst[k] = src[k];
  }
}

// The body of the file from byte `begin`, a block per root: the children in chunks of blockDim.x, whose
// places the block adds up, then a warp per leaf; 32 cells at a time, the values
// of on cells side by side.
template <int ESZ>
__global__ void __launch_bounds__(256) k_file_write(const __grid_constant__ DMap M,
                                                    const FileRoot* __restrict__ roots,
                                                    uint8_t* __restrict__ body,
                                                    unsigned long long begin) {
  __shared__ uint32_t s_leaf[256], s_at[256], s_sum[8];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const FileRoot r = roots[blockIdx.x];
  uint8_t* const base = body + (r.at - begin);
  if (threadIdx.x < 3) {
    const int32_t key = threadIdx.x == 0 ? r.x : threadIdx.x == 1 ? r.y : r.z;
    if (ESZ == 0 || ESZ >= 4)
      reinterpret_cast<int32_t*>(base)[threadIdx.x] = key;
    else
      for (int k = 0; k < 4; ++k)
        base[4 * threadIdx.x + k] = static_cast<uint8_t>(static_cast<uint32_t>(key) >> (8 * k));
  }
  const unsigned long long* im = M.imask + static_cast<size_t>(r.inner) * M.iwords;
  for (int w = int(threadIdx.x); w < M.iwords; w += blockDim.x) put_word<ESZ>(base + 12 + 8 * w, im[w]);
  uint32_t done = 12u + 8u * M.iwords;  // bytes of the root written or placed so far
  for (int c0 = 0; c0 < M.isize; c0 += blockDim.x) {
    const int c = c0 + int(threadIdx.x);
    uint32_t leaf = kNone, bytes = 0;
    if (c < M.isize && ((im[c >> 6] >> (c & 63)) & 1ull)) {
      leaf = M.ichild[static_cast<size_t>(r.inner) * M.isize + c];
      bytes = 8u * M.lwords + (ESZ ? leaf_count(M, leaf) * ESZ : 0u);
    }
    uint32_t incl = bytes;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= unsigned(o)) incl += v;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    uint32_t before = done + incl - bytes;
    for (unsigned k = 0; k < 8; ++k) {
      if (k < warp) before += s_sum[k];
      done += s_sum[k];
    }
    s_leaf[threadIdx.x] = leaf;
    s_at[threadIdx.x] = before;
    __syncthreads();
    for (int j = int(warp); j < 256 && c0 + j < M.isize; j += 8) {
      const uint32_t lf = s_leaf[j];
      if (lf == kNone) continue;
      uint8_t* dst = base + s_at[j];
      const unsigned long long* lm = M.lmask + static_cast<size_t>(lf) * M.lwords;
      for (int w = int(lane); w < M.lwords; w += 32) put_word<ESZ>(dst + 8 * w, lm[w]);
      if (!ESZ) continue;
      dst += 8 * M.lwords;
      const uint8_t* src = M.ldata + static_cast<size_t>(lf) * M.lsize * ESZ;
      for (int i0 = 0; i0 < M.lsize; i0 += 32) {
        const int i = i0 + int(lane);
        const bool on = i < M.lsize && ((lm[i >> 6] >> (i & 63)) & 1ull);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) copy_value<ESZ>(dst + size_t(__popc(m & ((1u << lane) - 1u))) * ESZ, src + size_t(i) * ESZ);
        dst += size_t(__popc(m)) * ESZ;
      }
    }
    __syncthreads();
  }
}

// The leaves of a file into the grid, a warp per leaf. The leaves are distinct, so
// no other warp writes to this one's.
template <int ESZ>
__global__ void __launch_bounds__(256) k_file_read(const __grid_constant__ DMap M,
                                                   const FileLeaf* __restrict__ leaves, uint32_t n,
                                                   const uint8_t* __restrict__ body) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i0 >= n) return;
  const FileLeaf f = leaves[i0];
  uint32_t lf = kNone;
  if (lane == 0) lf = leaf_of(M, f.x, f.y, f.z, true);
  lf = __shfl_sync(0xffffffffu, lf, 0);
  if (lf == kNone) return;  // the pool is full: run again after it grew
  const uint8_t* src = body + f.at;
  for (int w = int(lane); w < M.lwords; w += 32) {
    const unsigned long long v = get_word<ESZ>(src + 8 * w);
    if (v) atomicOr(M.lmask + static_cast<size_t>(lf) * M.lwords + w, v);
  }
  if (!ESZ) return;
  const uint8_t* val = src + 8 * M.lwords;
  uint8_t* cells = M.ldata + static_cast<size_t>(lf) * M.lsize * ESZ;
  unsigned long long v = 0;
  for (int i0 = 0; i0 < M.lsize; i0 += 32) {
    const int i = i0 + int(lane);
    if ((i0 & 63) == 0) v = get_word<ESZ>(src + 8 * (i0 >> 6));
    const bool on = i < M.lsize && ((v >> (i & 63)) & 1ull);
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) copy_value<ESZ>(cells + size_t(i) * ESZ, val + size_t(__popc(m & ((1u << lane) - 1u))) * ESZ);
    val += size_t(__popc(m)) * ESZ;
  }
}

// The roots of the file in ascending key order, with their places; *bytes: the body's.
int file_roots(MapCore* m, std::vector<FileRoot>& roots, unsigned long long* bytes) {
  int st = core_sync(m);
  if (st) return st;
  const size_t cap = size_t(m->h_ctr[C_ROOTS]);
  roots.clear();
  *bytes = 0;
  if (!cap) return BXG_OK;
  BXG_CUDA(m, m->s_out2.ensure(cap * sizeof(FileRoot)));
  BXG_CUDA(m, m->s_tmp.ensure(8));
  BXG_CUDA(m, cudaMemsetAsync(m->s_tmp.p, 0, 8, m->stream));
  const uint32_t warps = m->dm.hmask + 1;
  const unsigned blocks = std::min<uint32_t>((warps + 7) / 8, uint32_t(m->sm_count) * 8);
  k_file_roots<<<blocks, 256, 0, m->stream>>>(m->dm, m->s_out2.as<FileRoot>(),
                                              m->s_tmp.as<unsigned long long>());
  BXG_LAUNCHED(m);
  unsigned long long n = 0;
  roots.resize(cap);
  BXG_CUDA(m, cudaMemcpyAsync(&n, m->s_tmp.p, 8, cudaMemcpyDeviceToHost, m->stream));
  BXG_CUDA(m, cudaMemcpyAsync(roots.data(), m->s_out2.p, cap * sizeof(FileRoot),
                              cudaMemcpyDeviceToHost, m->stream));
  BXG_CUDA(m, cudaStreamSynchronize(m->stream));
  roots.resize(size_t(n));
  std::sort(roots.begin(), roots.end(), [](const FileRoot& a, const FileRoot& b) {
    return a.x != b.x ? a.x < b.x : a.y != b.y ? a.y < b.y : a.z < b.z;
  });
  for (FileRoot& r : roots) {
    r.at = *bytes;
    *bytes += r.bytes;
  }
  return BXG_OK;
}

}  // namespace
}  // namespace bxg

using namespace bxg;

extern "C" int bxg_grid_serialize(bxg_grid g, const char* type_name, void* out, size_t cap,
                                  size_t* n_out) {
  if (!g || !type_name) return BXG_ERR_INVALID_ARG;
  MapCore* m = const_cast<MapCore*>(core_of_handle(g));
  cudaSetDevice(m->device);
  std::vector<FileRoot> roots;
  unsigned long long bytes = 0;
  int st = file_roots(m, roots, &bytes);
  if (st) return st;
  const DMap& d = m->dm;
  char header[256];
  std::snprintf(header, sizeof(header), "Bonxai::VoxelGrid<%s,%d,%d>(%lf)\n", type_name, d.ib,
                d.lb, m->res);
  const size_t head = std::strlen(header);
  const size_t total = head + 4 + size_t(bytes);
  if (n_out) *n_out = total;
  if (!out) return BXG_OK;
  if (total > cap) return set_error(m, BXG_ERR_CAPACITY, "output buffer too small");
  uint8_t* p = static_cast<uint8_t*>(out);
  std::memcpy(p, header, head);
  const uint32_t nroots = uint32_t(roots.size());
  std::memcpy(p + head, &nroots, 4);
  if (!nroots) return BXG_OK;
  BXG_CUDA(m, m->s_in2.ensure(roots.size() * sizeof(FileRoot)));
  BXG_CUDA(m, cudaMemcpyAsync(m->s_in2.p, roots.data(), roots.size() * sizeof(FileRoot),
                              cudaMemcpyHostToDevice, m->stream));
  // in pieces: the map may have left little device memory
  for (uint32_t r0 = 0, r1; r0 < nroots; r0 = r1) {
    const unsigned long long begin = roots[r0].at;
    unsigned long long end = begin + roots[r0].bytes;
    for (r1 = r0 + 1; r1 < nroots && end + roots[r1].bytes - begin <= kFilePiece; ++r1)
      end += roots[r1].bytes;
    BXG_CUDA(m, m->s_out.ensure(size_t(end - begin)));
    const FileRoot* dr = m->s_in2.as<FileRoot>() + r0;
    uint8_t* body = m->s_out.as<uint8_t>();
    const unsigned n = r1 - r0;
    switch (d.esz) {
      case 0: k_file_write<0><<<n, 256, 0, m->stream>>>(d, dr, body, begin); break;
      case 1: k_file_write<1><<<n, 256, 0, m->stream>>>(d, dr, body, begin); break;
      case 2: k_file_write<2><<<n, 256, 0, m->stream>>>(d, dr, body, begin); break;
      case 4: k_file_write<4><<<n, 256, 0, m->stream>>>(d, dr, body, begin); break;
      default: k_file_write<8><<<n, 256, 0, m->stream>>>(d, dr, body, begin); break;
    }
    BXG_LAUNCHED(m);
    BXG_CUDA(m, cudaMemcpyAsync(p + head + 4 + begin, body, size_t(end - begin),
                                cudaMemcpyDeviceToHost, m->stream));
    BXG_CUDA(m, cudaStreamSynchronize(m->stream));
  }
  return BXG_OK;
}

namespace {
// The cells of a file's body as one batch in the order of the file, the last value of a cell
// winning as setValue calls in that order would. The body has been found to hold them all.
int set_in_file_order(bxg_grid g, MapCore* m, const uint8_t* p, uint32_t nroots, size_t cells) {
  const DMap& d = m->dm;
  auto take = [&](void* dst, size_t k) {
    std::memcpy(dst, p, k);
    p += k;
  };
  std::vector<int32_t> xyz;
  std::vector<uint8_t> vals;
  xyz.reserve(3 * cells);
  vals.reserve(cells * size_t(d.esz));
  std::vector<uint64_t> iw(d.iwords), lw(d.lwords);
  const int im = (1 << d.ib) - 1, lm = (1 << d.lb) - 1;
  for (uint32_t r = 0; r < nroots; r++) {
    int32_t key[3];
    take(key, 12);
    take(iw.data(), iw.size() * 8);
    for (int a = 0; a < d.iwords; a++)
      for (uint64_t bits = iw[a]; bits; bits &= bits - 1) {
        const int ii = a * 64 + __builtin_ctzll(bits);
        const int xb = key[0] | ((ii & im) << d.lb), yb = key[1] | (((ii >> d.ib) & im) << d.lb),
                  zb = key[2] | (((ii >> (2 * d.ib)) & im) << d.lb);
        take(lw.data(), lw.size() * 8);
        for (int b = 0; b < d.lwords; b++)
          for (uint64_t cb = lw[b]; cb; cb &= cb - 1) {
            const int ci = b * 64 + __builtin_ctzll(cb);
            xyz.push_back(xb | (ci & lm));
            xyz.push_back(yb | ((ci >> d.lb) & lm));
            xyz.push_back(zb | ((ci >> (2 * d.lb)) & lm));
            if (d.esz) {
              vals.insert(vals.end(), p, p + d.esz);
              p += d.esz;
            }
          }
      }
  }
  if (d.esz) return bxg_grid_set_values(g, xyz.data(), vals.data(), xyz.size() / 3, nullptr);
  return bxg_grid_set_cells_on(g, xyz.data(), xyz.size() / 3, nullptr, nullptr);
}
}  // namespace

extern "C" int bxg_grid_deserialize(bxg_grid g, const void* data, size_t n) {
  if (!g || !data) return BXG_ERR_INVALID_ARG;
  MapCore* m = const_cast<MapCore*>(core_of_handle(g));
  const DMap& d = m->dm;
  const uint8_t* p = static_cast<const uint8_t*>(data);
  const uint8_t* end = p + n;
  // header line (serialization.hpp:126-151): prefix, type, bits, resolution
  const uint8_t* nl = static_cast<const uint8_t*>(std::memchr(p, '\n', n));
  if (!nl) return set_error(m, BXG_ERR_INVALID_ARG, "Header wasn't recognized");
  const std::string header(reinterpret_cast<const char*>(p), nl - p);
  if (header.rfind("Bonxai::VoxelGrid<", 0) != 0)
    return set_error(m, BXG_ERR_INVALID_ARG, "Header wasn't recognized");
  const size_t lt = header.rfind('>');
  const size_t c2 = header.rfind(',', lt);
  const size_t c1 = header.rfind(',', c2 - 1);
  if (lt == std::string::npos || c1 == std::string::npos || c2 == std::string::npos)
    return set_error(m, BXG_ERR_INVALID_ARG, "Header wasn't recognized");
  const int ib = std::atoi(header.substr(c1 + 1, c2 - c1 - 1).c_str());
  const int lb = std::atoi(header.substr(c2 + 1, lt - c2 - 1).c_str());
  if (ib != d.ib || lb != d.lb)
    return set_error(m, BXG_ERR_INVALID_ARG, "inner/leaf bits do not match this grid");
  p = nl + 1;
  auto take = [&](void* dst, size_t k) -> bool {
    if (size_t(end - p) < k) return false;
    std::memcpy(dst, p, k);
    p += k;
    return true;
  };
  uint32_t nroots = 0;
  if (!take(&nroots, 4)) return set_error(m, BXG_ERR_INVALID_ARG, "truncated stream");
  // The leaves and where their masks lie. Roots that are not distinct root keys (the
  // reference writes none) may name a cell twice: then the values are set in the
  // order of the file, one batch of cells.
  const uint8_t* const body = p;
  std::vector<FileLeaf> leaves;
  std::vector<uint64_t> iw(d.iwords), lw(d.lwords);
  std::unordered_set<uint64_t> seen;
  bool plain = true;
  size_t cells = 0;
  const int im = (1 << d.ib) - 1, low = (1 << (d.ib + d.lb)) - 1;
  for (uint32_t r = 0; r < nroots; r++) {
    int32_t key[3];
    if (!take(key, 12) || !take(iw.data(), iw.size() * 8))
      return set_error(m, BXG_ERR_INVALID_ARG, "truncated stream");
    // three keys do not fit 64 bits: a mix of all their bits tells most apart, and a
    // match only means the general path
    uint64_t h = uint32_t(key[0]);
    h = (h ^ (h >> 29)) * 0x9E3779B97F4A7C15ull + uint32_t(key[1]);
    h = (h ^ (h >> 29)) * 0x9E3779B97F4A7C15ull + uint32_t(key[2]);
    h = (h ^ (h >> 29)) * 0x9E3779B97F4A7C15ull;
    plain &= ((key[0] | key[1] | key[2]) & low) == 0 && seen.insert(h).second;
    for (int a = 0; a < d.iwords; a++)
      for (uint64_t bits = iw[a]; bits; bits &= bits - 1) {
        const int ii = a * 64 + __builtin_ctzll(bits);
        if (ii >= d.isize) plain = false;  // a bit beyond an inner node of eight children
        FileLeaf f;
        f.x = key[0] | ((ii & im) << d.lb);
        f.y = key[1] | (((ii >> d.ib) & im) << d.lb);
        f.z = key[2] | (((ii >> (2 * d.ib)) & im) << d.lb);
        f.pad = 0;
        f.at = uint64_t(p - body);
        if (!take(lw.data(), lw.size() * 8))
          return set_error(m, BXG_ERR_INVALID_ARG, "truncated stream");
        size_t on = 0;
        for (uint64_t v : lw) on += size_t(__builtin_popcountll(v));
        if (d.lsize < 64 && (lw[0] >> d.lsize)) plain = false;
        if (size_t(end - p) < on * size_t(d.esz))
          return set_error(m, BXG_ERR_INVALID_ARG, "truncated stream");
        p += on * size_t(d.esz);
        cells += on;
        if (on) leaves.push_back(f);
      }
  }
  if (!cells) return BXG_OK;
  if (!plain || leaves.size() >= 0x7FFFFFFFu)
    return set_in_file_order(g, m, body, nroots, cells);
  cudaSetDevice(m->device);
  // room for the leaves that the grid does not have yet, at most all; what cannot be had
  // now may not be needed, and otherwise the pools grow on demand
  if (core_reserve(m, leaves.size(), nroots)) m->err.clear();
  BXG_CUDA(m, m->s_in.ensure(size_t(p - body)));
  BXG_CUDA(m, m->s_in2.ensure(leaves.size() * sizeof(FileLeaf)));
  BXG_CUDA(m, cudaMemcpyAsync(m->s_in.p, body, size_t(p - body), cudaMemcpyHostToDevice,
                              m->stream));
  BXG_CUDA(m, cudaMemcpyAsync(m->s_in2.p, leaves.data(), leaves.size() * sizeof(FileLeaf),
                              cudaMemcpyHostToDevice, m->stream));
  const uint32_t nl32 = uint32_t(leaves.size());
  const unsigned blocks = (nl32 + 7) / 8;
  const FileLeaf* dl = m->s_in2.as<FileLeaf>();
  const uint8_t* db = m->s_in.as<uint8_t>();
  return run_with_growth(m, [&]() -> int {
    switch (m->dm.esz) {
      case 0: k_file_read<0><<<blocks, 256, 0, m->stream>>>(m->dm, dl, nl32, db); break;
      case 1: k_file_read<1><<<blocks, 256, 0, m->stream>>>(m->dm, dl, nl32, db); break;
      case 2: k_file_read<2><<<blocks, 256, 0, m->stream>>>(m->dm, dl, nl32, db); break;
      case 4: k_file_read<4><<<blocks, 256, 0, m->stream>>>(m->dm, dl, nl32, db); break;
      default: k_file_read<8><<<blocks, 256, 0, m->stream>>>(m->dm, dl, nl32, db); break;
    }
    BXG_LAUNCHED(m);
    return BXG_OK;
  });
}
