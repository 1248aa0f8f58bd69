// Voxel list building by a bitmap of the reference map: make_unique
// (GV/voxellist/TemplateVoxelList.hpp:143-212) without a sort.
//
// insertPointCloud keeps a list's ids sorted and unique.  Ids are voxel
// numbers, so one bit per voxel holds the merged set already sorted and unique:
// mark the list's own ids and the points' ids, count the bits per 1024 words,
// scan the counts, and write the ids of the set bits in order.  An entry's
// voxel is the list's old voxel, found back by the rank of its bit, with the new
// meaning set where a point fell.
//
// That holds for ascending ids inside the map.  The ids lie in storage that a
// caller may write (gvx_blist_data), so the mark kernel checks them, uses none
// that fails, and reports it beside the merged length: the sort takes the list
// then.
//
// What bounds it: launches (seven short ones and one wait) while the map has
// few million voxels; then the bitmap, read twice after it is cleared.  The sort
// of (id, index) pairs it replaces (radix sort, run heads, scan, merge, two
// waits) took 17 launches: clear, insert of 200k points into a 256^3 list,
// collide and read back took 214 us, now 119.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gvx_internal.cuh"

namespace gvx {
namespace {

constexpr int kTileWords = 1024;  // bitmap words per block of 256 threads
constexpr uint32_t kOutside = 0xffffffffu;

// Old ids and points to bits; keys[i] = point i's id, kOutside out of bounds
// (remove_out_of_bounds, TemplateVoxelList.hpp:318-341).  *unusable is set
// where an old id is no voxel of the map or not above the one before it.
__global__ void list_mark_kernel(const float* __restrict__ xyz, uint64_t n, gvx_dims d, float side,
                                 const uint32_t* __restrict__ old_ids, uint64_t n_old, uint32_t* __restrict__ keys,
                                 uint32_t* __restrict__ bits, uint32_t* __restrict__ unusable) {
  const uint64_t total = n_old + n;
  const uint32_t n_vox = d.x * d.y * d.z;  // below 2^30
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t id;
    if (i < n_old) {
      id = old_ids[i];
      if (id >= n_vox || (i > 0 && old_ids[i - 1] >= id)) {
        *unusable = 1u;
        id = kOutside;
      }
    } else {
      const uint64_t p = i - n_old;
      const uint32_t x = coord_to_voxel(xyz[3 * p], side), y = coord_to_voxel(xyz[3 * p + 1], side),
                     z = coord_to_voxel(xyz[3 * p + 2], side);
      id = (x < d.x && y < d.y && z < d.z) ? z * d.x * d.y + y * d.x + x : kOutside;
      keys[p] = id;
    }
    if (id != kOutside) atomicOr(bits + (id >> 5), 1u << (id & 31));
  }
}

// Thread t of a tile owns words 4 t .. 4 t + 3.
__device__ __forceinline__ uint4 tile_words(const uint32_t* __restrict__ bits, uint64_t n_words, uint64_t w) {
  if (w + 4 <= n_words) return __ldg(reinterpret_cast<const uint4*>(bits + w));
  uint4 v = make_uint4(0, 0, 0, 0);
  if (w < n_words) v.x = __ldg(bits + w);
  if (w + 1 < n_words) v.y = __ldg(bits + w + 1);
  if (w + 2 < n_words) v.z = __ldg(bits + w + 2);
  return v;
}

// Exclusive prefix of c over the block's 256 threads; the sum in *total.
__device__ __forceinline__ uint32_t block_prefix(uint32_t c, uint32_t* total) {
  __shared__ uint32_t warp_sum[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  uint32_t before = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) before += warp_sum[w];
    sum += warp_sum[w];
  }
  *total = sum;
  return before + inc - c;
}

__global__ void __launch_bounds__(256) bits_count_kernel(const uint32_t* __restrict__ bits, uint64_t n_words,
                                                         uint32_t* __restrict__ tiles) {
  const uint4 v = tile_words(bits, n_words, (uint64_t)blockIdx.x * kTileWords + 4 * threadIdx.x);
  uint32_t sum;
  block_prefix(__popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w), &sum);
  if (threadIdx.x == 0) tiles[blockIdx.x] = sum;
}

// Exclusive scan of the tile counts by one block; the total goes to tiles[n]
// and beside it, for one read-back, the mark kernel's flag.
__global__ void __launch_bounds__(1024) tiles_scan_kernel(uint32_t* __restrict__ tiles, uint32_t n,
                                                          const uint32_t* __restrict__ unusable) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  for (uint32_t base = 0; base < n; base += 1024) {
    const uint32_t i = base + threadIdx.x, c = i < n ? tiles[i] : 0u;
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    __syncthreads();  // carry, and the sums of the round before
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    uint32_t before = carry;
    for (int w = 0; w < warp; ++w) before += warp_sum[w];
    if (i < n) tiles[i] = before + inc - c;
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + inc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    tiles[n] = carry;
    tiles[n + 1] = *unusable;
  }
}

// Ids of the tile's bits in order and `fill` for each of their voxels; ranks
// (optional): the rank of each word's first bit.
__global__ void __launch_bounds__(256) bits_emit_kernel(const uint32_t* __restrict__ bits, uint64_t n_words,
                                                        const uint32_t* __restrict__ tiles, uint4 fill_lo, uint4 fill_hi,
                                                        uint32_t* __restrict__ ids, uint4* __restrict__ vox,
                                                        uint32_t* __restrict__ ranks) {
  const uint64_t w0 = (uint64_t)blockIdx.x * kTileWords + 4 * threadIdx.x;
  const uint4 v = tile_words(bits, n_words, w0);
  const uint32_t word[4] = {v.x, v.y, v.z, v.w};
  uint32_t sum;
  const uint32_t base = tiles[blockIdx.x];
  uint32_t k = base + block_prefix(__popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w), &sum);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (ranks != nullptr && word[i]) ranks[w0 + i] = k;
    for (uint32_t m = word[i]; m; m &= m - 1) ids[k++] = (uint32_t)(w0 + i) * 32u + (uint32_t)__ffs(m) - 1u;
  }
  for (uint32_t i = threadIdx.x; i < 2 * sum; i += 256) vox[2 * (uint64_t)base + i] = (i & 1) ? fill_hi : fill_lo;
}

__device__ __forceinline__ uint64_t rank_of(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ ranks, uint32_t id) {
  return (uint64_t)ranks[id >> 5] + __popc(bits[id >> 5] & ((1u << (id & 31)) - 1u));
}

// The old entries' voxels at their new places (an unusable id has none).
__global__ void list_move_kernel(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ ranks,
                                 const uint32_t* __restrict__ old_ids, const uint4* __restrict__ old_vox, uint64_t n_old,
                                 uint4* __restrict__ vox, const uint32_t* __restrict__ unusable) {
  if (*unusable != 0u) return;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_old; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = rank_of(bits, ranks, old_ids[i]);
    vox[2 * k] = old_vox[2 * i];
    vox[2 * k + 1] = old_vox[2 * i + 1];
  }
}

// The new points' meaning in their entries.
__global__ void list_meaning_kernel(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ ranks,
                                    const uint32_t* __restrict__ keys, uint64_t n, uint32_t meaning,
                                    uint32_t* __restrict__ vox) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t id = keys[i];
    if (id != kOutside) atomicOr(vox + rank_of(bits, ranks, id) * kBitVoxelWords + (meaning >> 5), 1u << (meaning & 31));
  }
}

unsigned grid_for(uint64_t n) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)device_sms() * 16));
}

uint64_t align64(uint64_t words) { return (words + 63) / 64 * 64; }
uint64_t bitmap_words(gvx_dims d) { return (num_voxels(d) + 31) / 32; }
uint64_t bitmap_tiles(gvx_dims d) { return (bitmap_words(d) + kTileWords - 1) / kTileWords; }

// The work area: bits and behind them the flag, tile counts with the merged
// length and the flag again, the points' ids, and (for a list with entries) ranks.
struct Layout {
  uint64_t tiles, keys, ranks, words;
  Layout(gvx_dims d, uint64_t n_old, uint64_t n)
      : tiles(align64(bitmap_words(d) + 1)),
        keys(tiles + align64(bitmap_tiles(d) + 2)),
        ranks(keys + align64(n)),
        words(ranks + (n_old ? bitmap_words(d) : 0)) {}
};

}  // namespace

uint64_t list_bits_work_words(gvx_dims d, uint64_t n_old, uint64_t n) { return Layout(d, n_old, n).words; }

cudaError_t launch_list_mark(uint32_t* d_work, gvx_dims d, float side, const float* d_xyz, uint64_t n, const uint32_t* d_old,
                             uint64_t n_old, const uint32_t** d_result, cudaStream_t s) {
  const Layout w(d, n_old, n);
  uint32_t *bits = d_work, *unusable = bits + bitmap_words(d), *tiles = d_work + w.tiles;
  const uint32_t nt = (uint32_t)bitmap_tiles(d);
  *d_result = tiles + nt;
  const cudaError_t e = cudaMemsetAsync(bits, 0, (bitmap_words(d) + 1) * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  list_mark_kernel<<<grid_for(n_old + n), 256, 0, s>>>(d_xyz, n, d, side, d_old, n_old, d_work + w.keys, bits, unusable);
  bits_count_kernel<<<nt, 256, 0, s>>>(bits, bitmap_words(d), tiles);
  tiles_scan_kernel<<<1, 1024, 0, s>>>(tiles, nt, unusable);
  return cudaGetLastError();
}

cudaError_t launch_list_emit(uint32_t* d_work, gvx_dims d, uint64_t n, const uint32_t* d_old, const uint8_t* d_old_vox,
                             uint64_t n_old, uint32_t meaning, uint32_t* d_ids, uint8_t* d_vox, cudaStream_t s) {
  const Layout w(d, n_old, n);
  const uint32_t *bits = d_work, *unusable = bits + bitmap_words(d);
  uint32_t* ranks = n_old ? d_work + w.ranks : nullptr;
  uint32_t f[kBitVoxelWords] = {};
  if (n_old == 0) f[meaning >> 5] = 1u << (meaning & 31);  // every entry holds a new point
  bits_emit_kernel<<<(unsigned)bitmap_tiles(d), 256, 0, s>>>(bits, bitmap_words(d), d_work + w.tiles,
                                                             make_uint4(f[0], f[1], f[2], f[3]),
                                                             make_uint4(f[4], f[5], f[6], f[7]), d_ids,
                                                             reinterpret_cast<uint4*>(d_vox), ranks);
  if (n_old) {
    list_move_kernel<<<grid_for(n_old), 256, 0, s>>>(bits, ranks, d_old, reinterpret_cast<const uint4*>(d_old_vox), n_old,
                                                     reinterpret_cast<uint4*>(d_vox), unusable);
    list_meaning_kernel<<<grid_for(n), 256, 0, s>>>(bits, ranks, d_work + w.keys, n, meaning,
                                                    reinterpret_cast<uint32_t*>(d_vox));
  }
  return cudaGetLastError();
}

}  // namespace gvx
