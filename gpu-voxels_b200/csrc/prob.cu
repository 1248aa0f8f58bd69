// ProbVoxelMap (one int8 log-odds occupancy per voxel) and its merge into a
// DistanceVoxelMap, the producer of EDT obstacles from probabilistic sensor
// fusion in gpu-voxels.
//   insert: kernelInsertGlobalPointCloud<ProbabilisticVoxel>
//           (GV/voxelmap/kernels/VoxelMapOperations.hpp:241-264) with
//           ProbabilisticVoxel::insert / updateOccupancy
//           (GV/voxel/ProbabilisticVoxel.hpp:44-100)
//   merge:  DistanceVoxelMap::mergeOccupied (GV/voxelmap/DistanceVoxelMap.hpp:109-136,
//           operators GV/voxelmap/DistanceVoxelMap.h:92-134)
// The reference updates a voxel with a plain read-modify-write, so points
// that share a voxel within one call can lose updates.  Here every point's
// update is applied (a compare-and-swap on the voxel's 32-bit word): the
// updates of one call are all the same saturating step, so the result does
// not depend on their order.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gvx_internal.cuh"

namespace gvx {
namespace {

// updateOccupancy for `meaning`, `times` times (constants
// GV/helpers/common_defines.h:50-63,154-161).  The steps go one way, so
// clamping once at the end equals clamping after each.
__device__ __forceinline__ int prob_steps(int cur, int mode, int delta, int times) {
  if (times == 0) return cur;
  if (mode == 0) return -128;  // eBVM_UNKNOWN / eBVM_UNDEFINED / unused meanings
  const int from = cur == -128 ? 0 : cur;  // an unknown voxel starts at probability 0.5
  return min(max(from + delta * times, -127), 127);
}

// The lanes of a warp whose voxels share a 32-bit word apply their updates with
// one compare-and-swap by the first of them: points of a sensor frame that
// follow each other mostly fall in one voxel, and a lane of its own for each
// made them retry against each other, an L2 round trip per try (307k points of
// four depth images: 23.4 us, now 8.6).  Where no lane's update changes its voxel
// (the updates of a call go one way, so a saturated voxel stays so) the warp has
// nothing to group: a map that has settled is only read (3M random points into a
// settled 256^3 map 20 us, 38 with the grouping; a fresh one 63).
__global__ void pvm_insert_kernel(uint32_t* __restrict__ words, uint32_t X, uint32_t Y, uint32_t Z, float side,
                                  const float* __restrict__ xyz, uint64_t n, int mode, int delta,
                                  uint32_t* __restrict__ outside) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  bool out = false;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < n; i0 += stride) {
    const uint64_t i = i0 + lane;
    uint32_t word = 0xffffffffu;  // no word: at most 2^28 of them
    int byte = 0;
    uint32_t old = 0u;
    bool moves = false;  // the lane's own update would change the voxel
    if (i < n) {
      const uint32_t x = coord_to_voxel(__ldg(xyz + 3 * i), side), y = coord_to_voxel(__ldg(xyz + 3 * i + 1), side),
                     z = coord_to_voxel(__ldg(xyz + 3 * i + 2), side);
      if (x < X && y < Y && z < Z) {
        const uint32_t id = (z * Y + y) * X + x;  // below 2^30
        word = id >> 2;
        byte = (int)(id & 3u);
        old = *reinterpret_cast<volatile uint32_t*>(words + word);
        const int cur = (int)(int8_t)(old >> (8 * byte));
        moves = prob_steps(cur, mode, delta, 1) != cur;
      } else {
        out = true;
      }
    }
    if (!__any_sync(0xffffffffu, moves)) continue;
    const unsigned same = __match_any_sync(0xffffffffu, word);
    const unsigned b0 = __ballot_sync(0xffffffffu, byte & 1), b1 = __ballot_sync(0xffffffffu, byte & 2);
    if (word != 0xffffffffu && __ffs(same) - 1 == lane) {
      const int times[4] = {__popc(same & ~b1 & ~b0), __popc(same & ~b1 & b0), __popc(same & b1 & ~b0), __popc(same & b1 & b0)};
      uint32_t* w = words + word;
      for (;;) {  // ends: each retry follows another thread's successful swap
        uint32_t upd = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          upd |= (uint32_t)(uint8_t)(int8_t)prob_steps((int)(int8_t)(old >> (8 * k)), mode, delta, times[k]) << (8 * k);
        if (upd == old) break;
        const uint32_t seen = atomicCAS(w, old, upd);
        if (seen == old) break;
        old = seen;
      }
    }
  }
  if (outside != nullptr && __any_sync(0xffffffffu, out) && lane == 0) *outside = 1u;
}

// 16 voxels per thread step: one 16-byte load of occupancies; occupied voxels
// get the site of their own coordinates plus the offset (32-bit wrap, as the
// reference's DistanceVoxel(Vector3ui) constructor, GV/voxel/DistanceVoxel.hpp:61-65).
__global__ void merge_occupied_kernel(uint32_t* __restrict__ dvm, const int8_t* __restrict__ pvm, uint32_t X, uint32_t Y,
                                      uint64_t n, uint32_t ox, uint32_t oy, uint32_t oz, int thr) {
  const uint64_t n16 = n / 16;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  auto put = [&](uint64_t id64) {
    const uint32_t id = (uint32_t)id64, row = id / X, x = id - row * X, z = row / Y, y = row - z * Y;  // below 2^30
    dvm[id] = (x + ox) | ((y + oy) << 10) | ((z + oz) << 20);
  };
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(pvm) + i);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if ((int)(int8_t)(w[k >> 2] >> ((k & 3) * 8)) > thr) put(i * 16 + k);
  }
  for (uint64_t id = n16 * 16 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; id < n; id += stride)
    if ((int)pvm[id] > thr) put(id);
}

unsigned grid_for(uint64_t n, int threads) {
  const int sms = device_sms();
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + threads - 1) / threads, (uint64_t)sms * 16));
}

}  // namespace

int prob_threshold(float val) {  // ProbabilisticVoxel::floatToProbability, GV/voxel/ProbabilisticVoxel.h:40-45
  float tmp = std::max(std::min(1.0f, val), 0.0f);
  tmp = (tmp * (127.0f - (-127.0f))) + (-127.0f);
  return (int)(int8_t)tmp;
}

cudaError_t launch_pvm_insert(int8_t* d_vox, gvx_dims d, float side, const float* d_xyz, uint64_t n, uint32_t meaning,
                              uint32_t* d_outside, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  int mode = 1, delta = 0;
  if (meaning == 0) delta = -10;                         // eBVM_FREE: sensor model free
  else if (meaning == 1 || meaning == 2) delta = 72;     // eBVM_OCCUPIED, eBVM_COLLISION: sensor model occupied
  else if (meaning >= 4 && meaning <= 254) delta = (int)meaning - 129;  // eBVM_SWEPT_VOLUME range as probability
  else mode = 0;                                         // eBVM_UNKNOWN, eBVM_UNDEFINED
  pvm_insert_kernel<<<grid_for(n, 256), 256, 0, s>>>(reinterpret_cast<uint32_t*>(d_vox), d.x, d.y, d.z, side, d_xyz, n,
                                                     mode, delta, d_outside);
  return cudaGetLastError();
}

cudaError_t launch_merge_occupied(uint32_t* d_dvm, const int8_t* d_pvm, gvx_dims d, const uint32_t off[3], float threshold,
                                  cudaStream_t s) {
  const uint64_t n = num_voxels(d);
  merge_occupied_kernel<<<grid_for(n / 16 + 1, 256), 256, 0, s>>>(d_dvm, d_pvm, d.x, d.y, n, off[0], off[1], off[2],
                                                                   prob_threshold(threshold));
  return cudaGetLastError();
}

}  // namespace gvx
