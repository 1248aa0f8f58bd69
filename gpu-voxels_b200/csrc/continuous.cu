// Continuous distance queries on an EDT'd DistanceVoxel map (no counterpart
// in gpu-voxels, whose queries stop at integer voxel distances): trilinear
// distance + spatial gradient and its adjoint, sphere-model clearance per arm
// configuration, and a hinge trajectory cost with a hand-written adjoint that
// recomputes the forward kinematics.
//
// Distance field: corner value D(i,j,k) = sqrt(squaredObstacleDistance) in
// voxel units at voxel centres (i + 0.5) * side (getVoxelCenter,
// GV/voxelmap/kernels/VoxelMapOperations.h:175-182); D = sqrt(INT32_MAX) where
// the map holds no site.  The interpolant is trilinear on the centre lattice,
// points are clamped to it (zero gradient along a clamped axis).
//
// Kinematics: the reference's DH convention (DHParameters::convertDHtoM,
// GV/robot/dh_robot/KinematicLink.cu:24-79) chained as
// KinematicChain::setConfiguration (GV/robot/dh_robot/KinematicChain.cu:104-124).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gvx_internal.cuh"
#include "trilinear.cuh"

namespace gvx {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__global__ void trilinear_kernel(MapView m, const float* __restrict__ xyz, uint64_t n, float* __restrict__ dist,
                                 float* __restrict__ grad) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const Tri t = trilinear(m, __ldg(xyz + 3 * i), __ldg(xyz + 3 * i + 1), __ldg(xyz + 3 * i + 2));
    dist[i] = t.d * m.side;
    if (grad != nullptr) {
      grad[3 * i] = t.gx;
      grad[3 * i + 1] = t.gy;
      grad[3 * i + 2] = t.gz;
    }
  }
}

__global__ void trilinear_bwd_kernel(MapView m, const float* __restrict__ xyz, uint64_t n,
                                     const float* __restrict__ gout, float* __restrict__ gxyz) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const Tri t = trilinear(m, __ldg(xyz + 3 * i), __ldg(xyz + 3 * i + 1), __ldg(xyz + 3 * i + 2));
    const float g = __ldg(gout + i);
    gxyz[3 * i] = g * t.gx;
    gxyz[3 * i + 1] = g * t.gy;
    gxyz[3 * i + 2] = g * t.gz;
  }
}

// ---------------------------------------------------------------------------
// Forward kinematics: frames F_0 = base, F_{j+1} = F_j * A_j(q_j),
// A_j = Rz(theta_j + q_j) Tz(d_j) Tx(a_j) Rx(alpha_j).  Link j spans origin
// o_j -> o_{j+1}; joint j turns about z_j (third column of F_j) through o_j.
// The chain runs in FP64, and sphere centres are formed in FP64 and rounded
// once to FP32: an FP32 chain of seven frames alone puts the centres ~1e-6 m
// off, 1e-4 voxel at 1 cm.  The distance queries themselves stay FP32.
//
// A block does the kinematics of all its configurations before its spheres:
// one thread per (configuration, joint) for the sines and cosines, one per
// (configuration, frame row) for the chain (row i of F_{j+1} needs row i of
// F_j alone).  With one lane of a warp walking the whole chain of the warp's
// configuration the rest of the warp idled through seven FP64 sincos and matrix
// products: cost and adjoint of 512 trajectories x 64 waypoints x 56 spheres
// through autograd took 306 us, then 146; 4096 clearances 22.5 us, then 13.4.
// The rest is bound by the queries' arithmetic (127 and 12.3 us with their packed form).
// ---------------------------------------------------------------------------
constexpr int kWarpsPerBlock = 8;
constexpr int kThreads = kWarpsPerBlock * 32;
constexpr int kMaxBlockConfigs = 64;
// Blocks of an SM the clearance and cost kernels keep room for: four (64
// registers) take 512 trajectories at once, where three (75 to 80 registers)
// left a second wave (cost 52 us against 50, 4096 clearances 11.9 against 10.3),
// though at 64 they spill 36 and 12 bytes a thread.
// The adjoint's FP64 sums spill at 64 and at 80 registers (91 us); left at 124 it takes 74.
constexpr int kArmBlocks = 4;

// Shared memory of a block for `configs` configurations.
struct ArmSmem {
  double* pose;    // per configuration: origins o_0 .. o_J, then axes z_0 .. z_{J-1}, 3 doubles each
  double* turn;    // per configuration and joint: sin, cos of theta + q
  double* twist;   // per joint: sin, cos of alpha
  float *t, *r;    // per sphere
  int* link;
};

__host__ __device__ __forceinline__ int pose_doubles(int J) { return 3 * (2 * J + 1); }
__host__ __device__ __forceinline__ size_t arm_smem_bytes(int J, int spheres, int configs) {
  return sizeof(double) * ((size_t)configs * (pose_doubles(J) + 2 * J) + 2 * J) + (size_t)spheres * 12;
}

// The block's view of the arm: alpha's sines and the sphere model, copied from
// the kernel's parameters (whose constant bank serves one address at a time).
// Synchronised by the first fk_block.
__device__ __forceinline__ ArmSmem arm_setup(const gvx_arm& arm, int configs, double* smem) {
  const int J = arm.n_joints, S = arm.n_spheres;
  ArmSmem a;
  a.pose = smem;
  a.turn = a.pose + (size_t)configs * pose_doubles(J);
  a.twist = a.turn + (size_t)configs * 2 * J;
  a.t = reinterpret_cast<float*>(a.twist + 2 * J);
  a.r = a.t + S;
  a.link = reinterpret_cast<int*>(a.r + S);
  for (int j = threadIdx.x; j < J; j += kThreads) sincos((double)arm.alpha[j], a.twist + 2 * j, a.twist + 2 * j + 1);
  for (int s = threadIdx.x; s < S; s += kThreads) {
    a.t[s] = arm.t[s];
    a.r[s] = arm.r[s];
    a.link[s] = arm.link[s];
  }
  return a;
}

// Poses of configurations q[0 .. n - 1] (J joint angles each).  All threads
// call; the poses are ready on return, and the caller synchronises before the next call.
__device__ __forceinline__ void fk_block(const gvx_arm& arm, const ArmSmem& a, const float* __restrict__ q, int n) {
  const int J = arm.n_joints;
  for (int i = threadIdx.x; i < n * J; i += kThreads)
    sincos((double)arm.theta[i % J] + (double)__ldg(q + i), a.turn + 2 * i, a.turn + 2 * i + 1);
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * n; i += kThreads) {
    const int w = i / 3, row = i - 3 * w;
    double* o = a.pose + (size_t)w * pose_doubles(J) + row;
    double* z = o + 3 * (J + 1);
    const double* turn = a.turn + (size_t)w * 2 * J;
    double r0 = arm.base[4 * row], r1 = arm.base[4 * row + 1], r2 = arm.base[4 * row + 2], origin = arm.base[4 * row + 3];
    for (int j = 0; j < J; ++j) {
      o[3 * j] = origin;
      z[3 * j] = r2;
      const double st = turn[2 * j], ct = turn[2 * j + 1], sa = a.twist[2 * j], ca = a.twist[2 * j + 1];
      const double l = arm.a[j];
      origin = r0 * (l * ct) + r1 * (l * st) + r2 * (double)arm.d[j] + origin;
      const double n0 = r0 * ct + r1 * st, n1 = r0 * (-st * ca) + r1 * (ct * ca) + r2 * sa,
                   n2 = r0 * (st * sa) + r1 * (-ct * sa) + r2 * ca;
      r0 = n0;
      r1 = n1;
      r2 = n2;
    }
    o[3 * J] = origin;
  }
  __syncthreads();
}

// Sphere centre in FP64 (the distance query splits it into cell and fraction
// in double, and the adjoint's moment arms use it as it is).
__device__ __forceinline__ void sphere_centre(const ArmSmem& a, const double* pose, int s, double c[3]) {
  const double* o = pose + 3 * a.link[s];
  const double t = a.t[s];
#pragma unroll
  for (int i = 0; i < 3; ++i) c[i] = fma(t, o[3 + i] - o[i], o[i]);
}

// Min clearance per configuration; one warp per configuration, lanes over spheres.
__global__ void __launch_bounds__(kThreads, kArmBlocks) sphere_clearance_kernel(MapView m, gvx_arm arm, const float* __restrict__ q,
                                                                    uint64_t n_cfg, int per_block,
                                                                    float* __restrict__ out) {
  extern __shared__ __align__(16) double s_arm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int J = arm.n_joints, S = arm.n_spheres;
  const ArmSmem a = arm_setup(arm, per_block, s_arm);
  const double inv = 1.0 / (double)m.side;
  for (uint64_t c0 = (uint64_t)blockIdx.x * per_block; c0 < n_cfg; c0 += (uint64_t)gridDim.x * per_block) {
    const int n = (int)min((uint64_t)per_block, n_cfg - c0);
    fk_block(arm, a, q + c0 * J, n);
    for (int w = warp; w < n; w += kWarpsPerBlock) {
      const double* pose = a.pose + (size_t)w * pose_doubles(J);
      float best = __int_as_float(0x7f800000);  // +inf
      for (int s = lane; s < S; s += 32) {
        double c[3];
        sphere_centre(a, pose, s, c);
        const Tri t = trilinear(m, c[0], c[1], c[2], inv);
        best = fminf(best, t.d * m.side - a.r[s]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(kFull, best, o));
      if (lane == 0) out[c0 + w] = best;
    }
    __syncthreads();
  }
}

// Hinge cost: one block per trajectory, warp w takes waypoints w, w+8, ...;
// fixed-order reductions keep the result deterministic.
__global__ void __launch_bounds__(kThreads, kArmBlocks) traj_cost_kernel(MapView m, gvx_arm arm, const float* __restrict__ q,
                                                             uint64_t n_traj, uint32_t n_wp, int per_block, float margin,
                                                             float* __restrict__ cost) {
  extern __shared__ __align__(16) double s_arm[];
  __shared__ float s_part[kWarpsPerBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int J = arm.n_joints, S = arm.n_spheres;
  const ArmSmem a = arm_setup(arm, per_block, s_arm);
  const double inv = 1.0 / (double)m.side;
  for (uint64_t traj = blockIdx.x; traj < n_traj; traj += gridDim.x) {
    float acc = 0.0f;
    for (uint32_t w0 = 0; w0 < n_wp; w0 += per_block) {  // per_block is a multiple of the warps
      const int n = (int)min((uint32_t)per_block, n_wp - w0);
      fk_block(arm, a, q + (traj * n_wp + w0) * J, n);
      for (int w = warp; w < n; w += kWarpsPerBlock) {
        const double* pose = a.pose + (size_t)w * pose_doubles(J);
        for (int s = lane; s < S; s += 32) {
          double c[3];
          sphere_centre(a, pose, s, c);
          const Tri t = trilinear(m, c[0], c[1], c[2], inv);
          acc += fmaxf(0.0f, margin - (t.d * m.side - a.r[s]));
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane == 0) s_part[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      float sum = 0.0f;
      for (int i = 0; i < kWarpsPerBlock; ++i) sum += s_part[i];
      cost[traj] = sum;
    }
    __syncthreads();
  }
}

// Sums acc[k] over the warp for every k: kJ values (a power of two) leave the
// sum of value lane / (32 / kJ) in each lane.  A step swaps half of the values
// a lane still holds with its partner, so 8 values take 9 exchanges (40 as one
// butterfly per value); the order of the additions is fixed.
template <int kJ>
__device__ __forceinline__ double sum_transposed(double (&acc)[kJ]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int held = kJ / 2; held >= 1; held >>= 1, o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < held; ++k) {
      const double mine = upper ? acc[k + held] : acc[k], other = upper ? acc[k] : acc[k + held];
      acc[k] = mine + __shfl_xor_sync(kFull, other, o);
    }
  }
  double sum = acc[0];
  for (; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
  return sum;
}

// Adjoint of the hinge cost.  For an active sphere s on link j,
//   d cost / d q_k = -grad d(c_s) . (z_k x (c_s - o_k))   for k <= j.
// One warp per waypoint, FK recomputed: each lane evaluates its spheres once
// and adds every joint's term to a per-joint accumulator in FP64 (the moment
// arm c_s - o_k formed in double, so nothing large cancels); the spatial
// gradient g_s stays FP32 (the trilinear query's own precision).
template <int kJ>  // joints rounded up to 8 or 16
__global__ void __launch_bounds__(kThreads) traj_cost_bwd_kernel(MapView m, gvx_arm arm, const float* __restrict__ q,
                                                                 uint64_t n_traj, uint32_t n_wp, int per_block, float margin,
                                                                 const float* __restrict__ gcost,
                                                                 float* __restrict__ gq) {
  extern __shared__ __align__(16) double s_arm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int J = arm.n_joints, S = arm.n_spheres;
  const ArmSmem a = arm_setup(arm, per_block, s_arm);
  const double inv = 1.0 / (double)m.side;
  const uint64_t n_items = n_traj * n_wp;
  for (uint64_t i0 = (uint64_t)blockIdx.x * per_block; i0 < n_items; i0 += (uint64_t)gridDim.x * per_block) {
    const int n = (int)min((uint64_t)per_block, n_items - i0);
    fk_block(arm, a, q + i0 * J, n);
    for (int w = warp; w < n; w += kWarpsPerBlock) {
      const double* pose = a.pose + (size_t)w * pose_doubles(J);
      const double* axes = pose + 3 * (J + 1);
      double acc[kJ];
#pragma unroll
      for (int k = 0; k < kJ; ++k) acc[k] = 0.0;
      bool touched = false;
      for (int s = lane; s < S; s += 32) {
        double c[3];
        sphere_centre(a, pose, s, c);
        const Tri t = trilinear(m, c[0], c[1], c[2], inv);
        if (margin - (t.d * m.side - a.r[s]) > 0.0f) {
          touched = true;
          const int js = a.link[s];
          const double gx = t.gx, gy = t.gy, gz = t.gz;
#pragma unroll
          for (int k = 0; k < kJ; ++k) {
            if (k > js) break;  // joints beyond the sphere's link do not move it
            const double* o = pose + 3 * k;
            const double* z = axes + 3 * k;
            const double lx = c[0] - o[0], ly = c[1] - o[1], lz = c[2] - o[2];
            acc[k] -= gx * (z[1] * lz - z[2] * ly) + gy * (z[2] * lx - z[0] * lz) + gz * (z[0] * ly - z[1] * lx);
          }
        }
      }
      const double sum = __any_sync(kFull, touched) ? sum_transposed<kJ>(acc) : 0.0;
      const int k = lane / (32 / kJ);
      if (lane % (32 / kJ) == 0 && k < J)
        gq[(i0 + w) * J + k] = (float)((double)__ldg(gcost + (i0 + w) / n_wp) * sum);
    }
    __syncthreads();
  }
}

int sms() { return device_sms(); }

unsigned blocks_for(uint64_t items, uint64_t per_block, uint64_t cap_per_sm) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + per_block - 1) / per_block, (uint64_t)sms() * cap_per_sm));
}

MapView view(const gvx_dvm* m) {
  return MapView{m->d_vox, (int)m->dims.x, (int)m->dims.y, (int)m->dims.z, m->side,
                 (reinterpret_cast<uintptr_t>(m->d_vox) & 15u) == 0, num_voxels(m->dims)};
}

// Every integer up to 2^24, and the distance of an empty corner: roots whose bits
// differ from sqrtf's, each value in both halves of the pair.
__global__ void roots_check_kernel(unsigned long long* __restrict__ mismatches) {
  constexpr int kLast = 1 << 24;
  unsigned long long bad = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= kLast + 1; i += gridDim.x * blockDim.x) {
    const float v = (float)(i <= kLast ? i : kMaxObstacleDistance), w = (float)(kLast - min(i, kLast));
    const float2 r = roots(make_float2(v, w));
    bad += __float_as_uint(r.x) != __float_as_uint(sqrtf(v));
    bad += __float_as_uint(r.y) != __float_as_uint(sqrtf(w));
  }
  if (bad) atomicAdd(mismatches, bad);
}

// 2^28 positions and sides from a counter: positions in and around a map, a few
// ulp around every half of a side (where cells and rounding ties meet), float
// positions, and any bits at all; sides of 1 mm to 1 m and any positive float.
// Counts coordinates whose bits differ from the divide's; beyond 1e299 both have
// to be as far, or no number.
__global__ void lattice_check_kernel(unsigned long long* __restrict__ mismatches) {
  unsigned long long bad = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 28); i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t h = (i + 1) * 0x9E3779B97F4A7C15ull;  // SplitMix64 (Steele, Lea, Flood, OOPSLA 2014)
    h = (h ^ (h >> 30)) * 0xBF58476D1CE4E5B9ull;
    h = (h ^ (h >> 27)) * 0x94D049BB133111EBull;
    h ^= h >> 31;
    const uint64_t g = h * 0xD6E8FEB86659FD93ull;
    float side = __uint_as_float((uint32_t)(g >> 33) % 0x7F7FFFFFu + 1u);
    if (i & 4) side = 0.001f + 0.999f * ((float)(g >> 40) * 0x1p-24f);
    const double unit = (double)(h >> 11) * 0x1p-53;
    double p = __longlong_as_double((long long)h);
    if ((i & 3) == 1) p = (unit * 4096.0 - 1024.0) * (double)side;
    if ((i & 3) == 2) p = __longlong_as_double(__double_as_longlong((double)((h >> 20) % 2050u) * 0.5 * (double)side) + (long long)(h & 7u) - 3);
    if ((i & 3) == 3) p = (float)((unit * 2048.0 - 512.0) * (double)side);
    const double got = lattice_coord(p, side, 1.0 / (double)side), want = p / (double)side - 0.5;
    const bool same = __double_as_longlong(got) == __double_as_longlong(want) || (isnan(got) && isnan(want)) ||
                      (fabs(got) > 1e299 && fabs(want) > 1e299 && signbit(got) == signbit(want));
    bad += !same;
  }
  if (bad) atomicAdd(mismatches, bad);
}

}  // namespace

cudaError_t check_query_arithmetic(unsigned long long* d_mismatches, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(d_mismatches, 0, 2 * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  roots_check_kernel<<<1024, 256, 0, s>>>(d_mismatches);
  lattice_check_kernel<<<4096, 256, 0, s>>>(d_mismatches + 1);
  return cudaGetLastError();
}

cudaError_t launch_trilinear(const gvx_dvm* m, const float* d_xyz, uint64_t n, float* d_dist, float* d_grad, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const QueryConfig q = query_config();
  trilinear_kernel<<<blocks_for(n, q.threads, q.blocks_per_sm), q.threads, 0, s>>>(view(m), d_xyz, n, d_dist, d_grad);
  return cudaGetLastError();
}

cudaError_t launch_trilinear_bwd(const gvx_dvm* m, const float* d_xyz, uint64_t n, const float* d_gout, float* d_gxyz,
                                 cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const QueryConfig q = query_config();
  trilinear_bwd_kernel<<<blocks_for(n, q.threads, q.blocks_per_sm), q.threads, 0, s>>>(view(m), d_xyz, n, d_gout, d_gxyz);
  return cudaGetLastError();
}

namespace {
// Configurations a block takes at a time: as many as leave about 8 blocks per
// SM (their kinematics run side by side), 8 to 64, a multiple of the warps.
int configs_per_block(uint64_t n) {
  const uint64_t each = n / ((uint64_t)sms() * 8 * kWarpsPerBlock) + 1;
  return kWarpsPerBlock * (int)std::min<uint64_t>(each, kMaxBlockConfigs / kWarpsPerBlock);
}

// The dynamic shared memory limit of a kernel, for arms that need more than the
// 48 KB every kernel may use.  The limit is the kernel's, not the call's, so every
// call raises it to the largest arm's size: with its own size a call would lower
// it between another thread's call here and that thread's launch.
template <auto kKernel>
cudaError_t allow_smem(size_t bytes) {
  constexpr auto kLimit = cudaFuncAttributeMaxDynamicSharedMemorySize;
  return bytes <= 48 * 1024 ? cudaSuccess
                            : cudaFuncSetAttribute(kKernel, kLimit, (int)arm_smem_bytes(GVX_MAX_JOINTS, GVX_MAX_SPHERES, kMaxBlockConfigs));
}

template <int kJ>
cudaError_t run_traj_cost_bwd(const gvx_dvm* m, const gvx_arm& arm, const float* d_q, uint64_t n_traj, uint32_t n_wp,
                              float margin, const float* d_gcost, float* d_gq, cudaStream_t s) {
  const int per = configs_per_block(n_traj * n_wp);
  const size_t smem = arm_smem_bytes(arm.n_joints, arm.n_spheres, per);
  const cudaError_t e = allow_smem<traj_cost_bwd_kernel<kJ>>(smem);
  if (e != cudaSuccess) return e;
  traj_cost_bwd_kernel<kJ><<<blocks_for(n_traj * n_wp, per, 16), kThreads, smem, s>>>(view(m), arm, d_q, n_traj, n_wp, per,
                                                                                       margin, d_gcost, d_gq);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_sphere_clearance(const gvx_dvm* m, const gvx_arm& arm, const float* d_q, uint64_t n_cfg, float* d_out,
                                    cudaStream_t s) {
  if (n_cfg == 0) return cudaSuccess;
  const int per = configs_per_block(n_cfg);
  const size_t smem = arm_smem_bytes(arm.n_joints, arm.n_spheres, per);
  const cudaError_t e = allow_smem<sphere_clearance_kernel>(smem);
  if (e != cudaSuccess) return e;
  sphere_clearance_kernel<<<blocks_for(n_cfg, per, 16), kThreads, smem, s>>>(view(m), arm, d_q, n_cfg, per, d_out);
  return cudaGetLastError();
}

cudaError_t launch_traj_cost(const gvx_dvm* m, const gvx_arm& arm, const float* d_q, uint64_t n_traj, uint32_t n_wp,
                             float margin, float* d_cost, cudaStream_t s) {
  if (n_traj == 0) return cudaSuccess;
  const int rounds = (int)std::min<uint64_t>((n_wp + kWarpsPerBlock - 1) / kWarpsPerBlock, kMaxBlockConfigs / kWarpsPerBlock);
  const int per = kWarpsPerBlock * std::max(rounds, 1);
  const size_t smem = arm_smem_bytes(arm.n_joints, arm.n_spheres, per);
  const cudaError_t e = allow_smem<traj_cost_kernel>(smem);
  if (e != cudaSuccess) return e;
  traj_cost_kernel<<<(unsigned)std::min<uint64_t>(n_traj, (uint64_t)sms() * 32), kThreads, smem, s>>>(
      view(m), arm, d_q, n_traj, n_wp, per, margin, d_cost);
  return cudaGetLastError();
}

cudaError_t launch_traj_cost_bwd(const gvx_dvm* m, const gvx_arm& arm, const float* d_q, uint64_t n_traj, uint32_t n_wp,
                                 float margin, const float* d_gcost, float* d_gq, cudaStream_t s) {
  if (n_traj == 0 || n_wp == 0) return cudaSuccess;
  return arm.n_joints <= 8 ? run_traj_cost_bwd<8>(m, arm, d_q, n_traj, n_wp, margin, d_gcost, d_gq, s)
                           : run_traj_cost_bwd<16>(m, arm, d_q, n_traj, n_wp, margin, d_gcost, d_gq, s);
}

}  // namespace gvx
