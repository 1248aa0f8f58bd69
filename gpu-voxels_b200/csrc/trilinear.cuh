// Trilinear distance field over an EDT'd DistanceVoxel map (device helpers
// shared by the continuous-query kernels and the batched schedule).
//
// Corner value D(i,j,k) = sqrt(squaredObstacleDistance) in voxel units at
// voxel centres (i + 0.5) * side (getVoxelCenter,
// GV/voxelmap/kernels/VoxelMapOperations.h:175-182); D = sqrt(INT32_MAX) where
// the map holds no site.  The interpolant is trilinear on the centre lattice,
// points are clamped to it (zero gradient along a clamped axis).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "gvx_internal.cuh"

namespace gvx {

struct MapView {
  const uint32_t* vox;
  int X, Y, Z;
  float side;
  bool aligned16;  // vox on a 16-byte boundary (the corner-pair loads below need it)
  uint64_t n;      // voxels in the map (a 16-byte word is read only when it lies inside)
};

// Distance (voxel units) from lattice point (i, j, k) to the site `v` holds.
__device__ __forceinline__ float corner_value(uint32_t v, int i, int j, int k) {
  const int ox = (int)dv_x(v), oy = (int)dv_y(v), oz = (int)dv_z(v);
  if (ox == (int)kUninit || oy == (int)kUninit || oz == (int)kUninit) return sqrtf((float)kMaxObstacleDistance);
  const int dx = i - ox, dy = j - oy, dz = k - oz;
  return sqrtf((float)(dx * dx + dy * dy + dz * dz));
}

// The two corners (i0, j, k) and (i1, j, k) of a cell edge along x.  They
// are neighbours in memory (i1 = i0 + 1, or i1 = i0 on a one-voxel axis);
// when both lie in one aligned 16-byte word (3 of 4 positions) a single
// 16-byte load fetches them, so a random-order query touches about 5 L1
// lines per point instead of 8 -- the queries are bound by those gathers.
__device__ __forceinline__ void corner_pair(const MapView& m, int i0, int i1, int j, int k, float& d0, float& d1) {
  const uint64_t idx = ((uint64_t)k * m.Y + j) * m.X + i0;
  const int o = (int)(idx & 3u);
  uint32_t v0, v1;
  if (m.aligned16 && i1 == i0 + 1 && o != 3 && idx - o + 4 <= m.n) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(m.vox + (idx - o)));
    v0 = o == 0 ? q.x : (o == 1 ? q.y : q.z);
    v1 = o == 0 ? q.y : (o == 1 ? q.z : q.w);
  } else {
    v0 = __ldg(m.vox + idx);
    v1 = __ldg(m.vox + idx + (uint64_t)(i1 - i0));
  }
  d0 = corner_value(v0, i0, j, k);
  d1 = corner_value(v1, i1, j, k);
}

// Lattice coordinate along one axis: u = p/side - 0.5 clamped to [0, n-1];
// returns the lower corner, the fraction and whether the axis is free.  The
// fraction is taken from the residual p - (i0 + 0.5) * side (one fused
// rounding) rather than from u, which keeps it accurate far from the origin.
__device__ __forceinline__ void axis_setup(float p, float side, int n, int& i0, int& i1, float& f, bool& free_axis) {
  const float u = __fsub_rn(__fdiv_rn(p, side), 0.5f);
  const float hi = (float)(n - 1);
  free_axis = (u >= 0.0f) && (u <= hi);
  const float uc = fminf(fmaxf(u, 0.0f), hi);  // NaN -> 0
  i0 = (int)floorf(uc);
  if (free_axis) {
    // choose the cell by the sign of the exact residual, not the rounded u
    if (i0 > 0 && fmaf(-((float)i0 + 0.5f), side, p) < 0.0f) --i0;
    else if (i0 < n - 1 && fmaf(-((float)i0 + 1.5f), side, p) >= 0.0f) ++i0;
  }
  i0 = min(i0, max(n - 2, 0));
  i1 = min(i0 + 1, n - 1);
  if (free_axis) {
    f = __fdiv_rn(fmaf(-((float)i0 + 0.5f), side, p), side);
    f = fminf(fmaxf(f, 0.0f), 1.0f);
  } else {
    f = uc - (float)i0;
  }
}

// p / side - 0.5 in double, with inv = 1 / side rounded: the quotient is p * inv
// with one residual correction (P. Markstein, IBM J. Res. Develop. 34(1), 1990)
// in place of three FP64 divides per point.  It is the divide's: p * inv is within
// 2 ulp of p / side, so the residual is exact in one fma (side has 24 significant
// bits), and the second fma's exact value is off by 2^-51 ulp at most, where a
// quotient by 24 bits lies 2^-25 ulp or more from a rounding midpoint.  An
// infinity, and what is far beyond any map, stays as it is.
// gvx_check_query_arithmetic compares it with the divide.
__device__ __forceinline__ double lattice_coord(double p, float side, double inv) {
  const double q0 = p * inv;
  return (fabs(q0) < 1e300 ? fma(fma(-q0, (double)side, p), inv, q0) : q0) - 0.5;
}

// The same split of an FP64 position (sphere centres from the FP64 forward
// kinematics): cell and fraction come from p / side - 0.5 in double, so only
// the fraction (in [0, 1]) is rounded to float -- an FP32 position alone would
// carry up to half an ulp of p (1.2e-5 voxel at 2.56 m with 1 cm voxels).
__device__ __forceinline__ void axis_setup(double p, float side, double inv, int n, int& i0, int& i1, float& f,
                                           bool& free_axis) {
  const double u = lattice_coord(p, side, inv);
  const double hi = (double)(n - 1);
  free_axis = (u >= 0.0) && (u <= hi);
  const double uc = fmin(fmax(u, 0.0), hi);  // NaN -> 0
  i0 = min((int)floor(uc), max(n - 2, 0));
  i1 = min(i0 + 1, n - 1);
  f = (float)(uc - (double)i0);
}

struct Tri {
  float d;           // voxel units
  float gx, gy, gz;  // d(distance)/d(position), dimensionless
};

// Trilinear distance and gradient at an FP32 position.  The query kernels
// wait on their gathers (a million random points of a 256^3 map: 27 us, the
// four pair loads alone 24), and this form's 32 registers keep every warp of an
// SM resident; with the corners fetched together and packed arithmetic, as below,
// it needs 48 to 64 registers and took 31 us.
__device__ __forceinline__ Tri trilinear(const MapView& m, float px, float py, float pz) {
  int i0, i1, j0, j1, k0, k1;
  float fx, fy, fz;
  bool ax, ay, az;
  axis_setup(px, m.side, m.X, i0, i1, fx, ax);
  axis_setup(py, m.side, m.Y, j0, j1, fy, ay);
  axis_setup(pz, m.side, m.Z, k0, k1, fz, az);
  float d000, d100, d010, d110, d001, d101, d011, d111;
  corner_pair(m, i0, i1, j0, k0, d000, d100);
  corner_pair(m, i0, i1, j1, k0, d010, d110);
  corner_pair(m, i0, i1, j0, k1, d001, d101);
  corner_pair(m, i0, i1, j1, k1, d011, d111);
  // interpolate along x, then y, then z
  const float e00 = fmaf(fx, d100 - d000, d000), e10 = fmaf(fx, d110 - d010, d010);
  const float e01 = fmaf(fx, d101 - d001, d001), e11 = fmaf(fx, d111 - d011, d011);
  const float g0 = fmaf(fy, e10 - e00, e00), g1 = fmaf(fy, e11 - e01, e01);
  Tri t;
  t.d = fmaf(fz, g1 - g0, g0);
  // partial derivatives of the interpolant in lattice units
  const float sx0 = fmaf(fy, (d110 - d010) - (d100 - d000), d100 - d000);
  const float sx1 = fmaf(fy, (d111 - d011) - (d101 - d001), d101 - d001);
  t.gx = ax ? fmaf(fz, sx1 - sx0, sx0) : 0.0f;
  const float sy0 = e10 - e00, sy1 = e11 - e01;
  t.gy = ay ? fmaf(fz, sy1 - sy0, sy0) : 0.0f;
  t.gz = az ? (g1 - g0) : 0.0f;
  return t;
}

// ---------------------------------------------------------------------------
// The same at an FP64 position (inv = 1 / side), for the arm kernels, which
// are bound by instruction issue: neighbouring spheres share cells, so their
// gathers mostly hit L1.  The eight corners are fetched first, by predicated
// loads without a branch between them (with a branch per pair that picked its
// two words at once, each pair waited for its load); the distances are computed
// in packed FP32 pairs, and the sites are checked for the empty value all at
// once.  The same floats as the scalar form.  512 trajectories x 64 waypoints x
// 56 spheres on a 256^3 map: cost 62 -> 50 us, adjoint 76 -> 74 us; 4096
// clearances, the whole call, 13.4 -> 12.3 us.
// ---------------------------------------------------------------------------

// The voxels idx and idx + step (step 1, or 0 on a one-voxel axis) of a map
// row, still in the words they came in: when both lie in one aligned 16-byte
// word of the map (3 of 4 positions) a single 16-byte load fetches them, so a
// random-order query touches about 5 L1 lines instead of 8.
struct CornerPair {
  uint32_t a, b, c, d;
  uint32_t at;  // which two of the four

  __device__ __forceinline__ void load(const uint32_t* vox, uint32_t n_wide, uint32_t idx, uint32_t step) {
    const uint32_t o = idx & 3u;
    const uint32_t wide = (o != 3u && idx < n_wide) ? 1u : 0u;
    at = wide ? o : 0u;
    const uint32_t* first = vox + (idx - at);
    asm("{\n"
        "  .reg .pred p;\n"
        "  setp.ne.u32 p, %6, 0;\n"
        "  @p ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n"
        "  @!p ld.global.nc.u32 %0, [%4];\n"
        "  @!p ld.global.nc.u32 %1, [%5];\n"
        "}\n"
        : "=&r"(a), "=&r"(b), "=&r"(c), "=&r"(d)
        : "l"(__cvta_generic_to_global(first)), "l"(__cvta_generic_to_global(first + step)), "r"(wide));
  }
  __device__ __forceinline__ uint32_t lower() const { return at == 0u ? a : (at == 1u ? b : c); }
  __device__ __forceinline__ uint32_t upper() const { return at == 0u ? b : (at == 1u ? c : d); }
};

// Whether a site may be empty (a field of 1023) or carry bits above its fields,
// over several words: z by the largest word; x and y by adding 1 to each field,
// after which `sum ^ word` has bits 10 and 20 set unless the addition carried
// into them, which it does for a field of 1023 (and for y = 1022 above x = 1023).
struct FarCheck {
  uint32_t ends = 0x00100400u, top = 0u;
  __device__ __forceinline__ void see(uint32_t v) {
    ends &= (v + 0x00100401u) ^ v;
    top = max(top, v);
  }
  __device__ __forceinline__ bool any() const { return ends != 0x00100400u || top >= kUninit << 20; }
};

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// v as a float on top of 2^23: the bits of a field of up to 23 bits below it
// are the value, and differences of two such floats are exact.
__device__ __forceinline__ float biased(uint32_t v) { return __uint_as_float(0x4B000000u | v); }

// Roots of integers, rounded to nearest as sqrtf rounds them: an approximate
// reciprocal root, one exact residual by fma and Markstein's correction
// (P. Markstein, IBM J. Res. Develop. 34(1), 1990).  Bit for bit sqrtf on
// every integer up to 2^24 and on kMaxObstacleDistance, which
// gvx_check_query_arithmetic compares.  2^-60 keeps the reciprocal finite at 0.
__device__ __forceinline__ float2 roots(float2 v) {
  const float2 w = __fadd2_rn(v, both(0x1p-60f));
  float2 y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(w.x));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(w.y));
  const float2 s = __fmul2_rn(v, y);
  const float2 r = __ffma2_rn(__fmul2_rn(s, both(-1.0f)), s, v);
  return __ffma2_rn(r, __fmul2_rn(y, both(0.5f)), s);
}

// Squared distances from the lattice points (i, j, k0) and (i, j, k1) to the
// sites u and v hold.  x is passed as biased(i), y as biased(j << 10), z as
// biased(k << 10) twice.
__device__ __forceinline__ float2 corner_squares(uint32_t u, uint32_t v, float x, float y, float2 z) {
  constexpr uint32_t low = 0x3ffu, mid = 0xffc00u;
  const float2 minus = both(-1.0f);
  const float2 dx = __ffma2_rn(make_float2(biased(u & low), biased(v & low)), minus, both(x));
  const float2 dy = __ffma2_rn(make_float2(biased(u & mid), biased(v & mid)), minus, both(y));
  const float2 dz = __ffma2_rn(make_float2(biased((u >> 10) & mid), biased((v >> 10) & mid)), minus, z);
  // dy and dz carry a factor 2^10; every sum is an integer below 2^22 (times a power of two): exact
  const float2 yz = __ffma2_rn(dy, dy, __fmul2_rn(dz, dz));
  return __ffma2_rn(yz, both(0x1p-20f), __fmul2_rn(dx, dx));
}

// The square of corner_value, for any word.
__device__ __forceinline__ float corner_square(uint32_t v, int i, int j, int k) {
  const int ox = (int)dv_x(v), oy = (int)dv_y(v), oz = (int)dv_z(v);
  if (ox == (int)kUninit || oy == (int)kUninit || oz == (int)kUninit) return (float)kMaxObstacleDistance;
  const int dx = i - ox, dy = j - oy, dz = k - oz;
  return (float)(dx * dx + dy * dy + dz * dz);
}

__device__ __forceinline__ Tri trilinear(const MapView& m, double px, double py, double pz, double inv) {
  int i0, i1, j0, j1, k0, k1;
  float fx, fy, fz;
  bool ax, ay, az;
  axis_setup(px, m.side, inv, m.X, i0, i1, fx, ax);
  axis_setup(py, m.side, inv, m.Y, j0, j1, fy, ay);
  axis_setup(pz, m.side, inv, m.Z, k0, k1, fz, az);
  const uint32_t row = (uint32_t)m.X, layer = row * (uint32_t)m.Y, step = (uint32_t)(i1 - i0);
  const uint32_t to_j1 = (uint32_t)(j1 - j0) * row, to_k1 = (uint32_t)(k1 - k0) * layer;
  const uint32_t n_wide = m.aligned16 && m.X > 1 ? (uint32_t)m.n & ~3u : 0u;  // voxels in whole 16-byte words
  const uint32_t idx = ((uint32_t)k0 * (uint32_t)m.Y + (uint32_t)j0) * row + (uint32_t)i0;
  CornerPair p00, p10, p01, p11;  // by j and k
  p00.load(m.vox, n_wide, idx, step);
  p10.load(m.vox, n_wide, idx + to_j1, step);
  p01.load(m.vox, n_wide, idx + to_k1, step);
  p11.load(m.vox, n_wide, idx + to_j1 + to_k1, step);
  const uint32_t v000 = p00.lower(), v100 = p00.upper(), v010 = p10.lower(), v110 = p10.upper();
  const uint32_t v001 = p01.lower(), v101 = p01.upper(), v011 = p11.lower(), v111 = p11.upper();
  FarCheck check;
  check.see(v000), check.see(v100), check.see(v010), check.see(v110);
  check.see(v001), check.see(v101), check.see(v011), check.see(v111);
  const float x0 = biased((uint32_t)i0), x1 = biased((uint32_t)i1);
  const float y0 = biased((uint32_t)j0 << 10), y1 = biased((uint32_t)j1 << 10);
  const float2 z = make_float2(biased((uint32_t)k0 << 10), biased((uint32_t)k1 << 10));
  // by i and j: the corners at k0 and k1
  float2 d00 = corner_squares(v000, v001, x0, y0, z), d10 = corner_squares(v100, v101, x1, y0, z);
  float2 d01 = corner_squares(v010, v011, x0, y1, z), d11 = corner_squares(v110, v111, x1, y1, z);
  if (check.any()) {
    d00 = make_float2(corner_square(v000, i0, j0, k0), corner_square(v001, i0, j0, k1));
    d10 = make_float2(corner_square(v100, i1, j0, k0), corner_square(v101, i1, j0, k1));
    d01 = make_float2(corner_square(v010, i0, j1, k0), corner_square(v011, i0, j1, k1));
    d11 = make_float2(corner_square(v110, i1, j1, k0), corner_square(v111, i1, j1, k1));
  }
  d00 = roots(d00), d10 = roots(d10), d01 = roots(d01), d11 = roots(d11);
  // interpolate along x, then y, then z
  const float2 minus = both(-1.0f);
  const float2 s0 = __ffma2_rn(d00, minus, d10), s1 = __ffma2_rn(d01, minus, d11);  // slopes along x
  const float2 e0 = __ffma2_rn(both(fx), s0, d00), e1 = __ffma2_rn(both(fx), s1, d01);
  const float2 sy = __ffma2_rn(e0, minus, e1);
  const float2 g = __ffma2_rn(both(fy), sy, e0);
  const float2 sx = __ffma2_rn(both(fy), __ffma2_rn(s0, minus, s1), s0);
  Tri t;
  t.d = fmaf(fz, g.y - g.x, g.x);
  // partial derivatives of the interpolant in lattice units
  t.gx = ax ? fmaf(fz, sx.y - sx.x, sx.x) : 0.0f;
  t.gy = ay ? fmaf(fz, sy.y - sy.x, sy.x) : 0.0f;
  t.gz = az ? (g.y - g.x) : 0.0f;
  return t;
}

}  // namespace gvx
