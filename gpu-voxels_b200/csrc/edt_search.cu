// Exact EDT of maps whose sites all lie in their own voxels (after clearMap
// and insertPointCloud, or voxelize_edt's occupancy bits): the same map as
// the proximate-site sweeps of edt.cu, found by searching every row.
//
// What a pass returns.  devicePBAintersection3DY (GV/voxelmap/kernels/
// VoxelMapOperationsPBA.hpp:265-276) is used only in `top's bisector >= new
// bisector` (phase 2) and `row <= bisector` (phase 3).  At an integer row two
// sites' squared distances are integers, so a bisector that is not an integer
// is at least 1/2046 away from every row (rows are below 1024), while its two
// float roundings move it by less than 2^-12, and an integer bisector is
// computed exactly.  So phase 3's test equals `squared distance to the lower
// site <= squared distance to the upper one`, and a pop in phase 2 removes a
// site only when at every row the site below it is at least as near or the
// new site is nearer.  Row r of a column therefore ends with the site that
// minimises (d_j + (r - j)^2, j), d_j the squared offset of row j's site from
// the column: the nearest site, the lowest row on a tie.  The pair fits one
// 32-bit key, ordered as an unsigned integer: the squared distance (below
// 2^21) in bits 10 and up, j (below 2^9) in bits 1 to 9.
//
// How it is found.  The winner j(r) never decreases with r, so once j is
// known at two rows every row between them looks only at the candidates
// between the two winners.  A block takes 32 columns: 32 consecutive z of one
// (x) plane for pass Y and of one (y) plane for pass X, all keys in shared
// memory (key[row][lane], no bank conflicts).  Its 8 warps first find the
// winners at 8 rows (segment_starts), then each warp refines its eighth of the
// column to every 8th row and then to every row, with one add-and-min per
// candidate and row (a step by 16 rows between the two was 8 % slower: more
// loops, each with its own range to find).  The lanes of a warp share the candidate range (the union of theirs):
// neighbours in z see nearly the same obstacles, so the union is 1.06 .. 1.27
// times a lane's own range at the coarse steps and about 1.7 times at the last
// (512^3 depth scene); with lanes along x, as the sweeps have them, it was up to
// 7.9 times.
//
// What bounds it: instruction issue (67 % of the cycles in pass Y, 60 % in pass X;
// 352^3 depth scene) and the 2-cycle integer pipe (60 % and 57 %; a candidate
// costs one add-and-min, no divide, no per-lane control flow); DRAM is a third
// busy.  Measured on a B200 against the sweeps of edt.cu (whole calls, warm): 512^3
// depth scene 790 us against 1710 (pass Y 345, pass X 429); 128^3 with 50k box
// points 36 against 183 (the sweeps walk 128 rows one after another per pass, here
// 8 warps share a column); 203 x 331 x 157 in three calls 139 against 491; 24 uneven
// maps of 64 to 384 per axis in one batch 1505 against 2606.
//
// The searching loops are kept rolled: unrolled over a warp's rows the code
// outgrew the instruction caches (at 352^3 the largest stall was 'no
// instruction', 4.0 of 10.7 cycles per issue).
//
// Layouts (after the workspace's counters; zw = chunks of 32 z):
//   bits   [zw][X][Y]      bit z & 31 set where the voxel is occupied
//   near   [zw][X][Y]      nearest sites outside the chunk, counted from its
//                          first z: the one below in the low half (kNoneBelow =
//                          none), the one above in the high half (kNoneAbove)
//   field  [zw][Y][X][32]  pass Y's keys (bit 0: the site lies above z)
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "gvx_internal.cuh"

namespace gvx {
namespace {

constexpr unsigned kFullMask = 0xffffffffu;
constexpr int kWarps = 8;
constexpr int kMaxLen = 512;  // longest searched column: a block's keys fill 64 KB
// Real keys stay below 2^31.  A row without a site gets kMissing: adding a
// squared row offset (below 2^28) does not wrap, and the steps that carry a
// key along a segment of 64 rows (`shift_key`) cannot bring it below kNoSite.
constexpr uint32_t kNoSite = 0xC0000000u, kMissing = 0xC4000000u;
// The `least` entry of candidates without a site stands for this key; no real
// key reaches it.
constexpr uint32_t kFar = 0xffffu << 15;
constexpr uint32_t kRowBits = 0x3feu;  // twice the row in a key
// A z offset to a missing site: its square times 1024 is kMissing or above
// (from every z of the chunk), still far enough below 2^32.
constexpr int kNoneBelow = -1792, kNoneAbove = 1823;

__host__ __device__ __forceinline__ int z_chunks(int Z) { return (Z + 31) >> 5; }
__host__ __device__ __forceinline__ uint64_t bits_words(int X, int Y, int Z) { return (uint64_t)z_chunks(Z) * X * Y; }

// Rows per warp (a multiple of 16) of a column of length L.
__host__ __device__ __forceinline__ int seg_rows(int L) { return 16 * ((L + 127) >> 7); }

// Shared memory of a block: keys; weights 1024 d^2, d from 1 - rows to rows;
// winners at the segment starts; 1/32 of the least distance in every 16
// candidates (16 bits); then `extra` words.  At 512 rows a third of an SM's
// shared memory to the byte.
__host__ __device__ __forceinline__ int key_rows(int L) { return (L + 3) & ~3; }
__host__ __device__ __forceinline__ int weight_words(int L) { return 2 * kWarps * seg_rows(L); }
__host__ __device__ __forceinline__ int least_words(int L) { return kWarps * seg_rows(L); }
__host__ __device__ __forceinline__ int search_smem_words(int L, int extra) {
  return key_rows(L) * 32 + weight_words(L) + kWarps * 32 + least_words(L) + extra;
}

// 1024 d^2 for d = -511 .. 512, copied into every block's shared memory (16
// bytes a copy; computing them took 40 instructions of each warp).
struct WeightTable {
  uint32_t w[2 * kMaxLen];
  constexpr WeightTable() : w() {
    for (int i = 0; i < 2 * kMaxLen; ++i) w[i] = (uint32_t)((i - kMaxLen + 1) * (i - kMaxLen + 1)) << 10;
  }
};
__device__ const __align__(16) WeightTable g_weights{};

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

struct Search {
  uint32_t* key;      // this lane's column: key[row * 32]
  const uint32_t* w;  // weight of offset d at w[d]; w[d - 3] is 16-byte aligned for d a multiple of 4
  uint32_t* bnd;      // this lane's winners at the segment starts: bnd[i * 32]
  uint16_t* least;    // this lane's least distance / 32 of candidates 16 g .. 16 g + 15: least[g * 32]
  int L;
};

// The block's tables; the weights arrive with the caller's cp_async_wait_all
// and barrier.
__device__ __forceinline__ Search search_setup(uint32_t* smem, int L, uint32_t** extra) {
  const int lane = threadIdx.x & 31;
  Search s;
  s.L = L;
  s.key = smem + lane;
  uint32_t* w = smem + key_rows(L) * 32;
  const int off = kWarps * seg_rows(L) - 1;  // the word of d = 0; the table's starts at kMaxLen - 1
  for (int i = threadIdx.x; i < weight_words(L) / 4; i += kWarps * 32)
    cp_async16(w + 4 * i, g_weights.w + (kMaxLen - 1 - off) + 4 * i);
  s.w = w + off;
  uint32_t* bnd = w + weight_words(L);
  bnd[threadIdx.x] = 0xffffffffu;
  s.bnd = bnd + lane;
  uint32_t* least = bnd + kWarps * 32;
  s.least = reinterpret_cast<uint16_t*>(least) + lane;
  *extra = least + least_words(L);
  for (int r = L + (threadIdx.x >> 5); r < key_rows(L); r += kWarps) s.key[r * 32] = kMissing;
  return s;
}

// The key at row r + i of the candidate that has key k at row r; d2 = 2 * (r -
// candidate's row).
__device__ __forceinline__ uint32_t shift_key(uint32_t k, int d2, int i) { return k + (uint32_t)((d2 + i) * i) * 1024u; }

// The least of `best` and four candidates at their weights.
__device__ __forceinline__ uint32_t least_of(const uint32_t (&c)[4], uint32_t d0, uint32_t d1, uint32_t d2, uint32_t d3,
                                             uint32_t best) {
  best = __viaddmin_u32(c[0], d0, best);
  best = __viaddmin_u32(c[1], d1, best);
  best = __viaddmin_u32(c[2], d2, best);
  return __viaddmin_u32(c[3], d3, best);
}

// Candidates against the rows r0 + kStep * {1 .. kN}, r0 a multiple of 8:
// best[i] = the least key.  lo2, hi2: twice the first and the last candidate
// (warp-uniform); some: all ones, 0 in a column without a site.  Four
// candidates per round (rows outside the range are valid candidates too).  A
// round's weights are consecutive words of the table, read as 16-byte
// broadcasts.  A long range is a jump of the winner between two obstacles: its
// two ends are tried first, and 16 candidates in between only where the least
// of them, moved to the nearest of the rows, could still win in some column
// (352^3 depth scene: 5 % of the 4-row groups had 60 candidates or more and
// took more than half of all rounds).
template <int kStep, int kN>
__device__ __forceinline__ void refine(const Search& s, int r0, int lo2, int hi2, uint32_t some, uint32_t (&best)[kN]) {
#pragma unroll
  for (int i = 0; i < kN; ++i) best[i] = 0xffffffffu;
  auto round = [&](const uint32_t* k, const uint32_t* w) {
    const uint32_t c[4] = {k[0], k[32], k[64], k[96]};
    if constexpr (kStep == 1) {  // the (row, candidate) differences of a round are consecutive
      uint32_t d[12];
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        const uint4 v = *reinterpret_cast<const uint4*>(w + 4 * g - 3);
        d[4 * g] = v.x, d[4 * g + 1] = v.y, d[4 * g + 2] = v.z, d[4 * g + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < kN; ++i) best[i] = least_of(c, d[i + 4], d[i + 3], d[i + 2], d[i + 1], best[i]);
    } else {
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        const uint4 v = *reinterpret_cast<const uint4*>(w + kStep * (i + 1) - 3);
        best[i] = least_of(c, v.w, v.z, v.y, v.x, best[i]);
      }
    }
  };
  lo2 &= ~7;
  if (hi2 - lo2 < 80) {
    const uint32_t* k = s.key + lo2 * 16;
    const uint32_t* w = s.w + (r0 - (lo2 >> 1));
    const uint32_t* const k_end = s.key + hi2 * 16;
#pragma unroll 1
    for (; k <= k_end; k += 128, w -= 4) round(k, w);
    return;
  }
  int j2 = hi2 & ~7;  // the far end first
  bool far_end = true;
#pragma unroll 1
  while (true) {
    round(s.key + j2 * 16, s.w + (r0 - (j2 >> 1)));
    j2 = far_end ? lo2 : j2 + 8;
    far_end = false;
    if (j2 > hi2) break;
    if ((j2 & 31) == 0) {
      uint32_t limit = best[0];
#pragma unroll
      for (int i = 1; i < kN; ++i) limit = max(limit, best[i]);
      limit &= some;
#pragma unroll 1
      for (; j2 + 32 <= hi2; j2 += 32) {
        const int first = j2 >> 1, gap = max(max(r0 + kStep - first - 15, first - r0 - kN * kStep), 0);
        if (__any_sync(kFullMask, ((uint32_t)s.least[j2] << 15) + s.w[gap] <= limit)) break;
      }
    }
  }
}

// Candidates j0 .. j1 - 1 (j0 a multiple of 16) against one row outside them
// (a multiple of 16) that already has the key `have`: 16 at a time, where the
// least of them, moved to their end nearest to the row, could win.
__device__ __forceinline__ uint32_t scan_row(const Search& s, int row, int j0, int j1, uint32_t have) {
#pragma unroll 1
  for (int j = j0; j < j1; j += 16) {
    const int gap = row < j ? j - row : row - min(j + 15, j1 - 1);
    const uint32_t reach = ((uint32_t)s.least[j * 2] << 15) + s.w[gap];
    if (!__any_sync(kFullMask, reach <= have && reach < kFar)) continue;
#pragma unroll
    for (int t = 0; t < 16; t += 4) {
      if (j + t < j1) {
        const uint32_t* k = s.key + (j + t) * 32;
        const uint4 v = *reinterpret_cast<const uint4*>(s.w + (row - j - t) - 3);
        have = __viaddmin_u32(k[0], v.w, have);
        have = __viaddmin_u32(k[32], v.z, have);
        have = __viaddmin_u32(k[64], v.y, have);
        have = __viaddmin_u32(k[96], v.x, have);
      }
    }
  }
  return have;
}

// Winners at the segment starts (rows 0, S, 2 S ..), into s.bnd.  A warp holds
// its own segment's candidates against the starts at both its ends; another
// start gets them only where some column's least key of the segment, moved to
// the segment's near end, could still beat what the start's neighbours found.
// (All candidates against all 8 starts cost 8 add-and-mins per row; this 2 and
// a minimum.)
__device__ __forceinline__ void segment_starts(const Search& s, int warp, int S, int seg0, int seg1) {
  uint32_t least = 0xffffffffu;
  if (seg0 < s.L) {
    uint32_t b0 = 0xffffffffu, b1 = 0xffffffffu;
    const uint32_t* k = s.key + seg0 * 32;
    const uint32_t* w = s.w - 3;
#pragma unroll 1
    for (int j = seg0; j < seg1; j += 16) {
      uint32_t few = 0xffffffffu;
#pragma unroll
      for (int t = 0; t < 16; t += 4) {
        if (j + t < seg1) {
          const uint32_t k0 = k[t * 32], k1 = k[t * 32 + 32], k2 = k[t * 32 + 64], k3 = k[t * 32 + 96];
          const uint4 a = *reinterpret_cast<const uint4*>(w - t), b = *reinterpret_cast<const uint4*>(w - t + S);
          b0 = __viaddmin_u32(k0, a.w, b0);
          b1 = __viaddmin_u32(k0, b.w, b1);
          b0 = __viaddmin_u32(k1, a.z, b0);
          b1 = __viaddmin_u32(k1, b.z, b1);
          b0 = __viaddmin_u32(k2, a.y, b0);
          b1 = __viaddmin_u32(k2, b.y, b1);
          b0 = __viaddmin_u32(k3, a.x, b0);
          b1 = __viaddmin_u32(k3, b.x, b1);
          few = __vimin3_u32(few, k0, k1);
          few = __vimin3_u32(few, k2, k3);
        }
      }
      s.least[j * 2] = (uint16_t)min(few >> 15, 0xffffu);
      least = min(least, few);
      k += 512;
      w -= 16;
    }
    atomicMin(s.bnd + warp * 32, b0);
    if (warp + 1 < kWarps) atomicMin(s.bnd + (warp + 1) * 32, b1);
  }
  __syncthreads();
  if (seg0 < s.L) {
    const bool some = least < kNoSite;
    least &= ~1023u;
    // the worst of all starts against the nearest any of them can be: mostly
    // nothing is left to look at one by one
    uint32_t worst = 0u;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const uint32_t have = *reinterpret_cast<volatile uint32_t*>(s.bnd + i * 32);
      if (i != warp && i != warp + 1 && i * S < s.L) worst = max(worst, have);
    }
    const bool look = __any_sync(kFullMask, some && least + s.w[S] <= worst);
#pragma unroll 1
    for (int i = 0; look && i < kWarps && i * S < s.L; ++i) {
      if (i == warp || i == warp + 1) continue;
      const int gap = i < warp ? seg0 - i * S : i * S - (seg1 - 1);
      // a start's key only ever falls: a stale one only lets the scan run
      const uint32_t have = *reinterpret_cast<volatile uint32_t*>(s.bnd + i * 32);
      if (__any_sync(kFullMask, some && least + s.w[gap] <= have)) atomicMin(s.bnd + i * 32, scan_row(s, i * S, seg0, seg1, have));
    }
  }
  __syncthreads();
}

// Every row of the block's columns, after the keys are in shared memory
// (called by all threads; synchronises).  out.begin(none) tells whether the
// lane's column has no site; then the warp's rows come in ascending groups:
// out.rows(r, k, same) has the least keys of rows r .. r + 7 (same: one site
// for all eight in every column); then out.finish().
template <class Out>
__device__ __forceinline__ void search_rows(const Search& s, Out& out) {
  const int S = seg_rows(s.L);
  const int warp = __shfl_sync(kFullMask, threadIdx.x >> 5, 0);
  const int seg0 = warp * S, seg1 = min(seg0 + S, s.L);
  __syncthreads();
  segment_starts(s, warp, S, seg0, seg1);
  if (seg0 >= s.L) return;
  const uint32_t last = (uint32_t)(s.L - 1) << 1;  // as a key: only its row counts
  uint32_t cur = s.bnd[warp * 32];
  const uint32_t end = seg0 + S < s.L ? s.bnd[(warp + 1) * 32] : last;
  const bool none = cur >= kNoSite;
  out.begin(none);
  // Columns without a site leave the warp's candidate range alone.
  const uint32_t some = none ? 0u : 0xffffffffu, or_lo = ~some & kRowBits, and_hi = some & kRowBits;
  int lo2, hi2;
  auto range = [&](uint32_t klo, uint32_t khi) {
    lo2 = (int)__reduce_min_sync(kFullMask, (klo & kRowBits) | or_lo);
    hi2 = (int)__reduce_max_sync(kFullMask, khi & and_hi);
  };
  uint32_t n[8];  // winners at the ends of the 8-row groups
  auto group_ends = [&](auto rows) {
    constexpr int kN = decltype(rows)::value;
    uint32_t b[kN];
    refine<8, kN>(s, seg0, lo2, hi2, some, b);
#pragma unroll
    for (int i = 0; i < 8; ++i) n[i] = i < kN ? b[i < kN ? i : 0] : end;
  };
  range(cur, end);
  if (lo2 >= hi2) {
#pragma unroll
    for (int i = 0; i < 8; ++i) n[i] = 8 * i + 8 < S ? shift_key(cur, 2 * seg0 - lo2, 8 * (i + 1)) : end;
  } else if (S == 16) {
    group_ends(std::integral_constant<int, 1>{});
  } else if (S == 32) {
    group_ends(std::integral_constant<int, 3>{});
  } else if (S == 48) {
    group_ends(std::integral_constant<int, 5>{});
  } else {
    group_ends(std::integral_constant<int, 7>{});
  }
#pragma unroll 1
  for (int r = seg0; r < seg1; r += 8) {
    uint32_t b[7];
    range(cur, r + 8 < s.L ? n[0] : last);
    const bool same = lo2 >= hi2;
    if (same) {
#pragma unroll
      for (int i = 0; i < 7; ++i) b[i] = shift_key(cur, 2 * r - lo2, i + 1);
    } else {
      refine<1, 7>(s, r, lo2, hi2, some, b);
    }
    const uint32_t o[8] = {cur, b[0], b[1], b[2], b[3], b[4], b[5], b[6]};
    out.rows(r, o, same);
    cur = n[0];
#pragma unroll
    for (int i = 0; i < 7; ++i) n[i] = n[i + 1];
  }
  out.finish();
}

// ---------------------------------------------------------------------------
// Launches of a step chain (programmatic dependent launch): a kernel's blocks
// may take their places while the one before drains.  wait_for_previous comes
// before the first access to what that kernel wrote -- it returns once the
// previous kernel has ended and its writes are visible -- and start_next once a
// block needs nothing more from the launch order.  Two kernels before the
// current one are complete as well: the previous one waited for them.  With
// the rolled loops above this took 128^3 with queries from 45 to 37 us and
// 203 x 331 x 157 from 168 to 145.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;"); }

// A word that an earlier kernel of the chain writes.  That kernel may still run
// when this one begins, so the word is not read-only for this kernel's lifetime:
// no __ldg and no const __restrict__ parameter (either lets the compiler read
// through the non-coherent path, and early).  Volatile keeps the load after
// wait_for_previous.
__device__ __forceinline__ uint32_t load_chained(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}

// Pass Y's rows into `field`, byte offsets in 32 bits (512 x 512 x 1023: 1.1 GB).
struct OutY {
  uint32_t* field;
  uint32_t first, row_bytes;  // of this lane's row 0; from a row to the next
  int Y;
  __device__ __forceinline__ void begin(bool) {}
  __device__ __forceinline__ void rows(int r, const uint32_t (&k)[8], bool) {
    char* base = reinterpret_cast<char*>(field);
    uint32_t at = first + (uint32_t)r * row_bytes;
    if (r + 8 <= Y) {
#pragma unroll
      for (int i = 0; i < 8; ++i, at += row_bytes) *reinterpret_cast<uint32_t*>(base + at) = k[i];
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i, at += row_bytes)
        if (r + i < Y) *reinterpret_cast<uint32_t*>(base + at) = k[i];
    }
  }
  __device__ __forceinline__ void finish() {}
};

// Pass Y of plane x, chunk c: the nearest site in the (y, z) plane.
__device__ __forceinline__ void item_y(uint32_t* smem, const uint32_t* bits, const uint32_t* near, uint32_t* field, int X, int Y, int Z, int x, int c) {
  const int lane = threadIdx.x & 31;
  uint32_t* extra;
  const Search s = search_setup(smem, Y, &extra);
  start_next();
  wait_for_previous();
  uint2* col = reinterpret_cast<uint2*>(extra);  // (bits, near) of every y
  const uint64_t base = ((uint64_t)c * X + x) * Y;
  for (int y = threadIdx.x; y < Y; y += kWarps * 32) col[y] = make_uint2(load_chained(bits + base + y), load_chained(near + base + y));
  cp_async_wait_all();
  __syncthreads();
  // The nearest site of the (x, y) column by phase 1's rule
  // (kernelPBAphase1FloodZ, GV/voxelmap/kernels/VoxelMapOperationsPBA.hpp:63-124):
  // the lower of two equally near ones.  Without a site above the reference
  // puts one at 1023, and where that is nearer the voxel stays uninitialised
  // (only possible when Z is above 512).
  // Four lanes make the 32 keys of one y, two quads of z each (odd y the upper
  // quad first: no bank conflicts).
#pragma unroll 1
  for (int y0 = (threadIdx.x >> 5) * 8; y0 < Y; y0 += kWarps * 8) {  // eight y per warp
    const int y = min(y0 + (lane >> 2), Y - 1);
    const bool store = y0 + (lane >> 2) < Y;
    const uint2 q = col[y];
    const bool plain = Z <= 512 && !__any_sync(kFullMask, q.x != 0u);
    uint4* keys = reinterpret_cast<uint4*>(smem) + y * 8;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int quad = (lane & 3) + 4 * ((y ^ half) & 1), l = 4 * quad;
      int below = (int)(short)(q.y & 0xffffu), above = (int)q.y >> 16;
      uint32_t k[4];
      if (plain) {
        const int dl = 32 * (l - below), du = 32 * (above - l);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t a = (uint32_t)(dl + 32 * i), b = (uint32_t)(du - 32 * i);
          k[i] = min(a * a + (uint32_t)(2 * y), b * b + (uint32_t)(2 * y + 1));
        }
      } else {
        // the chunk's own sites: the nearest outside these four z, then the distances step by step
        const uint32_t lo = q.x & ((1u << l) - 1u), hi = (q.x >> l) >> 4, four = (q.x >> l) & 15u;
        if (lo) below = 31 - __clz(lo);
        if (hi) above = l + 3 + __ffs(hi);
        int dl[4], du[4];
        dl[0] = (four & 1u) ? 0 : l - below;
        du[3] = above - l - 3;
#pragma unroll
        for (int i = 1; i < 4; ++i) {
          dl[i] = (four >> i & 1u) ? 0 : dl[i - 1] + 1;
          du[3 - i] = (four >> (4 - i) & 1u) ? 1 : du[4 - i] + 1;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t lower = (uint32_t)(dl[i] * dl[i]) * 1024u + (uint32_t)(2 * y);
          const uint32_t upper = (uint32_t)(du[i] * du[i]) * 1024u + (uint32_t)(2 * y + 1);
          if (Z > 512 && upper >= kMissing && 1023 - (c * 32 + l + i) < dl[i]) lower = kMissing;
          k[i] = min(lower, upper);
        }
      }
      if (c * 32 + 32 > Z) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c * 32 + l + i >= Z) k[i] = kMissing;
      }
      if (store) keys[quad] = make_uint4(k[0], k[1], k[2], k[3]);
    }
  }
  OutY out{field, (((uint32_t)c * Y * X + x) * 32 + lane) * 4u, (uint32_t)X * 128u, Y};
  search_rows(s, out);
}

__device__ __forceinline__ float sqrt_approx(float v) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// Pass X's rows on their way to the map: the winner's key of pass Y is
// fetched from `field` while the next rows are searched; the site's z is z +-
// sqrt(d - dy^2), an exact square whose root (below 1024) the approximate
// square root gives to 2^-12.  A site's word is made once where several rows
// share it.  The words go out 8 x (a 32-byte sector) per z, 16 z at a time
// through 512 bytes per warp: whole sectors with 16-byte stores where the map's
// rows are aligned (vec), else word by word.
struct OutX {
  const uint32_t* src;  // row 0 of this lane's column in `field`
  uint32_t* stage;
  uint32_t* dst;        // map word (first z of the chunk, y, 0)
  uint32_t layer;
  int X, z_rows;        // z rows of the chunk inside the map
  int y2;               // 2 * y
  float zf;             // 2^23 + 2^22 + z
  bool vec, none;
  uint32_t mask;        // row bits of a key, 0 where the column has no site
  uint32_t key[8], v[8];
  int r = -1;           // first of the eight pending rows
  bool one;             // they share key[0]

  __device__ __forceinline__ void begin(bool no_site) {
    none = no_site;
    mask = no_site ? 0u : kRowBits;
  }
  __device__ __forceinline__ void fetch(int i, uint32_t k) {
    key[i] = k & mask;
    v[i] = load_chained(src + key[i] * 16u);
  }
  __device__ __forceinline__ void rows(int r_new, const uint32_t (&k)[8], bool same) {
    if (r >= 0) put();
    r = r_new;
    one = same;
    fetch(0, k[0]);
    if (!same) {
#pragma unroll
      for (int i = 1; i < 8; ++i) fetch(i, k[i]);
    }
  }
  __device__ __forceinline__ uint32_t word(int i) const {
    const uint32_t y2s = v[i] & kRowBits;
    const int dy2 = y2 - (int)y2s;
    const int m4 = (int)(v[i] >> 10) * 4 - dy2 * dy2;  // (2 dz)^2, below 2^22
    const float dz2 = sqrt_approx(__uint_as_float(0x4B000000u | (uint32_t)m4) - 8388608.0f);
    const float half = __uint_as_float((v[i] << 31) ^ 0xBF000000u);  // +0.5 above, -0.5 below
    const uint32_t zs = __float_as_uint(__fmaf_rn(dz2, half, zf));   // z in the low bits
    return none ? kDvUninit : (zs << 20) + ((y2s * 1024u + key[i]) >> 1);
  }
  __device__ __forceinline__ void put() {
    uint32_t w[8];
    w[0] = word(0);
    if (one) {
#pragma unroll
      for (int i = 1; i < 8; ++i) w[i] = w[0];
    } else {
#pragma unroll
      for (int i = 1; i < 8; ++i) w[i] = word(i);
    }
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      // word of (z, x): z * 8 + x, the two halves of a z swapped where z & 4 (no bank conflicts)
      uint4* mine = reinterpret_cast<uint4*>(stage + (lane & 15) * 8);
      const int sw = (lane >> 2) & 1;
      __syncwarp();
      if ((lane >> 4) == g) {
        mine[sw] = make_uint4(w[0], w[1], w[2], w[3]);
        mine[sw ^ 1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
      __syncwarp();
      if (vec && r + 8 <= X) {
        const int zl = lane >> 1, h = lane & 1;
        const uint4 o = *reinterpret_cast<const uint4*>(stage + zl * 8 + (h ^ ((zl >> 2) & 1)) * 4);
        const int z = g * 16 + zl;
        if (z < z_rows) *reinterpret_cast<uint4*>(dst + (uint64_t)((uint32_t)z * layer + (uint32_t)(r + h * 4))) = o;
      } else {
        const int sx = lane & 7;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int zl = t * 4 + (lane >> 3), z = g * 16 + zl;
          const uint32_t o = stage[zl * 8 + (sx ^ (zl & 4))];
          if (r + sx < X && z < z_rows) dst[(uint64_t)((uint32_t)z * layer + (uint32_t)(r + sx))] = o;
        }
      }
    }
  }
  __device__ __forceinline__ void finish() {
    if (r >= 0) put();
  }
};

// Pass X of plane y, chunk c: the nearest site of the map, written to the map.
__device__ __forceinline__ void item_x(uint32_t* smem, const uint32_t* field, uint32_t* map, int X,
                                       int Y, int Z, int y, int c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* extra;
  const Search s = search_setup(smem, X, &extra);
  wait_for_previous();
  const uint32_t* src = field + ((uint64_t)c * Y + y) * X * 32 + lane;
  // The item's rows are one piece of `field`: copied to the keys' place 16
  // bytes at a time, then a key's row bits (pass Y's row and side) replaced by x.
  {
    const uint4* in = reinterpret_cast<const uint4*>(src - lane);
    uint4* keys = reinterpret_cast<uint4*>(smem);
    for (int i = threadIdx.x; i < X * 8; i += kWarps * 32) cp_async16(keys + i, in + i);
    cp_async_wait_all();
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < X * 8; i += kWarps * 32) {
      uint4 k = keys[i];
      const uint32_t x2 = (uint32_t)(i >> 3) << 1;
      k.x = (k.x & ~1023u) | x2;
      k.y = (k.y & ~1023u) | x2;
      k.z = (k.z & ~1023u) | x2;
      k.w = (k.w & ~1023u) | x2;
      keys[i] = k;
    }
  }
  OutX out;
  out.src = src;
  out.stage = extra + warp * 128;
  out.layer = (uint32_t)X * (uint32_t)Y;
  out.dst = map + (uint64_t)(c * 32) * out.layer + (uint64_t)y * X;
  out.X = X;
  out.z_rows = Z - c * 32;
  out.y2 = 2 * y;
  out.zf = __uint_as_float(0x4B400000u | (uint32_t)(c * 32 + lane));
  out.vec = (X & 3) == 0 && (reinterpret_cast<uintptr_t>(map) & 15u) == 0;
  search_rows(s, out);
}

// Resident blocks the registers must allow: pass Y four (64 registers; four fit
// the shared memory up to 384 rows, and 69 registers took three, 24 maps' pass
// Y 682 us against 634, though the batch form spills 16 bytes at 64), pass X three
// (at 64 registers it spills more: 512^3 447 -> 486 us).
constexpr int kStageWords = kWarps * 128;
int smem_y(int Y) { return search_smem_words(Y, 2 * Y) * 4; }
int smem_x(int X) { return search_smem_words(X, kStageWords) * 4; }

__global__ void __launch_bounds__(kWarps * 32, 4)
    search_y_kernel(const uint32_t* bits, const uint32_t* near, uint32_t* field, int X, int Y, int Z, const uint32_t* skip) {
  extern __shared__ __align__(16) uint32_t s_rows[];
  if (skip != nullptr) {
    wait_for_previous();
    if (load_chained(skip) != 0u) return;
  }
  item_y(s_rows, bits, near, field, X, Y, Z, blockIdx.x, blockIdx.y);
}

__global__ void __launch_bounds__(kWarps * 32, 3)
    search_x_kernel(const uint32_t* field, uint32_t* map, int X, int Y, int Z, const uint32_t* skip) {
  extern __shared__ __align__(16) uint32_t s_rows[];
  if (skip != nullptr) {
    wait_for_previous();
    if (load_chained(skip) != 0u) return;
  }
  item_x(s_rows, field, map, X, Y, Z, blockIdx.x, blockIdx.y);
}

// insertPointCloud into the occupancy bits (coordinates as
// kernelInsertGlobalPointCloud, GV/voxelmap/kernels/VoxelMapOperations.hpp:266-300).
__global__ void zbits_insert_kernel(uint32_t* __restrict__ bits, int X, int Y, int Z, float side,
                                    const float* __restrict__ xyz, uint64_t n, uint32_t* __restrict__ outside) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  bool out = false;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t x = coord_to_voxel(__ldg(xyz + 3 * i), side), y = coord_to_voxel(__ldg(xyz + 3 * i + 1), side),
                   z = coord_to_voxel(__ldg(xyz + 3 * i + 2), side);
    if (x < (uint32_t)X && y < (uint32_t)Y && z < (uint32_t)Z)
      atomicOr(bits + ((uint64_t)(z >> 5) * X + x) * Y + y, 1u << (z & 31));
    else out = true;
  }
  if (outside != nullptr && __any_sync(kFullMask, out) && (threadIdx.x & 31) == 0) *outside = 1u;
}

// `near` from `bits`, one thread per (x, y) column (y fastest): one scan up
// for the sites below each chunk, one down for those above.
template <int kMaxChunks>
__device__ __forceinline__ void near_column(const uint32_t* bits, uint32_t* near, uint32_t layer, int chunks, uint32_t f) {
  uint32_t m[kMaxChunks], below[kMaxChunks];
#pragma unroll
  for (int c = 0; c < kMaxChunks; ++c) m[c] = c < chunks ? load_chained(bits + (uint64_t)c * layer + f) : 0u;
  int last = -1;
#pragma unroll
  for (int c = 0; c < kMaxChunks; ++c) {
    below[c] = (uint32_t)(last < 0 ? kNoneBelow : last - c * 32) & 0xffffu;
    if (m[c]) last = c * 32 + 31 - __clz(m[c]);
  }
  int next = -1;
#pragma unroll
  for (int c = kMaxChunks - 1; c >= 0; --c) {
    if (c < chunks) near[(uint64_t)c * layer + f] = below[c] | (uint32_t)(next < 0 ? kNoneAbove : next - c * 32) << 16;
    if (m[c]) next = c * 32 + __ffs(m[c]) - 1;
  }
}

template <int kMaxChunks>
__global__ void __launch_bounds__(256) near_kernel(const uint32_t* bits, uint32_t* near, uint32_t layer, int chunks,
                                                   const uint32_t* skip) {
  wait_for_previous();
  if (skip != nullptr && load_chained(skip) != 0u) return;
  const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f < layer) near_column<kMaxChunks>(bits, near, layer, chunks, f);
}

// Occupancy bits of a filled map.  A voxel holding another site than its own
// sets *other_sites: the sweeps of edt.cu take the map then.  A block reads 32
// x by 8 y columns of one chunk (a warp one y, a lane one x, 32 loads in
// flight) and stores the words with y fastest through shared memory.  With 32
// y per block 320 x 320 x 96 made 300 blocks, two per SM (13.8 us, now 9.2).
constexpr int kTileY = 8;
__device__ __forceinline__ bool zbits_tile(const uint32_t* __restrict__ vox, uint32_t* __restrict__ bits, int X, int Y, int Z,
                                           int bx, int by, int bz, uint32_t (&tile)[kTileY][33]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = bx * 32 + lane, y = by * kTileY + warp, z0 = bz * 32;
  const uint64_t layer = (uint64_t)X * Y;
  bool other = false;
  uint32_t word = 0u;
  if (x < X && y < Y) {
    vox += (uint64_t)z0 * layer + (uint64_t)y * X + x;
    const uint32_t own = (uint32_t)x | (uint32_t)y << 10 | (uint32_t)z0 << 20;
    uint32_t v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = z0 + i < Z ? __ldg(vox + (uint64_t)i * layer) : kDvUninit;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if (v[i] != kDvUninit) {
        word |= 1u << i;
        other |= v[i] != own + ((uint32_t)i << 20);
      }
    }
  }
  tile[warp][lane] = word;
  __syncthreads();
  const int xo = bx * 32 + (threadIdx.x >> 3), yo = by * kTileY + (threadIdx.x & 7);
  if (xo < X && yo < Y) bits[((uint64_t)bz * X + xo) * Y + yo] = tile[threadIdx.x & 7][threadIdx.x >> 3];
  return other;
}

__global__ void __launch_bounds__(256) zbits_from_map_kernel(const uint32_t* __restrict__ map, uint32_t* __restrict__ bits,
                                                             int X, int Y, int Z, uint32_t* __restrict__ other_sites) {
  __shared__ uint32_t tile[kTileY][33];
  const bool other = zbits_tile(map, bits, X, Y, Z, blockIdx.x, blockIdx.y, blockIdx.z, tile);
  if (__any_sync(kFullMask, other) && (threadIdx.x & 31) == 0) atomicOr(other_sites, 1u);
}

// ---------------------------------------------------------------------------
// The same steps over every map of a batch; each map's areas lie in its own
// workspace past the counters, its other-sites flag in word Z + 2.
// ---------------------------------------------------------------------------
struct Areas {
  uint32_t *bits, *near, *field;
};
__host__ __device__ __forceinline__ Areas areas(uint32_t* area, int X, int Y, int Z) {
  const uint64_t step = (bits_words(X, Y, Z) + 31) / 32 * 32;
  return Areas{area, area + step, area + 2 * step};
}
__device__ __forceinline__ Areas areas(const BatchMap& m) { return areas(m.scratch + edt_sync_words(m.Z), m.X, m.Y, m.Z); }
__device__ __forceinline__ uint32_t* other_flag(const BatchMap& m) { return m.scratch + m.Z + 2; }

// Last k with prefix[k] <= g.
template <class T>
__device__ __forceinline__ uint32_t owner(const T* __restrict__ prefix, uint32_t n, T g) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(prefix + mid) <= g) lo = mid; else hi = mid;
  }
  return lo;
}

// Grid of the kernels below: block row r takes the maps r, r + gridDim.y, ..,
// with as many blocks as the `work` blocks of the largest map, at most `widest`.
// (Always the widest, 300 maps of 20^3 launched 38,400 blocks of near_batch_kernel
// for 600 blocks of work: 81 us of a 182 us step.)
dim3 map_rows(const BatchItems& it, uint64_t work, unsigned widest) {
  return dim3((unsigned)std::min<uint64_t>(work, widest), std::min(it.n_maps, 65535u));
}

__global__ void zbits_clear_batch_kernel(const BatchMap* __restrict__ maps, uint32_t n_maps) {
  for (uint32_t k = blockIdx.y; k < n_maps; k += gridDim.y) {
    const BatchMap m = maps[k];
    if (blockIdx.x == 0 && threadIdx.x == 0) *other_flag(m) = 0u;
    uint32_t* bits = areas(m).bits;
    const uint64_t n = bits_words(m.X, m.Y, m.Z);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) bits[i] = 0u;
  }
}

// point i belongs to map k with offsets[k] <= i < offsets[k + 1]
__global__ void zbits_insert_batch_kernel(const BatchMap* __restrict__ maps, uint32_t n_maps, const float* __restrict__ xyz,
                                          const uint64_t* __restrict__ offsets, uint64_t n) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const BatchMap m = maps[owner(offsets, n_maps, i)];
    const uint32_t x = coord_to_voxel(__ldg(xyz + 3 * i), m.side), y = coord_to_voxel(__ldg(xyz + 3 * i + 1), m.side),
                   z = coord_to_voxel(__ldg(xyz + 3 * i + 2), m.side);
    if (x < (uint32_t)m.X && y < (uint32_t)m.Y && z < (uint32_t)m.Z)
      atomicOr(areas(m).bits + ((uint64_t)(z >> 5) * m.X + x) * m.Y + y, 1u << (z & 31));
  }
}

// the blocks of a row stride over its map's tiles
__global__ void __launch_bounds__(256) zbits_from_map_batch_kernel(const BatchMap* __restrict__ maps, uint32_t n_maps) {
  __shared__ uint32_t tile[kTileY][33];
  for (uint32_t k = blockIdx.y; k < n_maps; k += gridDim.y) {
    const BatchMap m = maps[k];
    uint32_t* bits = areas(m).bits;
    const int tx = (m.X + 31) >> 5, ty = (m.Y + kTileY - 1) / kTileY, tiles = tx * ty * z_chunks(m.Z);
    bool other = false;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      other |= zbits_tile(m.vox, bits, m.X, m.Y, m.Z, t % tx, t / tx % ty, t / (tx * ty), tile);
      __syncthreads();
    }
    if (__any_sync(kFullMask, other) && (threadIdx.x & 31) == 0) atomicOr(other_flag(m), 1u);
  }
}

template <int kMaxChunks>
__device__ __forceinline__ void near_map(const BatchMap& m) {
  const Areas a = areas(m);
  const uint32_t layer = (uint32_t)m.X * (uint32_t)m.Y;
  for (uint32_t f = blockIdx.x * blockDim.x + threadIdx.x; f < layer; f += gridDim.x * blockDim.x)
    near_column<kMaxChunks>(a.bits, a.near, layer, z_chunks(m.Z), f);
}

// each map with the registers and loads of its own height
__global__ void __launch_bounds__(256) near_batch_kernel(const BatchMap* __restrict__ maps, uint32_t n_maps, int skip_other) {
  wait_for_previous();
  for (uint32_t k = blockIdx.y; k < n_maps; k += gridDim.y) {
    const BatchMap m = maps[k];
    if (skip_other && load_chained(other_flag(m)) != 0u) continue;
    const int chunks = z_chunks(m.Z);
    if (chunks <= 4) near_map<4>(m);
    else if (chunks <= 8) near_map<8>(m);
    else if (chunks <= 16) near_map<16>(m);
    else near_map<32>(m);
  }
}

__global__ void __launch_bounds__(kWarps * 32, 4)
    search_y_batch_kernel(const BatchMap* __restrict__ maps, const long long* __restrict__ prefix, uint32_t n_maps,
                          int skip_other) {
  extern __shared__ __align__(16) uint32_t s_rows[];
  const uint32_t k = owner(prefix, n_maps, (long long)blockIdx.x);
  const BatchMap m = maps[k];
  if (skip_other) {
    wait_for_previous();
    if (load_chained(other_flag(m)) != 0u) return;
  }
  const int item = (int)((long long)blockIdx.x - __ldg(prefix + k)), c = item / m.X;
  const Areas a = areas(m);
  item_y(s_rows, a.bits, a.near, a.field, m.X, m.Y, m.Z, item - c * m.X, c);
}

__global__ void __launch_bounds__(kWarps * 32, 3)
    search_x_batch_kernel(const BatchMap* __restrict__ maps, const long long* __restrict__ prefix, uint32_t n_maps,
                          int skip_other) {
  extern __shared__ __align__(16) uint32_t s_rows[];
  const uint32_t k = owner(prefix, n_maps, (long long)blockIdx.x);
  const BatchMap m = maps[k];
  if (skip_other) {
    wait_for_previous();
    if (load_chained(other_flag(m)) != 0u) return;
  }
  const int item = (int)((long long)blockIdx.x - __ldg(prefix + k)), c = item / m.Y;
  item_x(s_rows, areas(m).field, m.vox, m.X, m.Y, m.Z, item - c * m.Y, c);
}

// Dynamic shared memory attributes, once per device.
cudaError_t search_setup_once() {
  constexpr int kMaxDevices = 64;
  static std::once_flag once[kMaxDevices];
  static cudaError_t err[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [&] {
    cudaError_t r = cudaFuncSetAttribute(search_y_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_y(kMaxLen));
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(search_x_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_x(kMaxLen));
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(search_y_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_y(kMaxLen));
    if (r == cudaSuccess)
      r = cudaFuncSetAttribute(search_x_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_x(kMaxLen));
    err[dev] = r;
  });
  return err[dev];
}

// A launch that may begin while the kernel before it in the stream drains (it
// calls wait_for_previous).
template <class... P, class... A>
cudaError_t launch_next(void (*kernel)(P...), dim3 grid, int smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// near, pass Y and pass X from the occupancy bits.
cudaError_t launch_from_bits(uint32_t* map, const Areas& a, gvx_dims d, const uint32_t* skip, cudaStream_t s) {
  cudaError_t e = search_setup_once();
  if (e != cudaSuccess) return e;
  const int X = (int)d.x, Y = (int)d.y, Z = (int)d.z, zw = z_chunks(Z);
  const uint32_t layer = d.x * d.y;
  const auto near = zw <= 4 ? near_kernel<4> : zw <= 8 ? near_kernel<8> : zw <= 16 ? near_kernel<16> : near_kernel<32>;
  e = launch_next(near, dim3((layer + 255) / 256), 0, s, a.bits, a.near, layer, zw, skip);
  if (e == cudaSuccess) e = launch_next(search_y_kernel, dim3(X, zw), smem_y(Y), s, a.bits, a.near, a.field, X, Y, Z, skip);
  if (e == cudaSuccess) e = launch_next(search_x_kernel, dim3(Y, zw), smem_x(X), s, a.field, map, X, Y, Z, skip);
  return e;
}

}  // namespace

// Columns up to kMaxLen rows: a block's keys fill 64 KB of shared memory, three
// blocks an SM.  Z is free: the lanes of the last z chunk idle, and even with
// one z of 32 in use the search is the faster one (512 x 512 x 1: 85 us, the
// sweeps 318; 512 x 512 x 16: 97 against 454; 16^3: 19 against 29).
bool search_takes(gvx_dims d) { return d.x <= (uint32_t)kMaxLen && d.y <= (uint32_t)kMaxLen; }

uint64_t search_words(gvx_dims d) {
  const uint64_t n = bits_words((int)d.x, (int)d.y, (int)d.z);
  return 2 * ((n + 31) / 32 * 32) + 32 * n;
}

uint64_t search_bits_words(gvx_dims d) { return bits_words((int)d.x, (int)d.y, (int)d.z); }

cudaError_t launch_search_voxelize(uint32_t* d_vox, uint32_t* area, gvx_dims d, float side, const float* d_xyz, uint64_t n,
                                   uint32_t* d_outside, cudaStream_t s) {
  const Areas a = areas(area, (int)d.x, (int)d.y, (int)d.z);
  if (n > 0) {
    const unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)device_sms() * 16);
    zbits_insert_kernel<<<blocks, 256, 0, s>>>(a.bits, (int)d.x, (int)d.y, (int)d.z, side, d_xyz, n, d_outside);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return launch_from_bits(d_vox, a, d, nullptr, s);
}

cudaError_t launch_search_filled(uint32_t* d_vox, uint32_t* area, gvx_dims d, uint32_t* d_other, cudaStream_t s) {
  const Areas a = areas(area, (int)d.x, (int)d.y, (int)d.z);
  const dim3 grid((d.x + 31) / 32, (d.y + kTileY - 1) / kTileY, (unsigned)z_chunks((int)d.z));
  zbits_from_map_kernel<<<grid, 256, 0, s>>>(d_vox, a.bits, (int)d.x, (int)d.y, (int)d.z, d_other);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? launch_from_bits(d_vox, a, d, d_other, s) : e;
}

long long search_items(gvx_dims d, int pass) {
  return (long long)z_chunks((int)d.z) * (pass == 1 ? d.x : d.y);
}

namespace {
cudaError_t launch_from_bits_batch(const BatchMap* d_table, const BatchItems& it, int skip_other, cudaStream_t s) {
  cudaError_t e = search_setup_once();
  if (e != cudaSuccess) return e;
  e = launch_next(near_batch_kernel, map_rows(it, ((uint64_t)it.x_max * it.y_max + 255) / 256, 128), 0, s, d_table, it.n_maps,
                  skip_other);
  if (e == cudaSuccess)
    e = launch_next(search_y_batch_kernel, dim3((unsigned)it.total[4]), smem_y((int)it.y_max), s, d_table, it.d_prefix[4],
                    it.n_maps, skip_other);
  if (e == cudaSuccess)
    e = launch_next(search_x_batch_kernel, dim3((unsigned)it.total[5]), smem_x((int)it.x_max), s, d_table, it.d_prefix[5],
                    it.n_maps, skip_other);
  return e;
}
}  // namespace

cudaError_t launch_search_voxelize_batch(const BatchMap* d_table, const BatchItems& it, const float* d_xyz,
                                         const uint64_t* d_offsets, uint64_t n_total, cudaStream_t s) {
  const uint64_t words = bits_words((int)it.x_max, (int)it.y_max, (int)it.z_max);
  zbits_clear_batch_kernel<<<map_rows(it, (words + 255) / 256, 64), 256, 0, s>>>(d_table, it.n_maps);
  if (n_total > 0) {
    const unsigned blocks = (unsigned)std::min<uint64_t>((n_total + 255) / 256, (uint64_t)device_sms() * 16);
    zbits_insert_batch_kernel<<<blocks, 256, 0, s>>>(d_table, it.n_maps, d_xyz, d_offsets, n_total);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? launch_from_bits_batch(d_table, it, 0, s) : e;
}

cudaError_t launch_search_filled_batch(const BatchMap* d_table, const BatchItems& it, cudaStream_t s) {
  const uint64_t tiles = (uint64_t)((it.x_max + 31) / 32) * ((it.y_max + kTileY - 1) / kTileY) * z_chunks((int)it.z_max);
  zbits_from_map_batch_kernel<<<map_rows(it, tiles, 64), 256, 0, s>>>(d_table, it.n_maps);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? launch_from_bits_batch(d_table, it, 1, s) : e;
}

}  // namespace gvx
