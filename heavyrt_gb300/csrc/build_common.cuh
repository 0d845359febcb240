// Device helpers shared by the single-geometry build (build.cu) and the
// segmented multi-geometry build (build_batch.cu).
#pragma once

#include "hrt_common.cuh"

namespace hrt
{
namespace bc
{

constexpr int      kScanItems  = 16;    // items per thread of the look-back scans
constexpr uint32_t kFlagAgg    = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask  = (1u << 30) - 1u;
constexpr uint32_t kSpinLimit  = 1u << 22;  // bounded look-back wait

__device__ __forceinline__ void store_relaxed(uint32_t* p, uint32_t v)
{
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t load_relaxed(const uint32_t* p)
{
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t atomic_add_acq_rel(uint32_t* p, uint32_t v)
{
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// A node written by other threads of the same kernel, read through L2 in two
// 16-byte loads: {boxMin, leftOffset}, {boxMax, escapeIndex}.
__device__ __forceinline__ void load_node_cg(const BVHNode32* n, float4& lo, float4& hi)
{
  const float4* p = reinterpret_cast<const float4*>(n);
  lo = __ldcg(p);
  hi = __ldcg(p + 1);
}

// A finished LR node in one 256-bit read-only load (its type is 4-byte aligned,
// so a plain copy is eight loads; LR arrays start at an allocation's boundary).
__device__ __forceinline__ BVHNode32 load_node(const BVHNode32* n)
{
  BVHNode32 v;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v.boxMin[0]), "=f"(v.boxMin[1]), "=f"(v.boxMin[2]), "=r"(v.leftOffset), "=f"(v.boxMax[0]),
        "=f"(v.boxMax[1]), "=f"(v.boxMax[2]), "=r"(v.escapeIndex)
      : "l"(n));
  return v;
}

// SpreadBits / ZIndex3D, core/builders/lbvh.cpp:25-39.
__device__ __forceinline__ uint32_t spread_bits(int x, int offset)
{
  x = (x | (x << 10)) & 0x000F801F;
  x = (x | (x << 4)) & 0x00E181C3;
  x = (x | (x << 2)) & 0x03248649;
  x = (x | (x << 2)) & 0x09249249;
  return (uint32_t)x << offset;
}

// Morton code of one triangle (kernel1D_EvalMortonCodesFromTriangles,
// core/builders/lbvh.cpp:259-287): box centre, or the centroid
// 0.33333333*(v1+v2+v3) when the geometry has fewer than 256 triangles,
// quantised against the scene box with truncation toward zero.
__device__ __forceinline__ uint32_t morton_code(const float4& a, const float4& b, const float4& c, uint32_t nTris,
                                                const float* bmin, const float* scale)
{
  const float pa[3] = {a.x, a.y, a.z}, pb[3] = {b.x, b.y, b.z}, pc[3] = {c.x, c.y, c.z};
  int q[3];
#pragma unroll
  for (int k = 0; k < 3; k++)
  {
    float center;
    if (nTris < 256)
      center = __fmul_rn(0.33333333f, __fadd_rn(__fadd_rn(pa[k], pb[k]), pc[k]));
    else
    {
      const float mn = lm_min(pa[k], lm_min(pb[k], pc[k]));
      const float mx = lm_max(pa[k], lm_max(pb[k], pc[k]));
      center = __fmul_rn(__fadd_rn(mn, mx), 0.5f);
    }
    q[k] = __float2int_rz(__fmul_rn(scale[k], __fsub_rn(center, bmin[k])));
  }
  return spread_bits(q[0], 0) | spread_bits(q[1], 1) | spread_bits(q[2], 2);
}

// The four 8-bit digits of a warp's codes to a block's counters (4 x 256);
// `mask` = the lanes that are `in`, lane 0 among them.  A warp whose codes agree
// in a digit adds once.
__device__ __forceinline__ void count_digits(uint32_t code, bool in, uint32_t mask, uint32_t* hist)
{
  const uint32_t first = __shfl_sync(0xFFFFFFFFu, code, 0);
  const uint32_t differ = __reduce_or_sync(0xFFFFFFFFu, in ? code ^ first : 0u);
#pragma unroll
  for (int p = 0; p < 4; p++)
  {
    const uint32_t d = (code >> (8 * p)) & 0xFFu;
    if (((differ >> (8 * p)) & 0xFFu) == 0u)
    {
      if ((threadIdx.x & 31u) == 0u) atomicAdd(&hist[p * 256 + d], (uint32_t)__popc(mask));
    }
    else if (in)
      atomicAdd(&hist[p * 256 + d], 1u);
  }
}

// ZIndexMultCoeff on the box widened by 1e-4 (core/builders/lbvh.cpp:41-51,263).
// cubic = 1 (the engine's HRT_MORTON_CUBIC frame, no reference counterpart):
// x, y and z share the scale of the longest widened extent, so a cell of the
// Morton grid is a cube and a flat scene (a heightfield) does not spend a
// third of the code's bits splitting its thin axis; the codes are still
// 3 x 10 bits in [0, 1023] per axis.
__device__ __forceinline__ void zindex_scale(const float* mn, const float* mx, BuildParams* params, int cubic = 0)
{
  float ext[4];
  for (int c = 0; c < 4; c++)
  {
    params->bmin[c] = mn[c];
    params->bmax[c] = mx[c];
    const float lo = __fsub_rn(mn[c], 1e-4f);
    const float hi = __fadd_rn(mx[c], 1e-4f);
    ext[c] = __fsub_rn(hi, lo);
  }
  const float emax = lm_max(ext[0], lm_max(ext[1], ext[2]));
  for (int c = 0; c < 4; c++)
  {
    const float e = (cubic && c < 3) ? emax : ext[c];
    float inv = __fdiv_rn(1.0f, e);
    if (c < 3 && fabsf(e) < 1e-20f) inv = 0.0f;
    params->scale[c] = __fmul_rn(1024.0f, inv);
  }
}

__device__ __forceinline__ int clz_delta(uint32_t a, uint32_t b)
{
  const uint32_t x = a ^ b;
  return x == 0u ? 32 : __clz(x);
}

// A tree's unique codes: written by an earlier kernel, or in shared memory.
struct GlobalCodes
{
  const uint32_t* c;
  __device__ __forceinline__ uint32_t operator[](int j) const { return __ldg(c + j); }
};
struct SharedCodes
{
  const uint32_t* c;
  __device__ __forceinline__ uint32_t operator[](int j) const { return c[j]; }
};

// delta() of core/builders/lbvh.cpp:386-403 against a code held in a
// register: the codes are unique after compaction, so this is the count of
// leading zeros of their XOR (32 for equal codes, -1 out of range).
template <typename Codes> __device__ __forceinline__ int karras_delta(const Codes& c, int L, uint32_t ci, int j)
{
  return j < 0 || j >= L ? -1 : clz_delta(ci, c[j]);
}

// Node i's code and its neighbours' deltas, exchanged across the warp: lane l
// handles absolute code index g (-1: no node); the neighbours' codes come
// from the adjacent lanes by __shfl_up_sync / __shfl_down_sync when those
// lanes hold indices g - 1 and g + 1 of the same tree, from memory otherwise
// (the warp's first and last lanes, tree boundaries of a segmented build).
// Every lane of the warp must call this.
__device__ __forceinline__ void karras_neighbours(const uint32_t* __restrict__ all, int segBase, int L, int i,
                                                  bool active, uint32_t& ci, int& dPrev, int& dNext)
{
  const int g = active ? segBase + i : -1;
  ci = active ? __ldg(all + g) : 0u;
  const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, ci, 1);
  const int gUp = __shfl_up_sync(0xFFFFFFFFu, g, 1);
  const uint32_t down = __shfl_down_sync(0xFFFFFFFFu, ci, 1);
  const int gDown = __shfl_down_sync(0xFFFFFFFFu, g, 1);
  const int lane = (int)(threadIdx.x & 31u);
  dPrev = -1;
  dNext = -1;
  if (!active) return;
  if (i >= 1) dPrev = clz_delta(ci, (lane > 0 && gUp == g - 1) ? up : __ldg(all + g - 1));
  if (i + 1 < L) dNext = clz_delta(ci, (lane < 31 && gDown == g + 1) ? down : __ldg(all + g + 1));
}

// kernel1D_Karras12 (core/builders/lbvh.cpp:405-441) for internal node i of a
// tree over L unique codes c (ci = c[i], dPrev / dNext = its deltas to the
// codes before and after it): direction from the neighbours' deltas, the
// range end by exponential then binary search, the split by binary search;
// children in the LR numbering (internal 0..L-2, leaves L-1..2L-2), `other` =
// the far end of the node's leaf range.
template <typename Codes>
__device__ __forceinline__ void karras_node(const Codes& c, int L, int i, uint32_t ci, int dPrev, int dNext,
                                            uint32_t& left, uint32_t& right, int& other)
{
  const int dl = dNext - dPrev;
  const int d = (dl > 0) - (dl < 0);
  const int dmin = d > 0 ? dPrev : (d < 0 ? dNext : 32);  // delta(i, i - d)
  int lmax = 2;
  while (karras_delta(c, L, ci, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t > 0; t >>= 1)
    if (karras_delta(c, L, ci, i + (l + t) * d) > dmin) l += t;
  const int j = i + l * d;
  const int dnode = karras_delta(c, L, ci, j);
  int s = 0;
  for (int t = (l + 1) >> 1; t > 0; t = (t == 1 ? 0 : (t + 1) >> 1))
    if (karras_delta(c, L, ci, i + (s + t) * d) > dnode) s += t;
  const int gamma = i + s * d + (d < 0 ? d : 0);
  left = ((i < j ? i : j) == gamma) ? (uint32_t)(L - 1 + gamma) : (uint32_t)gamma;
  right = ((i > j ? i : j) == gamma + 1) ? (uint32_t)(L - 1 + gamma + 1) : (uint32_t)(gamma + 1);
  other = j;
}

// A tree of distinct 30-bit codes is at most 31 levels deep; a climb longer
// than this is a cycle of inconsistent links.
constexpr int kMaxDepth = 40;

__device__ __forceinline__ uint32_t atomic_add_acq_rel_cta(uint32_t* p, uint32_t v)
{
  uint32_t old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], %2;"
               : "=r"(old)
               : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v)
               : "memory");
  return old;
}

// Index of the segment containing position x: the largest s with
// offsets[s] <= x, for ascending offsets[0..count] (offsets[0] = 0).
__device__ __forceinline__ uint32_t find_segment(const uint32_t* __restrict__ offsets, uint32_t count, uint32_t x)
{
  uint32_t lo = 0, hi = count;  // answer in [lo, hi)
  while (hi - lo > 1)
  {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(offsets + mid) <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Exclusive prefix of tile `tile` of a single-pass scan, by one warp (all 32
// lanes call): publishes the tile's sum, then looks back over the earlier
// tiles' words 32 at a time (decoupled look-back; the words carry flag and
// value together).  A thread walking back one word per load spends a load's
// latency on each tile that has no prefix yet; the run compaction of 2M codes took 37 us, with this and wide accesses 14.
// A wait that runs out is reported and ends the walk.
__device__ __forceinline__ uint32_t warp_look_back(uint32_t* tileStatus, uint32_t tile, uint32_t sum,
                                                   uint32_t* errorWord)
{
  const uint32_t lane = threadIdx.x & 31u;
  if (tile == 0)
  {
    if (lane == 0) store_relaxed(tileStatus, kFlagPrefix | sum);
    return 0u;
  }
  if (lane == 0) store_relaxed(tileStatus + tile, kFlagAgg | sum);
  uint32_t excl = 0;
  int64_t t = (int64_t)tile - 1;
  uint32_t spins = 0;
  while (true)
  {
    // lane k reads tile t - k; before the first tile stands a prefix of 0
    const int64_t mine = t - (int64_t)lane;
    const uint32_t w = mine >= 0 ? load_relaxed(tileStatus + mine) : kFlagPrefix;
    const uint32_t empty = __ballot_sync(0xFFFFFFFFu, (w & ~kValueMask) == 0u);
    const uint32_t prefix = __ballot_sync(0xFFFFFFFFu, (w & ~kValueMask) == kFlagPrefix);
    // lanes before the first empty word, up to and with the first prefix, count
    const uint32_t ready = empty ? (empty & (0u - empty)) - 1u : 0xFFFFFFFFu;
    const uint32_t ends = prefix & ready;
    const uint32_t use = ends ? ((ends & (0u - ends)) << 1) - 1u : ready;
    uint32_t v = (use >> lane) & 1u ? (w & kValueMask) : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    excl += v;
    if (ends) break;
    const int step = __popc(use);
    t -= step;
    if (step == 0)
    {
      if (++spins > kSpinLimit)
      {
        if (lane == 0) atomicOr(errorWord, kErrWaitTimeout);
        break;
      }
      if (spins > 64) __nanosleep(32);
    }
  }
  if (lane == 0) store_relaxed(tileStatus + tile, kFlagPrefix | (excl + sum));
  return excl;
}

// One tile (THREADS x kScanItems codes) of the run compaction
// (kernel1D_AppendInit + exclusive_scan + kernel1D_AppendComplete,
// core/builders/lbvh.cpp:289-319,762-767) as a single-pass scan with decoupled
// look-back: a position starts a run when its code differs from its
// predecessor's or (segmented build) when it starts a segment; run starts are
// appended to (compressed, runStarts) in order and the last tile writes the
// run count to *total.
//
// A thread takes 16 consecutive codes by four 128-bit loads and the runs leave
// through shared memory, so both sides move whole lines.
template <int THREADS>
__device__ __forceinline__ void compact_runs_tile(const uint32_t* __restrict__ keys, uint32_t n,
                                                  const uint32_t* __restrict__ segOffsets, uint32_t segCount,
                                                  uint32_t* __restrict__ compressed, uint32_t* __restrict__ runStarts,
                                                  uint32_t* tileStatus, uint32_t* tileCounter, uint32_t* total,
                                                  uint32_t* errorWord)
{
  constexpr uint32_t kTile = THREADS * kScanItems;
  static_assert(kScanItems == 16, "four 128-bit loads a thread");
  __shared__ uint32_t s_tile, s_prefix;
  __shared__ uint32_t s_warp[THREADS / 32 + 1];
  __shared__ uint32_t s_key[kTile];
  __shared__ uint16_t s_at[kTile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(tileCounter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t tileBase = tile * kTile, base = tileBase + tid * kScanItems;

  uint32_t key[kScanItems];
  if (base + kScanItems <= n)
  {
    // base is a multiple of 16 and the array starts at an allocation's boundary
    const uint4* p = reinterpret_cast<const uint4*>(keys + base);
#pragma unroll
    for (int q = 0; q < kScanItems / 4; q++)
    {
      const uint4 v = p[q];
      key[4 * q] = v.x; key[4 * q + 1] = v.y; key[4 * q + 2] = v.z; key[4 * q + 3] = v.w;
    }
  }
  else
  {
#pragma unroll
    for (int k = 0; k < kScanItems; k++) key[k] = base + k < n ? keys[base + k] : 0u;
  }
  uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, key[kScanItems - 1], 1);
  if (lane == 0) prev = (base > 0 && base - 1 < n) ? keys[base - 1] : 0u;
  uint32_t flags = 0, cnt = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++)
  {
    const uint32_t i = base + k;
    bool f = (i < n) && (i == 0 || key[k] != prev);
    if (segOffsets != nullptr && i < n && !f)
    {
      const uint32_t s = find_segment(segOffsets, segCount, i);
      f = (segOffsets[s] == i);
    }
    prev = key[k];
    flags |= (f ? 1u : 0u) << k;
    cnt += f ? 1u : 0u;
  }
  // block exclusive scan of cnt
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0)
  {
    constexpr int kWarps = THREADS / 32;
    uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
    uint32_t run = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, run, o);
      if (lane >= o) run += y;
    }
    const uint32_t sum = __shfl_sync(0xFFFFFFFFu, run, 31);
    if (lane < kWarps) s_warp[lane] = run - w;
    if (lane == 0) s_warp[kWarps] = sum;
    const uint32_t excl = warp_look_back(tileStatus, tile, sum, errorWord);
    if (lane == 0)
    {
      s_prefix = excl;
      const uint32_t tiles = (n + kTile - 1) / kTile;
      if (tile == tiles - 1) *total = (excl + sum <= n) ? excl + sum : n;
    }
  }
  __syncthreads();
  uint32_t local = s_warp[warp] + incl - cnt;
#pragma unroll
  for (int k = 0; k < kScanItems; k++)
    if (flags & (1u << k))
    {
      s_key[local] = key[k];
      s_at[local] = (uint16_t)(tid * kScanItems + k);
      local++;
    }
  __syncthreads();
  const uint32_t count = s_warp[THREADS / 32], prefix = s_prefix;
  for (uint32_t q = tid; q < count; q += THREADS)
    if (prefix + q < n)  // always true unless a look-back wait gave up (reported through errorWord)
    {
      compressed[prefix + q] = s_key[q];
      runStarts[prefix + q] = tileBase + s_at[q];
    }
}

}  // namespace bc
}  // namespace hrt
