// LBVH build on the GPU: scene box, Morton codes, stable sort, run compaction,
// leaves, Karras hierarchy, atomic bottom-up refit and the 64-byte traversal
// records.  Every stage reproduces the integer and float results of HeavyRT's
// LBVHBuilder (core/builders/lbvh.cpp) bit for bit; float arithmetic is written
// with explicit round-to-nearest intrinsics so that no multiply-add is fused.
#include <algorithm>

#include "build_common.cuh"
#include "hrt_kernels.cuh"
#include "leaf_tree.cuh"

namespace hrt
{
namespace
{

constexpr int kThreads = 256;

// ---------------------------------------------------------------- vertices and scene box
// The build's inputs read once: the indices copied, the vertices packed to
// float4 (w = 1), and in the same pass their box and the Morton scale
// (kernel1D_RedunctionFromVertices, core/builders/lbvh.cpp:228-239;
// ZIndexMultCoeff on the box widened by 1e-4, :41-51,263): each block leaves its
// part's bounds, the last block to finish (counted in *done, zero before)
// combines them.  min/max are exact, so only the sign of a zero bound can
// depend on the order; it never reaches a Morton code (+0 and -0 give the same
// quantised offset).  `reset` also clears the build's counters in params.
//
// The sources may be host memory read over the host link (page-locked, or
// pageable where the GPU translates through the host's page tables): reads are
// whole lines, tightly packed vertices by way of shared memory.  Bound by the
// link: 38 MB of numpy arrays in 186 us (205 GB/s); copied to the device first
// 210 + 10 us, and the load 890 us instead of 824.
//
// read_part: block `block` of `blocks` of THREADS threads takes its part of
// the vertices to out and to their bounds, its part of the indices to idx.
// sRaw: 3 * THREADS float4 of shared memory.
template <int THREADS>
__device__ __forceinline__ void read_part(const uint8_t* raw, uint64_t stride, uint32_t n, float4* out,
                                          const uint32_t* idxSrc, uint32_t* idx, uint64_t nIdx, uint32_t block,
                                          uint32_t blocks, float4* sRaw, float (&mn)[4], float (&mx)[4])
{
  constexpr uint32_t kTile = 4 * THREADS;  // vertices of a step (12-byte stride)
  auto take = [&](uint32_t i, float x, float y, float z) {
    const float v[4] = {x, y, z, 1.0f};
    out[i] = make_float4(x, y, z, 1.0f);
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
      mn[k] = lm_min(mn[k], v[k]);
      mx[k] = lm_max(mx[k], v[k]);
    }
  };
  const bool aligned = (reinterpret_cast<uintptr_t>(raw) & 15u) == 0u;
  if (stride == 12 && aligned)
  {
    for (uint64_t v0 = (uint64_t)block * kTile; v0 < n; v0 += (uint64_t)blocks * kTile)
    {
      const uint32_t count = (uint32_t)min((uint64_t)kTile, n - v0);
      const uint32_t pieces = 3 * count / 4;  // whole 16-byte pieces
      const float4* src = reinterpret_cast<const float4*>(raw + 12 * v0);
#pragma unroll
      for (int q = 0; q < 3; q++)
      {
        const uint32_t k = q * THREADS + threadIdx.x;
        if (k < pieces) sRaw[k] = src[k];
      }
      float* words = reinterpret_cast<float*>(sRaw);
      if (threadIdx.x < 3 * count - 4 * pieces)
        words[4 * pieces + threadIdx.x] = reinterpret_cast<const float*>(src)[4 * pieces + threadIdx.x];
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; q++)
      {
        const uint32_t k = q * THREADS + threadIdx.x;
        if (k < count) take((uint32_t)(v0 + k), words[3 * k], words[3 * k + 1], words[3 * k + 2]);
      }
      __syncthreads();
    }
  }
  else if (stride == 16 && aligned)
  {
    for (uint32_t i = block * THREADS + threadIdx.x; i < n; i += blocks * THREADS)
    {
      const float4 p = reinterpret_cast<const float4*>(raw)[i];
      take(i, p.x, p.y, p.z);
    }
  }
  else
    for (uint32_t i = block * THREADS + threadIdx.x; i < n; i += blocks * THREADS)
    {
      const float* p = reinterpret_cast<const float*>(raw + (size_t)i * stride);
      take(i, p[0], p[1], p[2]);
    }
  if (idxSrc != idx)
  {
    const uint64_t step = (uint64_t)blocks * THREADS, first = (uint64_t)block * THREADS + threadIdx.x;
    const uint64_t whole = (reinterpret_cast<uintptr_t>(idxSrc) & 15u) == 0u ? nIdx / 4 : 0;  // idx starts an allocation
#pragma unroll 4
    for (uint64_t k = first; k < whole; k += step)
      reinterpret_cast<uint4*>(idx)[k] = reinterpret_cast<const uint4*>(idxSrc)[k];
    for (uint64_t k = 4 * whole + first; k < nIdx; k += step) idx[k] = idxSrc[k];
  }
}

// The bounds of a block's threads to thread 0.
template <int THREADS> __device__ __forceinline__ void block_bounds(float (&mn)[4], float (&mx)[4])
{
  __shared__ float smn[THREADS / 32][4], smx[THREADS / 32][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 4; k++)
    {
      mn[k] = lm_min(mn[k], __shfl_down_sync(0xFFFFFFFFu, mn[k], o));
      mx[k] = lm_max(mx[k], __shfl_down_sync(0xFFFFFFFFu, mx[k], o));
    }
  if (lane == 0)
    for (int k = 0; k < 4; k++) { smn[warp][k] = mn[k]; smx[warp][k] = mx[k]; }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < THREADS / 32; w++)
      for (int k = 0; k < 4; k++) { mn[k] = lm_min(mn[k], smn[w][k]); mx[k] = lm_max(mx[k], smx[w][k]); }
}

struct ReadArgs
{
  const uint8_t*  raw;
  uint64_t        stride;
  uint32_t        n;
  float4*         out;
  const uint32_t* idxSrc;
  uint32_t*       idx;
  uint64_t        nIdx;
  float4*         partial;
  uint32_t*       done;
  BuildParams*    params;
  int             cubic, reset;
};

__device__ __forceinline__ void read_inputs(const ReadArgs& a, uint32_t block, uint32_t blocks)
{
  float mn[4] = {1e10f, 1e10f, 1e10f, 1e10f}, mx[4] = {-1e10f, -1e10f, -1e10f, -1e10f};
  __shared__ float4 s_raw[3 * kThreads];
  __shared__ bool   s_last;
  read_part<kThreads>(a.raw, a.stride, a.n, a.out, a.idxSrc, a.idx, a.nIdx, block, blocks, s_raw, mn, mx);
  block_bounds<kThreads>(mn, mx);
  if (threadIdx.x == 0)
  {
    a.partial[2 * block + 0] = make_float4(mn[0], mn[1], mn[2], mn[3]);
    a.partial[2 * block + 1] = make_float4(mx[0], mx[1], mx[2], mx[3]);
    s_last = bc::atomic_add_acq_rel(a.done, 1u) == blocks - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  for (int k = 0; k < 4; k++) { mn[k] = 1e10f; mx[k] = -1e10f; }
  for (uint32_t b = threadIdx.x; b < blocks; b += kThreads)
  {
    const float4 lo = __ldcg(a.partial + 2 * b), hi = __ldcg(a.partial + 2 * b + 1);
    mn[0] = lm_min(mn[0], lo.x); mn[1] = lm_min(mn[1], lo.y); mn[2] = lm_min(mn[2], lo.z); mn[3] = lm_min(mn[3], lo.w);
    mx[0] = lm_max(mx[0], hi.x); mx[1] = lm_max(mx[1], hi.y); mx[2] = lm_max(mx[2], hi.z); mx[3] = lm_max(mx[3], hi.w);
  }
  block_bounds<kThreads>(mn, mx);
  if (threadIdx.x != 0) return;
  bc::zindex_scale(mn, mx, a.params, a.cubic);
  if (a.reset)
  {
    a.params->nLeaves = 0;
    a.params->error = 0;
    a.params->rootRecord = 0;
    a.params->pad = 0;
  }
}

__global__ void __launch_bounds__(kThreads) k_read_inputs(ReadArgs a) { read_inputs(a, blockIdx.x, gridDim.x); }

// ---------------------------------------------------------------- Morton codes
// kernel1D_EvalMortonCodesFromTriangles, core/builders/lbvh.cpp:259-287: box
// centre (or the centroid 0.33333333*(v1+v2+v3) when fewer than 256
// triangles), quantised against the scene box with truncation toward zero.
//
// The same pass counts the codes' four 8-bit digits for the sort (hist, zero
// before) and keeps the unsorted codes: reading the codes again for either was
// 12 us of a 2M-triangle build.  A block takes kMortonItems consecutive tiles,
// so neighbouring triangles, which share their upper digits, meet in one
// block's counters; a warp whose codes agree in a digit adds once.
constexpr int kMortonItems = 16;

__global__ void __launch_bounds__(kThreads) k_morton(const float4* __restrict__ v, const uint32_t* __restrict__ idx,
                                                     uint32_t nTris, uint32_t nVerts, const BuildParams* __restrict__ params,
                                                     uint32_t* __restrict__ keys, uint32_t* __restrict__ unsorted,
                                                     uint32_t* __restrict__ vals, uint32_t* __restrict__ hist,
                                                     uint32_t* errorWord)
{
  __shared__ uint32_t s_hist[4 * 256];
  for (int k = threadIdx.x; k < 4 * 256; k += kThreads) s_hist[k] = 0u;
  __syncthreads();
#pragma unroll 1
  for (int it = 0; it < kMortonItems; it++)
  {
    const uint64_t i64 = ((uint64_t)blockIdx.x * kMortonItems + it) * kThreads + threadIdx.x;
    const bool in = i64 < nTris;
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, in);
    if (mask == 0u) break;
    const uint32_t i = (uint32_t)i64;
    uint32_t code = 0;
    if (in)
    {
      uint32_t ia = idx[3 * (size_t)i + 0], ib = idx[3 * (size_t)i + 1], ic = idx[3 * (size_t)i + 2];
      if (ia >= nVerts || ib >= nVerts || ic >= nVerts)
      {
        atomicOr(errorWord, kErrIndexRange);
        ia = ib = ic = 0;
      }
      code = bc::morton_code(v[ia], v[ib], v[ic], nTris, params->bmin, params->scale);
      keys[i] = code;
      unsorted[i] = code;
      vals[i] = i;
    }
    bc::count_digits(code, in, mask, s_hist);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 4 * 256; k += kThreads)
    if (s_hist[k]) atomicAdd(&hist[k], s_hist[k]);
}

// ---------------------------------------------------------------- run compaction
// kernel1D_AppendInit + exclusive_scan + kernel1D_AppendComplete
// (core/builders/lbvh.cpp:289-319,762-767) as one single-pass scan with
// decoupled look-back: flag = code differs from its predecessor; flagged
// positions are appended to (compressed, runStarts) in order.
constexpr uint32_t kScanTile = kThreads * bc::kScanItems;

__global__ void __launch_bounds__(kThreads) k_compact_runs(const uint32_t* __restrict__ keys, uint32_t n,
                                                           uint32_t* __restrict__ compressed,
                                                           uint32_t* __restrict__ runStarts, uint32_t* tileStatus,
                                                           uint32_t* tileCounter, BuildParams* params,
                                                           uint32_t* errorWord)
{
  bc::compact_runs_tile<kThreads>(keys, n, nullptr, 0u, compressed, runStarts, tileStatus, tileCounter,
                                  &params->nLeaves, errorWord);
}

// ---------------------------------------------------------------- Karras 2012
// delta() and kernel1D_Karras12, core/builders/lbvh.cpp:386-441.  The codes
// are unique after compaction, so delta(i,j) is the count of leading zeros of
// their XOR (32 for equal codes, -1 out of range, as the reference defines).
__device__ __forceinline__ void karras(const uint32_t* __restrict__ codes, const BuildParams* __restrict__ params,
                                       BVHNode32* __restrict__ lr, uint32_t* __restrict__ parent,
                                       uint32_t* __restrict__ visit, uint32_t* __restrict__ rangeEnd, uint32_t block,
                                       uint32_t blocks)
{
  const int L = (int)params->nLeaves;
  // one node per thread; a warp's 32 consecutive nodes exchange their codes
  // for the direction test (karras_neighbours), so the loop bound is uniform
  // over the warp
  const int lane = (int)(threadIdx.x & 31u);
  for (int base = (int)(block * kThreads + (threadIdx.x & ~31u)); base < L - 1; base += blocks * kThreads)
  {
    const int i = base + lane;
    const bool active = i < L - 1;
    uint32_t ci;
    int dPrev, dNext;
    bc::karras_neighbours(codes, 0, L, i, active, ci, dPrev, dNext);
    if (!active) continue;
    uint32_t left, right;
    int other;
    bc::karras_node(bc::GlobalCodes{codes}, L, i, ci, dPrev, dNext, left, right, other);
    lr[i].leftOffset = left;
    lr[i].escapeIndex = right;
    parent[left] = (uint32_t)i;
    parent[right] = (uint32_t)i;
    rangeEnd[i] = (uint32_t)other;
    visit[i] = 0u;
  }
}

__global__ void __launch_bounds__(kThreads) k_karras(const uint32_t* __restrict__ codes,
                                                     const BuildParams* __restrict__ params, BVHNode32* __restrict__ lr,
                                                     uint32_t* __restrict__ parent, uint32_t* __restrict__ visit,
                                                     uint32_t* __restrict__ rangeEnd)
{
  karras(codes, params, lr, parent, visit, rangeEnd, blockIdx.x, gridDim.x);
}

// A refit's new vertices and, by the blocks after the first readBlocks, its
// unchanged hierarchy's links: the reads wait on the host link and the links
// on L2 (a refit of 500,000 triangles with its frame 266 us, 242 so).
__global__ void __launch_bounds__(kThreads) k_read_and_link(ReadArgs a, uint32_t readBlocks,
                                                            const uint32_t* __restrict__ codes,
                                                            const BuildParams* __restrict__ params,
                                                            BVHNode32* __restrict__ lr, uint32_t* __restrict__ parent,
                                                            uint32_t* __restrict__ visit, uint32_t* __restrict__ rangeEnd)
{
  if (blockIdx.x < readBlocks) read_inputs(a, blockIdx.x, readBlocks);
  else karras(codes, params, lr, parent, visit, rangeEnd, blockIdx.x - readBlocks, gridDim.x - readBlocks);
}

// ---------------------------------------------------------------- traversal records
// One 64-byte record per internal node holding both children (the reference's
// sibling pair, core/BVH2CommonRT.cpp:91-92).  With a single leaf the record
// holds that leaf and an empty slot, as the reference pairs a lone root leaf
// with a dummy node (core/builders/lbvh.cpp:497-503, core/builders/cbvh.h:28-36).
__global__ void __launch_bounds__(kThreads) k_records(BuildParams* __restrict__ params,
                                                      const BVHNode32* __restrict__ lr,
                                                      const uint32_t* __restrict__ visit,
                                                      const uint32_t* __restrict__ runStarts, PairRec* __restrict__ recs)
{
  const uint32_t L = params->nLeaves;
  const uint32_t first = blockIdx.x * kThreads + threadIdx.x;
  if (first == 0 && L >= 2u && visit[0] != 2u) atomicOr(&params->error, kErrLayout);  // the refit reached the root
  if (L == 1u)
  {
    if (first == 0)
    {
      const BVHNode32 n = lr[0];
      PairRec r;
      r.a = make_float4(n.boxMin[0], n.boxMin[1], n.boxMin[2], n.boxMax[0]);
      r.b = make_float4(n.boxMax[1], n.boxMax[2], 0.0f, 0.0f);
      r.c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      r.d = make_uint4(kLeafBit | runStarts[0], kEmptyRef, 0u, 0u);
      recs[0] = r;
    }
    return;
  }
  for (uint32_t i = first; i + 1 < L; i += gridDim.x * kThreads)
  {
    const uint32_t left = lr[i].leftOffset, right = lr[i].escapeIndex;
    const BVHNode32 a = bc::load_node(lr + left);
    const BVHNode32 b = bc::load_node(lr + right);
    const uint32_t lref = (left < L - 1) ? left : (kLeafBit | runStarts[left - (L - 1)]);
    const uint32_t rref = (right < L - 1) ? right : (kLeafBit | runStarts[right - (L - 1)]);
    PairRec r;
    r.a = make_float4(a.boxMin[0], a.boxMin[1], a.boxMin[2], a.boxMax[0]);
    r.b = make_float4(a.boxMax[1], a.boxMax[2], b.boxMin[0], b.boxMin[1]);
    r.c = make_float4(b.boxMin[2], b.boxMax[0], b.boxMax[1], b.boxMax[2]);
    r.d = make_uint4(lref, rref, 0u, 0u);
    recs[i] = r;
  }
}

// ---------------------------------------------------------------- small geometries
// Inputs, box, codes, sort, runs and hierarchy of a geometry of at most
// kSmallTris triangles in one block: the arrays that the kernels above would
// write.  Each of those nine launches is shorter than the gap before it.  The
// sort is a bitonic one of (code, triangle) pairs, which are distinct, so its
// order is the stable one by code; steps within 64 pairs stay inside a warp.
// Bound by the block's chain of steps, so the gain goes as the geometry grows:
// a load of 512 triangles 147 us with one kernel a stage, 92 so; of 2,000 171
// and 132, of 4,096 186 and 178.  The commit of 240 instances, whose tree is
// such a geometry: 173 us, 97 so.
constexpr int      kSmallThreads = 512;
constexpr uint32_t kSmallTris = 4096, kSmallVerts = 3 * kSmallTris;

__global__ void __launch_bounds__(kSmallThreads) k_small_front(BuildBuffers b)
{
  __shared__ union __align__(16)
  {
    float4             raw[3 * kSmallThreads];
    unsigned long long pair[kSmallTris];
    uint32_t           code[kSmallTris];
  } sh;
  __shared__ BuildParams s_params;
  __shared__ uint32_t    s_warpRuns[kSmallThreads / 32];
  const uint32_t N = b.nTris, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;

  float mn[4] = {1e10f, 1e10f, 1e10f, 1e10f}, mx[4] = {-1e10f, -1e10f, -1e10f, -1e10f};
  read_part<kSmallThreads>(b.raw, b.rawStride, b.nVerts, b.verts, b.idxSrc, b.idx, 3 * (uint64_t)N, 0u, 1u, sh.raw, mn,
                           mx);
  block_bounds<kSmallThreads>(mn, mx);
  if (tid == 0)
  {
    bc::zindex_scale(mn, mx, &s_params, b.mortonCubic);
    s_params.nLeaves = s_params.error = s_params.rootRecord = s_params.pad = 0;
  }
  __syncthreads();

  // codes, padded to a power of two
  uint32_t P = 64;
  while (P < N) P <<= 1;
  for (uint32_t i = tid; i < P; i += kSmallThreads)
  {
    if (i >= N)
    {
      sh.pair[i] = ~0ull;
      continue;
    }
    uint32_t ia = b.idx[3 * i], ib = b.idx[3 * i + 1], ic = b.idx[3 * i + 2];
    if (ia >= b.nVerts || ib >= b.nVerts || ic >= b.nVerts)
    {
      atomicOr(&s_params.error, kErrIndexRange);
      ia = ib = ic = 0;
    }
    const uint32_t code = bc::morton_code(b.verts[ia], b.verts[ib], b.verts[ic], N, s_params.bmin, s_params.scale);
    b.keysUnsorted[i] = code;
    sh.pair[i] = (unsigned long long)code << 32 | i;
  }
  __syncthreads();

  for (uint32_t k = 2; k <= P; k <<= 1)
    for (uint32_t j = k >> 1; j > 0; j >>= 1)
    {
      for (uint32_t p = tid; p < P / 2; p += kSmallThreads)
      {
        const uint32_t i = 2 * p - (p & (j - 1));
        const unsigned long long x = sh.pair[i], y = sh.pair[i + j];
        if ((x > y) == ((i & k) == 0))
        {
          sh.pair[i] = y;
          sh.pair[i + j] = x;
        }
      }
      // a step within 64 pairs, before another such one, is the warp's own
      if (j > 32 || (j == 1 && k > 32)) __syncthreads();
      else __syncwarp();
    }
  __syncthreads();

  // runs: a warp's codes are consecutive
  constexpr int kPer = kSmallTris / kSmallThreads;
  uint32_t code[kPer], starts[kPer], runs = 0;
#pragma unroll
  for (int q = 0; q < kPer; q++)
  {
    const uint32_t i = (warp * kPer + q) * 32 + lane;
    code[q] = 0;
    bool start = false;
    if (i < N)
    {
      const unsigned long long x = sh.pair[i];
      code[q] = (uint32_t)(x >> 32);
      b.keys[i] = code[q];
      b.vals[i] = (uint32_t)x;
      start = i == 0 || (uint32_t)(sh.pair[i - 1] >> 32) != code[q];
    }
    starts[q] = __ballot_sync(0xFFFFFFFFu, start);
    runs += __popc(starts[q]);
  }
  if (lane == 0) s_warpRuns[warp] = runs;
  __syncthreads();
  uint32_t at = 0, L = 0;
#pragma unroll
  for (uint32_t w = 0; w < kSmallThreads / 32; w++)
  {
    at += w < warp ? s_warpRuns[w] : 0u;
    L += s_warpRuns[w];
  }
#pragma unroll
  for (int q = 0; q < kPer; q++)
  {
    if ((starts[q] >> lane) & 1u)
    {
      const uint32_t r = at + __popc(starts[q] & ((1u << lane) - 1u));
      sh.code[r] = code[q];
      b.compressed[r] = code[q];
      b.runStarts[r] = (warp * kPer + q) * 32 + lane;
    }
    at += __popc(starts[q]);
  }
  __syncthreads();

  const bc::SharedCodes codes{sh.code};
  for (int i = (int)tid; i < (int)L - 1; i += kSmallThreads)
  {
    const uint32_t ci = codes[i];
    uint32_t left, right;
    int other;
    bc::karras_node(codes, (int)L, i, ci, bc::karras_delta(codes, (int)L, ci, i - 1),
                    bc::karras_delta(codes, (int)L, ci, i + 1), left, right, other);
    b.lr[i].leftOffset = left;
    b.lr[i].escapeIndex = right;
    b.parent[left] = (uint32_t)i;
    b.parent[right] = (uint32_t)i;
    b.visit[N + i] = (uint32_t)other;
    b.visit[i] = 0u;
  }
  if (tid == 0)
  {
    s_params.nLeaves = L;
    *b.params = s_params;
  }
}

inline uint32_t grid_for(uint64_t n, int numSMs, int perSM = 8)
{
  uint64_t g = (n + kThreads - 1) / kThreads;
  const uint64_t cap = (uint64_t)numSMs * perSM;
  if (g > cap) g = cap;
  return g == 0 ? 1u : (uint32_t)g;
}

}  // namespace

namespace
{
constexpr size_t up256(size_t b) { return (b + 255) / 256 * 256; }
constexpr uint32_t kBoxBlocks = 1024;  // most blocks of k_read_inputs

// Build scratch: what starts at zero first (box and scan counters, scan tile
// status, the sort's scratch), then the box parts.
struct BuildScratch
{
  uint32_t *boxDone, *scanCounter, *scanStatus;
  void*     sort;
  float4*   partial;
  size_t    zeroBytes, bytes;
};
BuildScratch build_scratch(void* scratch, uint32_t nTris)
{
  const size_t scanTiles = (nTris + kScanTile - 1) / kScanTile;
  char* p = (char*)scratch;
  BuildScratch q;
  size_t at = 256;
  q.boxDone = (uint32_t*)p;
  q.scanCounter = q.boxDone + 1;
  q.scanStatus = (uint32_t*)(p + at);
  at += up256(4 * scanTiles);
  q.sort = p + at;
  at += up256(radix_sort_scratch_bytes(nTris));
  q.zeroBytes = at;
  q.partial = (float4*)(p + at);
  q.bytes = at + 2 * sizeof(float4) * kBoxBlocks;
  return q;
}

ReadArgs read_args(const BuildBuffers& b, float4* partial, uint32_t* done, BuildParams* params, int reset)
{
  return {b.raw, b.rawStride, b.nVerts, b.verts, b.idxSrc, b.idx, 3 * (uint64_t)b.nTris, partial, done, params,
          b.mortonCubic, reset};
}
uint32_t read_blocks(const BuildBuffers& b, int numSMs)
{
  return std::min(kBoxBlocks, grid_for(std::max<uint64_t>(b.nVerts, 3 * (uint64_t)b.nTris / 4), numSMs, 4));
}

// Leaves, boxes and (binary layout) pair records, from the sorted triangles,
// the unique codes and the hierarchy.  lists: build_list_words() of scratch.
cudaError_t build_tree(const BuildBuffers& b, uint32_t* lists, int numSMs, cudaStream_t s)
{
  const uint32_t N = b.nTris;
  bc::LeafTree t = {};
  t.verts = b.verts;
  t.idx = b.idx;
  t.sortedTri = b.vals;
  t.runStarts = b.runStarts;
  t.nTris = N;
  t.nVerts = b.nVerts;
  t.lr = b.lr;
  t.lrCount = b.lrCount;
  t.tris = b.tris;
  t.sortedIdx = b.sortedIdx;
  t.parent = b.parent;
  t.visit = b.visit;
  t.rangeEnd = b.visit + N;
  t.lists = lists;
  t.errorWord = &b.params->error;
  t.vertexRecords = b.vertexRecords;
  t.params = b.params;
  const cudaError_t e = bc::leaf_tree<false>(t, s);
  if (e != cudaSuccess) return e;
  if (b.recs) k_records<<<grid_for(N, numSMs, 8), kThreads, 0, s>>>(b.params, b.lr, b.visit, b.runStarts, b.recs);
  return cudaGetLastError();
}
}  // namespace

size_t build_list_words(uint32_t nTris) { return bc::list_words(nTris); }
size_t build_scratch_bytes(uint32_t nTris) { return build_scratch(nullptr, nTris).bytes; }

cudaError_t build_lbvh(const BuildBuffers& b, int numSMs, cudaStream_t s)
{
  const uint32_t N = b.nTris;
  if (N == 0) return cudaSuccess;
  const BuildScratch q = build_scratch(b.scratch, N);
  uint32_t* err = &b.params->error;
  if (N <= kSmallTris && b.nVerts <= kSmallVerts)
  {
    k_small_front<<<1, kSmallThreads, 0, s>>>(b);
    const cudaError_t se = cudaGetLastError();
    if (se != cudaSuccess) return se;
    return build_tree(b, b.keysAlt, numSMs, s);
  }
  cudaError_t e = cudaMemsetAsync(b.scratch, 0, q.zeroBytes, s);
  if (e != cudaSuccess) return e;
  // 1. inputs, scene box and Morton scale
  k_read_inputs<<<read_blocks(b, numSMs), kThreads, 0, s>>>(read_args(b, q.partial, q.boxDone, b.params, 1));
  // 2. Morton codes and their digits' counts
  constexpr uint32_t kPerBlock = kThreads * kMortonItems;
  k_morton<<<(N + kPerBlock - 1) / kPerBlock, kThreads, 0, s>>>(b.verts, b.idx, N, b.nVerts, b.params, b.keys,
                                                                 b.keysUnsorted, b.vals, (uint32_t*)q.sort, err);
  // 3. stable sort by code
  e = radix_sort_pairs(b.keys, b.vals, b.keysAlt, b.valsAlt, N, q.sort, err, numSMs, s, true);
  if (e != cudaSuccess) return e;
  // 4. unique codes and run starts
  k_compact_runs<<<(N + kScanTile - 1) / kScanTile, kThreads, 0, s>>>(b.keys, N, b.compressed, b.runStarts, q.scanStatus,
                                                                      q.scanCounter, b.params, err);
  // 5. hierarchy, leaves, boxes, records; the sort's spare array holds the lists
  k_karras<<<grid_for(N, numSMs, 8), kThreads, 0, s>>>(b.compressed, b.params, b.lr, b.parent, b.visit, b.visit + N);
  return build_tree(b, b.keysAlt, numSMs, s);
}

// Refit: the geometry's vertices moved, its triangles and their sorted order
// did not.  Leaves, triangle records and the sorted index buffer are rewritten
// from the new vertices in the existing order, the hierarchy's parent links are
// recomputed from the unchanged codes, and the boxes refit bottom-up; the
// Morton frame in params stays that of the build.  The geometry's new vertex
// box goes to boxOut (bmin/bmax).
cudaError_t refit_lbvh(const BuildBuffers& b, BuildParams* boxOut, int numSMs, cudaStream_t s)
{
  if (b.nTris == 0) return cudaSuccess;
  uint32_t* done = (uint32_t*)b.scratch;  // refit_scratch_bytes(): a counter, box parts, lists
  float4* partial = (float4*)((char*)b.scratch + 256);
  cudaError_t e = cudaMemsetAsync(done, 0, sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  const uint32_t reads = read_blocks(b, numSMs), links = grid_for(b.nTris, numSMs, 4);
  k_read_and_link<<<reads + links, kThreads, 0, s>>>(read_args(b, partial, done, boxOut, 0), reads, b.compressed, b.params,
                                                     b.lr, b.parent, b.visit, b.visit + b.nTris);
  return build_tree(b, (uint32_t*)(partial + 2 * kBoxBlocks), numSMs, s);
}

size_t refit_scratch_bytes(uint32_t nTris) { return 256 + 2 * sizeof(float4) * kBoxBlocks + 4 * build_list_words(nTris); }

}  // namespace hrt
