// Segmented LBVH build: many independent geometries built by one launch per
// stage over their concatenated triangles.
//
// Every geometry gets exactly the arrays its single build would produce (same
// scene box, Morton codes, stable order, runs, Karras tree, refit boxes and
// traversal records) at its own offsets:
//   triangles  [triOffsets[s], triOffsets[s+1])            keys, vals, TriRec, sorted index buffer
//   runs       [leafOffsets[s], leafOffsets[s+1])          compressed codes, run starts
//   LR nodes   [nodeOffsets[s], nodeOffsets[s] + 2L-1)     Karras + refit tree, local numbering
//   records    [recOffsets[s], recOffsets[s] + max(L-1,1)) child-pair records, local references
// The per-geometry box uses the geometry's own vertices and the centroid rule
// uses the geometry's own triangle count (core/builders/lbvh.cpp:279); the
// sort is the stable segmented radix sort; a run never crosses a segment.
#include "build_common.cuh"
#include "hrt_kernels.cuh"
#include "leaf_tree.cuh"

namespace hrt
{
namespace
{

constexpr int kThreads = 256;
using bc::find_segment;

// The inputs of all geometries read once, a block per chunk: vertices packed to
// float4 (w = 1) with the chunk's bounds (geometry s owns chunks
// [boxChunkOffsets[s], boxChunkOffsets[s + 1])), and indices copied.  The sources
// are the caller's arrays, one per geometry, wherever the kernel reaches them:
// reads over the host link are whole lines, tightly packed vertices by way of
// shared memory (as k_read_inputs in build.cu).  Min / max are exact, so the box
// is the reference's (core/builders/lbvh.cpp:228-239; init +-1e10, :53).
// 48 soups, 26 MB: copied by the host into one array and to the device 1,550 us,
// so 130 us.
__global__ void __launch_bounds__(kThreads) k_seg_read_inputs(BatchBuffers b)
{
  if (blockIdx.x >= b.nBoxChunks)
  {
    const uint32_t k = blockIdx.x - b.nBoxChunks;
    const uint32_t s = find_segment(b.idxChunkOffsets, b.G, k);
    const uint32_t first = (k - b.idxChunkOffsets[s]) * kBatchIdxChunk, t0 = b.triOffsets[s];
    const uint32_t n = 3u * (b.triOffsets[s + 1] - t0);  // at most 3 * 2^24 words
    const uint32_t end = min(first + kBatchIdxChunk, n);
    const uint32_t* src = b.rawIdx[s];
    uint32_t* dst = b.idx + 3 * (size_t)t0;
    uint32_t at = first;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0u)
    {
      const uint32_t pieces = (end - first) / 4;
#pragma unroll 4
      for (uint32_t q = threadIdx.x; q < pieces; q += kThreads)
      {
        const uint4 v = reinterpret_cast<const uint4*>(src + first)[q];
        uint32_t* o = dst + first + 4 * q;
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        o[3] = v.w;
      }
      at = first + 4 * pieces;
    }
    for (uint32_t i = at + threadIdx.x; i < end; i += kThreads) dst[i] = src[i];
    return;
  }
  const uint32_t k = blockIdx.x;
  const uint32_t s = find_segment(b.boxChunkOffsets, b.G, k);
  const uint32_t v0 = b.vertOffsets[s], first = (k - b.boxChunkOffsets[s]) * kBatchBoxChunk;
  const uint32_t end = min(first + kBatchBoxChunk, b.vertOffsets[s + 1] - v0);
  const uint8_t* raw = b.rawVerts[s] + (size_t)first * b.rawStride;  // first vertex of the chunk
  float4* out = b.verts + (size_t)v0 + first;
  const uint32_t n = end - first;
  float mn[4] = {1e10f, 1e10f, 1e10f, 1e10f}, mx[4] = {-1e10f, -1e10f, -1e10f, -1e10f};
  auto take = [&](uint32_t i, float x, float y, float z) {
    const float v[4] = {x, y, z, 1.0f};
    out[i] = make_float4(x, y, z, 1.0f);
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      mn[q] = lm_min(mn[q], v[q]);
      mx[q] = lm_max(mx[q], v[q]);
    }
  };
  const bool aligned = (reinterpret_cast<uintptr_t>(raw) & 15u) == 0u;
  if (b.rawStride == 12 && aligned)
  {
    __shared__ float4 s_raw[3 * kBatchBoxChunk / 4];
    float* words = reinterpret_cast<float*>(s_raw);
    const uint32_t pieces = 3 * n / 4;  // whole 16-byte pieces
#pragma unroll 6
    for (uint32_t q = threadIdx.x; q < pieces; q += kThreads) s_raw[q] = reinterpret_cast<const float4*>(raw)[q];
    for (uint32_t q = 4 * pieces + threadIdx.x; q < 3 * n; q += kThreads) words[q] = reinterpret_cast<const float*>(raw)[q];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kThreads) take(i, words[3 * i], words[3 * i + 1], words[3 * i + 2]);
  }
  else if (b.rawStride == 16 && aligned)
  {
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n; i += kThreads)
    {
      const float4 p = reinterpret_cast<const float4*>(raw)[i];
      take(i, p.x, p.y, p.z);
    }
  }
  else
    for (uint32_t i = threadIdx.x; i < n; i += kThreads)
    {
      const float* p = reinterpret_cast<const float*>(raw + (size_t)i * b.rawStride);
      take(i, p[0], p[1], p[2]);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      mn[q] = lm_min(mn[q], __shfl_down_sync(0xFFFFFFFFu, mn[q], o));
      mx[q] = lm_max(mx[q], __shfl_down_sync(0xFFFFFFFFu, mx[q], o));
    }
  __shared__ float smn[kThreads / 32][4], smx[kThreads / 32][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int q = 0; q < 4; q++) { smn[warp][q] = mn[q]; smx[warp][q] = mx[q]; }
  __syncthreads();
  if (threadIdx.x == 0)
  {
    for (int w = 1; w < kThreads / 32; w++)
      for (int q = 0; q < 4; q++) { mn[q] = lm_min(mn[q], smn[w][q]); mx[q] = lm_max(mx[q], smx[w][q]); }
    b.boxPartial[2 * k] = make_float4(mn[0], mn[1], mn[2], mn[3]);
    b.boxPartial[2 * k + 1] = make_float4(mx[0], mx[1], mx[2], mx[3]);
  }
}

// The chunks of each geometry combined, a warp each.
__global__ void __launch_bounds__(kThreads) k_seg_box_final(const uint32_t* __restrict__ chunkOffsets, uint32_t G,
                                                            const float4* __restrict__ partial, BuildParams* params,
                                                            int cubic)
{
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t s = (blockIdx.x * kThreads + threadIdx.x) >> 5; s < G; s += (gridDim.x * kThreads) >> 5)
  {
    float mn[4] = {1e10f, 1e10f, 1e10f, 1e10f}, mx[4] = {-1e10f, -1e10f, -1e10f, -1e10f};
    for (uint32_t k = chunkOffsets[s] + lane; k < chunkOffsets[s + 1]; k += 32)
    {
      const float4 a = partial[2 * k], c = partial[2 * k + 1];
      mn[0] = lm_min(mn[0], a.x); mn[1] = lm_min(mn[1], a.y); mn[2] = lm_min(mn[2], a.z); mn[3] = lm_min(mn[3], a.w);
      mx[0] = lm_max(mx[0], c.x); mx[1] = lm_max(mx[1], c.y); mx[2] = lm_max(mx[2], c.z); mx[3] = lm_max(mx[3], c.w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < 4; q++)
      {
        mn[q] = lm_min(mn[q], __shfl_down_sync(0xFFFFFFFFu, mn[q], o));
        mx[q] = lm_max(mx[q], __shfl_down_sync(0xFFFFFFFFu, mx[q], o));
      }
    if (lane == 0)
    {
      bc::zindex_scale(mn, mx, &params[s], cubic);
      params[s].nLeaves = 0;
      params[s].error = 0;
      params[s].rootRecord = 0;
      params[s].pad = 0;
    }
  }
}

// The codes, their digits' counts for the sort (hist, zero before) and the
// unsorted codes, as k_morton in build.cu.  Counted and copied in passes of
// their own, 7 + 5 us of a batch of 48 geometries.
constexpr int kMortonItems = 4;

__global__ void __launch_bounds__(kThreads) k_seg_morton(const float4* __restrict__ v, const uint32_t* __restrict__ idx,
                                                         const uint32_t* __restrict__ vertOffsets,
                                                         const uint32_t* __restrict__ triOffsets, uint32_t G,
                                                         uint32_t N, const BuildParams* __restrict__ params,
                                                         uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                         uint32_t* __restrict__ unsorted, uint32_t* __restrict__ hist,
                                                         uint32_t* errorWord)
{
  __shared__ uint32_t s_hist[4 * 256];
  for (int k = threadIdx.x; k < 4 * 256; k += kThreads) s_hist[k] = 0u;
  __syncthreads();
#pragma unroll 1
  for (int it = 0; it < kMortonItems; it++)
  {
    const uint64_t at = ((uint64_t)blockIdx.x * kMortonItems + it) * kThreads + threadIdx.x;
    const bool in = at < N;
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, in);
    if (mask == 0u) break;
    uint32_t code = 0;
    if (in)
    {
      const uint32_t t = (uint32_t)at;
      const uint32_t s = find_segment(triOffsets, G, t);
      const uint32_t nT = triOffsets[s + 1] - triOffsets[s];
      const uint32_t vb = vertOffsets[s], nV = vertOffsets[s + 1] - vb;
      uint32_t ia = idx[3 * (size_t)t + 0], ib = idx[3 * (size_t)t + 1], ic = idx[3 * (size_t)t + 2];
      if (ia >= nV || ib >= nV || ic >= nV)
      {
        atomicOr(errorWord, kErrIndexRange);
        ia = ib = ic = 0;
      }
      code = bc::morton_code(v[vb + ia], v[vb + ib], v[vb + ic], nT, params[s].bmin, params[s].scale);
      keys[t] = code;
      unsorted[t] = code;
      vals[t] = t;
    }
    bc::count_digits(code, in, mask, s_hist);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 4 * 256; k += kThreads)
    if (s_hist[k]) atomicAdd(&hist[k], s_hist[k]);
}

__global__ void __launch_bounds__(kThreads) k_seg_compact(const uint32_t* __restrict__ keys, uint32_t n,
                                                          const uint32_t* __restrict__ triOffsets, uint32_t G,
                                                          uint32_t* __restrict__ compressed,
                                                          uint32_t* __restrict__ runStarts, uint32_t* tileStatus,
                                                          uint32_t* tileCounter, uint32_t* total, uint32_t* errorWord)
{
  bc::compact_runs_tile<kThreads>(keys, n, triOffsets, G, compressed, runStarts, tileStatus, tileCounter, total,
                                  errorWord);
}

// Leaf counts and the per-geometry offsets of runs, internal nodes, LR nodes
// and records (one block; a chunked block scan over the geometries).
// counts: [0] runs (input), [1] internal nodes, [2] LR nodes, [3] records.
__global__ void __launch_bounds__(1024) k_seg_offsets(const uint32_t* __restrict__ runStarts,
                                                      const uint32_t* __restrict__ triOffsets, uint32_t G,
                                                      uint32_t* counts, uint32_t* leafOffsets, uint32_t* intOffsets,
                                                      uint32_t* nodeOffsets, uint32_t* recOffsets, BuildParams* params)
{
  const uint32_t L = counts[0];
  // first run of each geometry: the first run start >= the geometry's first triangle
  for (uint32_t s = threadIdx.x; s <= G; s += blockDim.x)
  {
    if (s == G)
    {
      leafOffsets[G] = L;
      continue;
    }
    const uint32_t t0 = triOffsets[s];
    uint32_t lo = 0, hi = L;
    while (lo < hi)
    {
      const uint32_t mid = (lo + hi) >> 1;
      if (runStarts[mid] < t0) lo = mid + 1;
      else hi = mid;
    }
    leafOffsets[s] = lo;
  }
  __syncthreads();
  __shared__ uint32_t s_carry[3];
  __shared__ uint32_t s_part[3][1024];
  if (threadIdx.x < 3) s_carry[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t base = 0; base < G; base += blockDim.x)
  {
    const uint32_t s = base + threadIdx.x;
    uint32_t a = 0, b = 0, c = 0;
    if (s < G)
    {
      const uint32_t Ls = leafOffsets[s + 1] - leafOffsets[s];
      params[s].nLeaves = Ls;
      a = Ls > 1 ? Ls - 1 : 0;             // internal nodes
      b = Ls > 0 ? 2 * Ls - 1 : 0;         // LR nodes
      c = Ls > 1 ? Ls - 1 : (Ls ? 1 : 0);  // records
    }
    s_part[0][threadIdx.x] = a;
    s_part[1][threadIdx.x] = b;
    s_part[2][threadIdx.x] = c;
    __syncthreads();
    // inclusive Hillis-Steele scan of the three columns
    for (uint32_t o = 1; o < blockDim.x; o <<= 1)
    {
      uint32_t x0 = 0, x1 = 0, x2 = 0;
      if (threadIdx.x >= o)
      {
        x0 = s_part[0][threadIdx.x - o];
        x1 = s_part[1][threadIdx.x - o];
        x2 = s_part[2][threadIdx.x - o];
      }
      __syncthreads();
      s_part[0][threadIdx.x] += x0;
      s_part[1][threadIdx.x] += x1;
      s_part[2][threadIdx.x] += x2;
      __syncthreads();
    }
    if (s < G)
    {
      intOffsets[s] = s_carry[0] + s_part[0][threadIdx.x] - a;
      nodeOffsets[s] = s_carry[1] + s_part[1][threadIdx.x] - b;
      recOffsets[s] = s_carry[2] + s_part[2][threadIdx.x] - c;
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1)
    {
      s_carry[0] += s_part[0][threadIdx.x];
      s_carry[1] += s_part[1][threadIdx.x];
      s_carry[2] += s_part[2][threadIdx.x];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
  {
    intOffsets[G] = s_carry[0];
    nodeOffsets[G] = s_carry[1];
    recOffsets[G] = s_carry[2];
    counts[1] = s_carry[0];
    counts[2] = s_carry[1];
    counts[3] = s_carry[2];
  }
}

__global__ void __launch_bounds__(kThreads) k_seg_karras(const uint32_t* __restrict__ compressed,
                                                         const uint32_t* __restrict__ leafOffsets,
                                                         const uint32_t* __restrict__ intOffsets,
                                                         const uint32_t* __restrict__ nodeOffsets, uint32_t G,
                                                         const uint32_t* __restrict__ counts, BVHNode32* __restrict__ lr,
                                                         uint32_t* __restrict__ parent, uint32_t* __restrict__ visit,
                                                         uint32_t* __restrict__ rangeEnd)
{
  const uint32_t Itot = counts[1];
  // one node per thread; a warp's 32 consecutive internal nodes exchange
  // their codes for the direction test (lanes may belong to different
  // geometries), so the loop bound is uniform over the warp
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t base = blockIdx.x * kThreads + (threadIdx.x & ~31u); base < Itot; base += gridDim.x * kThreads)
  {
    const uint32_t j = base + lane;
    const bool active = j < Itot;
    const uint32_t s = active ? find_segment(intOffsets, G, j) : 0u;
    const int L = active ? (int)(leafOffsets[s + 1] - leafOffsets[s]) : 0;
    const int i = active ? (int)(j - intOffsets[s]) : 0;
    uint32_t ci;
    int dPrev, dNext;
    bc::karras_neighbours(compressed, active ? (int)leafOffsets[s] : 0, L, i, active, ci, dPrev, dNext);
    if (!active) continue;
    uint32_t left, right;
    int other;
    bc::karras_node(bc::GlobalCodes{compressed + leafOffsets[s]}, L, i, ci, dPrev, dNext, left, right, other);
    const uint32_t nb = nodeOffsets[s];
    lr[nb + i].leftOffset = left;
    lr[nb + i].escapeIndex = right;
    parent[nb + left] = (uint32_t)i;
    parent[nb + right] = (uint32_t)i;
    rangeEnd[j] = (uint32_t)other;
    visit[j] = 0u;
  }
}

// Child-pair records per internal node (as k_records in build.cu; references
// local to the geometry: internal child -> record index, leaf -> first
// triangle of the geometry's sorted order).
__global__ void __launch_bounds__(kThreads) k_seg_records(const uint32_t* __restrict__ triOffsets,
                                                          const uint32_t* __restrict__ leafOffsets,
                                                          const uint32_t* __restrict__ intOffsets,
                                                          const uint32_t* __restrict__ nodeOffsets,
                                                          const uint32_t* __restrict__ recOffsets, uint32_t G,
                                                          const uint32_t* __restrict__ counts,
                                                          const BVHNode32* __restrict__ lr,
                                                          const uint32_t* __restrict__ runStarts,
                                                          const uint32_t* __restrict__ visit, PairRec* __restrict__ recs,
                                                          uint32_t* errorWord)
{
  if (recs == nullptr)
  {
    // 4-wide layouts keep no pair records: only the check of each root
    for (uint32_t s = blockIdx.x * kThreads + threadIdx.x; s < G; s += gridDim.x * kThreads)
      if (intOffsets[s + 1] > intOffsets[s] && visit[intOffsets[s]] != 2u) atomicOr(errorWord, kErrLayout);
    return;
  }
  const uint32_t Itot = counts[1];
  for (uint32_t j = blockIdx.x * kThreads + threadIdx.x; j < Itot; j += gridDim.x * kThreads)
  {
    const uint32_t s = find_segment(intOffsets, G, j);
    const uint32_t L = leafOffsets[s + 1] - leafOffsets[s];
    const uint32_t i = j - intOffsets[s];
    if (i == 0 && visit[j] != 2u) atomicOr(errorWord, kErrLayout);  // the refit reached this root twice
    const uint32_t nb = nodeOffsets[s], tb = triOffsets[s], lb = leafOffsets[s];
    const uint32_t left = lr[nb + i].leftOffset, right = lr[nb + i].escapeIndex;
    const BVHNode32 a = bc::load_node(lr + nb + left);
    const BVHNode32 b = bc::load_node(lr + nb + right);
    const uint32_t lref = (left < L - 1) ? left : (kLeafBit | (runStarts[lb + left - (L - 1)] - tb));
    const uint32_t rref = (right < L - 1) ? right : (kLeafBit | (runStarts[lb + right - (L - 1)] - tb));
    PairRec r;
    r.a = make_float4(a.boxMin[0], a.boxMin[1], a.boxMin[2], a.boxMax[0]);
    r.b = make_float4(a.boxMax[1], a.boxMax[2], b.boxMin[0], b.boxMin[1]);
    r.c = make_float4(b.boxMin[2], b.boxMax[0], b.boxMax[1], b.boxMax[2]);
    r.d = make_uint4(lref, rref, 0u, 0u);
    recs[recOffsets[s] + i] = r;
  }
}

// Last stage: run starts and triangle ids become local to their geometry, so
// every geometry's arrays read exactly like a single build's.
__global__ void __launch_bounds__(kThreads) k_seg_localize(const uint32_t* __restrict__ triOffsets,
                                                           const uint32_t* __restrict__ leafOffsets, uint32_t G,
                                                           uint32_t N, const uint32_t* __restrict__ counts,
                                                           uint32_t* __restrict__ runStarts, uint32_t* __restrict__ vals)
{
  const uint32_t Ltot = counts[0];
  for (uint32_t t = blockIdx.x * kThreads + threadIdx.x; t < N; t += gridDim.x * kThreads)
  {
    vals[t] -= triOffsets[find_segment(triOffsets, G, t)];
    if (t < Ltot) runStarts[t] -= triOffsets[find_segment(leafOffsets, G, t)];
  }
}

inline uint32_t grid_for(uint64_t n, int numSMs, int perSM = 8)
{
  uint64_t g = (n + kThreads - 1) / kThreads;
  const uint64_t cap = (uint64_t)numSMs * perSM;
  if (g > cap) g = cap;
  return g == 0 ? 1u : (uint32_t)g;
}

inline size_t align256(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

size_t build_batch_scratch_bytes(uint32_t nTris, uint32_t G)
{
  const size_t tiles = (nTris + kThreads * bc::kScanItems - 1) / (kThreads * bc::kScanItems);
  return align256(sizeof(uint32_t) * (4 + tiles)) + align256(radix_sort_segmented_scratch_bytes(nTris, G));
}

cudaError_t build_lbvh_batch(const BatchBuffers& b, int numSMs, cudaStream_t s)
{
  const uint32_t N = b.nTris, G = b.G;
  if (N == 0 || G == 0) return cudaSuccess;
  char* scratch = (char*)b.scratch;
  const size_t tiles = (N + kThreads * bc::kScanItems - 1) / (kThreads * bc::kScanItems);
  const size_t scanBytes = align256(sizeof(uint32_t) * (4 + tiles));
  uint32_t* scanCounter = (uint32_t*)scratch;
  uint32_t* scanStatus = scanCounter + 4;
  void* sortScratch = scratch + scanBytes;

  if (b.nBoxChunks + b.nIdxChunks) k_seg_read_inputs<<<b.nBoxChunks + b.nIdxChunks, kThreads, 0, s>>>(b);
  k_seg_box_final<<<(G + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, s>>>(b.boxChunkOffsets, G, b.boxPartial,
                                                                                  b.params, b.mortonCubic);
  // an odd number of sort passes starts from the spare arrays and ends in keys and vals
  const bool swap = radix_sort_segmented_passes(G) & 1;
  uint32_t *keys0 = swap ? b.keysAlt : b.keys, *vals0 = swap ? b.valsAlt : b.vals;
  constexpr uint32_t kPerBlock = kThreads * kMortonItems;
  cudaError_t e = cudaMemsetAsync(b.scratch, 0, build_batch_scratch_bytes(N, G), s);
  if (e != cudaSuccess) return e;
  k_seg_morton<<<(N + kPerBlock - 1) / kPerBlock, kThreads, 0, s>>>(b.verts, b.idx, b.vertOffsets, b.triOffsets, G, N,
                                                                     b.params, keys0, vals0, b.keysUnsorted,
                                                                     (uint32_t*)sortScratch, b.errorWord);
  e = radix_sort_pairs_segmented(keys0, vals0, swap ? b.keys : b.keysAlt, swap ? b.vals : b.valsAlt, N, b.triOffsets, G,
                                 sortScratch, b.errorWord, s);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(b.counts, 0, 4 * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  k_seg_compact<<<(uint32_t)tiles, kThreads, 0, s>>>(b.keys, N, b.triOffsets, G, b.compressed, b.runStarts, scanStatus,
                                                    scanCounter, b.counts, b.errorWord);
  k_seg_offsets<<<1, 1024, 0, s>>>(b.runStarts, b.triOffsets, G, b.counts, b.leafOffsets, b.intOffsets, b.nodeOffsets,
                                   b.recOffsets, b.params);
  const uint32_t g = grid_for(N, numSMs, 8);
  k_seg_karras<<<g, kThreads, 0, s>>>(b.compressed, b.leafOffsets, b.intOffsets, b.nodeOffsets, G, b.counts, b.lr,
                                      b.parent, b.visit, b.visit + N);
  bc::LeafTree t = {};
  t.verts = b.verts;
  t.idx = b.idx;
  t.sortedTri = b.vals;
  t.runStarts = b.runStarts;
  t.nTris = N;
  t.lr = b.lr;
  t.lrCount = b.lrCount;
  t.tris = b.tris;
  t.sortedIdx = b.sortedIdx;
  t.parent = b.parent;
  t.visit = b.visit;
  t.rangeEnd = b.visit + N;
  t.lists = b.keysAlt;  // free after the sort
  t.errorWord = b.errorWord;
  t.vertexRecords = b.vertexRecords;
  t.vertOffsets = b.vertOffsets;
  t.triOffsets = b.triOffsets;
  t.leafOffsets = b.leafOffsets;
  t.intOffsets = b.intOffsets;
  t.nodeOffsets = b.nodeOffsets;
  t.recOffsets = b.recOffsets;
  t.counts = b.counts;
  t.G = G;
  t.recs = b.recs;
  e = bc::leaf_tree<true>(t, s);
  if (e != cudaSuccess) return e;
  k_seg_records<<<g, kThreads, 0, s>>>(b.triOffsets, b.leafOffsets, b.intOffsets, b.nodeOffsets, b.recOffsets, G,
                                       b.counts, b.lr, b.runStarts, b.visit, b.recs, b.errorWord);
  k_seg_localize<<<g, kThreads, 0, s>>>(b.triOffsets, b.leafOffsets, G, N, b.counts, b.runStarts, b.vals);
  return cudaGetLastError();
}

}  // namespace hrt
