// Collapse of the LBVH (binary Karras tree) into 4-wide nodes, stored as FP32
// boxes, FP16 boxes rounded outward, or 8-bit offsets against a per-node FP32
// frame with power-of-two scales (also rounded outward).
//
// Collapse rule (HeavyRT's BVH2ToBVH4, core/builders/cbvh.cpp:226-311): a
// 4-wide node replaces a binary node and its two children; its slots are the
// grandchildren (or the child itself when that child is a leaf).  A binary
// node that would become a 4-wide node while both its children are leaves is
// instead merged into one leaf covering both runs (their sorted ranges are
// adjacent).  The root always stays a node.  With this rule the 4-wide nodes
// are exactly the binary internal nodes at even depth that are not merged.
//
// Largest-first rule (a build option): a 4-wide node starts from its binary
// node's two children and twice opens the internal slot with the most leaves
// under it (the leftmost of equals) into that slot's two children, in place.
// The slots' shapes alone decide, so a refit (same topology) keeps the tree.
// Which binary nodes become 4-wide nodes then depends on the choices above
// them: the roles are found top down, by one block until some hundred 4-wide
// nodes are in hand and then by a block for each of their subtrees (the roles
// do not depend on the order; the numbering is the same Karras-order scan as
// with the even-depth rule).
//
// Quantised boxes only ever contain the FP32 box they stand for, so a
// traversal of the quantised tree visits every node the FP32 tree would and
// can only add visits; the triangle test is unchanged.
#include <algorithm>

#include <cuda_fp16.h>

#include "build_common.cuh"
#include "hrt_kernels.cuh"

namespace hrt
{
namespace
{

constexpr int kThreads = 256;

// Depth of internal node i of one tree: walk up the parent chain (depth <= 30).
__device__ __forceinline__ uint8_t node_depth(const uint32_t* __restrict__ parent, uint32_t L, uint32_t i)
{
  uint32_t d = 0, n = i;
  while (n != 0 && d < 255)
  {
    const uint32_t p = parent[n];
    if (p + 1u >= L) break;  // only the root lacks an internal parent
    n = p;
    d++;
  }
  return (uint8_t)d;
}

__global__ void __launch_bounds__(kThreads) k_depth(BuildParams* __restrict__ params,
                                                    const uint32_t* __restrict__ parent,
                                                    const uint32_t* __restrict__ visit, uint8_t* __restrict__ depth)
{
  const uint32_t L = params->nLeaves;
  if (blockIdx.x == 0 && threadIdx.x == 0 && L >= 2u && visit[0] != 2u) atomicOr(&params->error, kErrLayout);
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i + 1 < L; i += gridDim.x * kThreads)
    depth[i] = node_depth(parent, L, i);
}

// First sorted triangle and one-past-last of the triangles under binary node s.
__device__ __forceinline__ void node_range(const BVHNode32* __restrict__ lr, const uint32_t* __restrict__ runStarts,
                                           uint32_t L, uint32_t nTris, uint32_t s, uint32_t& start, uint32_t& end)
{
  // leftmost / rightmost leaf under s: follow left (right) children down
  uint32_t a = s, b = s;
  while (a + 1u < L) a = lr[a].leftOffset;
  while (b + 1u < L) b = lr[b].escapeIndex;
  const uint32_t la = a - (L - 1), lb = b - (L - 1);
  start = runStarts[la];
  end = (lb + 1 < L) ? runStarts[lb + 1] : nTris;
}

// Whether internal node i, due to become a 4-wide node, becomes one leaf instead.
// mergeMode 0: merge when both children are leaves (the reference's rule);
// mergeMode M > 0: merge when the subtree holds at most M triangles.
__device__ __forceinline__ bool merges(const BVHNode32* __restrict__ lr, const uint32_t* __restrict__ runStarts,
                                       uint32_t L, uint32_t nTris, int mergeMode, uint32_t i)
{
  if (i == 0) return false;  // the root stays a node
  if (mergeMode == 0) return lr[i].leftOffset + 1u >= L && lr[i].escapeIndex + 1u >= L;
  if (mergeMode == 1) return false;  // an internal node holds two leaves at least, so two triangles
  uint32_t st, en;
  node_range(lr, runStarts, L, nTris, i, st, en);
  return en - st <= (uint32_t)mergeMode;
}

// Role of internal node i under the even-depth rule: 1 = 4-wide node, 2 =
// merged leaf, 0 = absorbed.
__device__ __forceinline__ uint8_t node_role(const BVHNode32* __restrict__ lr, const uint32_t* __restrict__ runStarts,
                                             uint32_t L, uint32_t nTris, uint8_t depth, int mergeMode, uint32_t i)
{
  if ((depth & 1u) != 0u) return 0;
  return merges(lr, runStarts, L, nTris, mergeMode, i) ? 2 : 1;
}

constexpr int kCollapseLargestFirst = 1;  // HRT_BVH4_COLLAPSE_LARGEST_FIRST

// The binary nodes that become the slots of the 4-wide node of internal node
// i (L >= 2), left to right; returns their count (2..4).  Even depth: each
// child's two children, or the child itself when it is a leaf.  Largest
// first: the two children, then twice the internal slot with the largest
// descendant count (most leaves; the leftmost of equals) replaced in place by
// its two children.
__device__ __forceinline__ int collapse_slots(const BVHNode32* __restrict__ lr, const uint32_t* __restrict__ lrCount,
                                              uint32_t L, int collapse, uint32_t i, uint32_t (&cand)[4])
{
  const uint32_t k0 = lr[i].leftOffset, k1 = lr[i].escapeIndex;
  if (collapse != kCollapseLargestFirst)
  {
    const bool in0 = k0 + 1u < L, in1 = k1 + 1u < L;
    const uint32_t a0 = in0 ? lr[k0].leftOffset : k0, b0 = in0 ? lr[k0].escapeIndex : 0u;
    const uint32_t a1 = in1 ? lr[k1].leftOffset : k1, b1 = in1 ? lr[k1].escapeIndex : 0u;
    cand[0] = a0;
    cand[1] = in0 ? b0 : a1;
    cand[2] = in0 ? a1 : b1;
    cand[3] = b1;
    return (in0 ? 2 : 1) + (in1 ? 2 : 1);
  }
  // Links and counts are read a round ahead of the choices that need them:
  // the children's, then those of the two nodes that the first opening brings.
  // Three dependent rounds instead of six (a leaf's count reads 0 and it is
  // never opened).
  struct Link
  {
    uint32_t id, left, right, count;  // count 0: a leaf
  };
  auto link = [&](uint32_t id) {
    Link q{id, 0u, 0u, 0u};
    if (id + 1u < L)
    {
      q.left = lr[id].leftOffset;
      q.right = lr[id].escapeIndex;
      q.count = lrCount[id];
    }
    return q;
  };
  const Link a = link(k0), b = link(k1);
  cand[0] = k0;
  cand[1] = k1;
  cand[2] = cand[3] = 0u;
  if (a.count == 0u && b.count == 0u) return 2;
  const bool open0 = a.count >= b.count;  // the leftmost of equals; a leaf's 0 is less than any node's 2
  const Link x = link(open0 ? a.left : b.left), y = link(open0 ? a.right : b.right);
  // slots now: x, y, b or a, x, y
  const Link s0 = open0 ? x : a, s1 = open0 ? y : x, s2 = open0 ? b : y;
  cand[0] = s0.id;
  cand[1] = s1.id;
  cand[2] = s2.id;
  const uint32_t most = max(s0.count, max(s1.count, s2.count));
  if (most == 0u) return 3;
  if (s0.count == most)
  {
    cand[0] = s0.left;
    cand[1] = s0.right;
    cand[2] = s1.id;
    cand[3] = s2.id;
  }
  else if (s1.count == most)
  {
    cand[1] = s1.left;
    cand[2] = s1.right;
    cand[3] = s2.id;
  }
  else
  {
    cand[2] = s2.left;
    cand[3] = s2.right;
  }
  return 4;
}

// One geometry's tree, or one of a batch's (segment seg): internal node i of
// it is node intBase + i of the role array.
struct SegTree
{
  const BVHNode32* lr;
  const uint32_t*  lrCount;
  const uint32_t*  runStarts;
  const uint32_t*  parent;
  TriRec*          tris;
  uint32_t         L, nTris, intBase, seg;
};

__device__ __forceinline__ SegTree seg_tree(const Bvh4Batch& b, uint32_t seg)
{
  SegTree t;
  t.seg = seg;
  t.lr = b.lr + b.nodeOffsets[seg];
  t.lrCount = b.lrCount + b.nodeOffsets[seg];
  t.parent = b.parent + b.nodeOffsets[seg];
  t.runStarts = b.runStarts + b.leafOffsets[seg];
  t.tris = b.tris + b.triOffsets[seg];
  t.L = b.leafOffsets[seg + 1] - b.leafOffsets[seg];
  t.nTris = b.triOffsets[seg + 1] - b.triOffsets[seg];
  t.intBase = b.intOffsets[seg];
  return t;
}

// What the role kernels walk: one tree (params) or a batch's trees.
struct RoleTrees
{
  const BuildParams* params;  // one tree: its leaf count; null for a batch
  SegTree            one;     // one tree (L from params)
  Bvh4Batch          batch;
  const uint32_t*    visit;  // one tree: arrivals at its root in the box refit
  uint32_t           nInt;  // a batch's internal nodes
  int                mergeMode;
};

__device__ __forceinline__ SegTree tree_of(const RoleTrees& r, uint32_t j)
{
  if (r.params != nullptr)
  {
    SegTree t = r.one;
    t.L = r.params->nLeaves;
    return t;
  }
  return seg_tree(r.batch, bc::find_segment(r.batch.intOffsets, r.batch.G, j));
}

// The internal slots of the largest-first 4-wide node of internal node i of
// `t`: marked as 4-wide nodes (returned, as role-array indices) or merged
// leaves.  Returns their count.
__device__ __forceinline__ int mark_slots(const SegTree& t, int mergeMode, uint32_t i, uint8_t* __restrict__ role,
                                          uint32_t (&next)[4])
{
  uint32_t cand[4];
  const int nc = collapse_slots(t.lr, t.lrCount, t.L, kCollapseLargestFirst, i, cand);
  int cnt = 0;
#pragma unroll
  for (int k = 0; k < 4; k++)
  {
    if (k >= nc) break;
    const uint32_t c = cand[k];
    if (c + 1u >= t.L) continue;  // a leaf slot
    const bool m = merges(t.lr, t.runStarts, t.L, t.nTris, mergeMode, c);
    role[t.intBase + c] = m ? 2 : 1;
    if (!m)
    {
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q == cnt) next[q] = t.intBase + c;
      cnt++;
    }
  }
  return cnt;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v)
{
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= (uint32_t)o) v += y;
  }
  return v;
}

// A tree of distinct 30-bit codes is at most 31 binary levels deep, and a
// 4-wide level descends at least one.
constexpr int kCollapseLevels = 34;

// The top of the largest-first roles, one block: level after level from the
// roots until the level holds kTopFrontier 4-wide nodes or none.  The last
// level is left in front[0 or 1]; state = {its size, which}.  role is zeroed
// beforehand.  A level is a few dependent loads; one SM's loads bound larger ones.
constexpr uint32_t kTopThreads = 1024, kTopFrontier = 512;

__global__ void __launch_bounds__(kTopThreads)
    k_roles_top(RoleTrees r, uint32_t* __restrict__ front0, uint32_t* __restrict__ front1, uint32_t* state,
                uint8_t* __restrict__ role, uint32_t* errorWord)
{
  __shared__ uint32_t s_count[kCollapseLevels + 2];
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  for (uint32_t k = tid; k < kCollapseLevels + 2; k += kTopThreads) s_count[k] = 0u;
  __syncthreads();
  uint32_t cap;
  if (r.params != nullptr)
  {
    const uint32_t L = r.params->nLeaves;
    cap = L > 0 ? L - 1 : 0u;
    if (tid == 0 && L >= 2)
    {
      if (r.visit[0] != 2u) atomicOr(errorWord, kErrLayout);
      role[0] = 1;
      front0[0] = 0u;
      s_count[0] = 1u;
    }
  }
  else
  {
    cap = r.nInt;
    for (uint32_t seg = tid; seg < r.batch.G; seg += kTopThreads)
      if (r.batch.leafOffsets[seg + 1] - r.batch.leafOffsets[seg] >= 2u)
      {
        const uint32_t j = r.batch.intOffsets[seg], at = atomicAdd(&s_count[0], 1u);
        role[j] = 1;
        if (at < cap) front0[at] = j;
      }
  }
  __syncthreads();
  int lvl = 0;
  uint32_t n = min(s_count[0], cap);
  while (n > 0 && n < kTopFrontier && lvl < kCollapseLevels)
  {
    const uint32_t* in = (lvl & 1) ? front1 : front0;
    uint32_t* out = (lvl & 1) ? front0 : front1;
    for (uint32_t b0 = tid & ~31u; b0 < n; b0 += kTopThreads)
    {
      const uint32_t f = b0 + lane;
      uint32_t next[4] = {0u, 0u, 0u, 0u};
      int cnt = 0;
      if (f < n)
      {
        const uint32_t j = in[f];
        const SegTree t = tree_of(r, j);
        cnt = mark_slots(t, r.mergeMode, j - t.intBase, role, next);
      }
      const uint32_t incl = warp_inclusive((uint32_t)cnt);
      uint32_t base = 0;
      if (lane == 31 && incl) base = atomicAdd(&s_count[lvl + 1], incl);
      base = __shfl_sync(0xFFFFFFFFu, base, 31) + incl - (uint32_t)cnt;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k < cnt && base + k < cap) out[base + k] = next[k];
    }
    __syncthreads();  // the level's list (global, this block's own) and count are complete
    lvl++;
    n = s_count[lvl];
    if (n > cap)  // more nodes than the tree has: the links are inconsistent
    {
      if (tid == 0) atomicOr(errorWord, kErrLayout);
      n = cap;
    }
  }
  if (tid == 0)
  {
    state[0] = n;
    state[1] = (uint32_t)(lvl & 1);
  }
}

// The subtrees below the top's last level, a block each: nodes wait on a stack
// in shared memory, up to a block's threads are taken at a time.  Near the
// stack's end fewer are taken, down to one: then it grows by at most three a
// level, for which kSubReserve entries are kept.  (2M-triangle heightfield,
// 555,081 4-wide nodes: one launch per level with a list in global memory took
// 34 launches and 106 us of kernels; a top up to 4,096 nodes and a warp per
// subtree 52 + 33 us, up to 512 nodes 16 + 83; a top up to 512 and a block per subtree 14 + 28 us.)
constexpr int kSubThreads = 256, kSubStack = 4096, kSubReserve = 3 * kCollapseLevels + 8;

__global__ void __launch_bounds__(kSubThreads)
    k_roles_sub(RoleTrees r, const uint32_t* __restrict__ front0, const uint32_t* __restrict__ front1,
                const uint32_t* __restrict__ state, uint8_t* __restrict__ role, uint32_t* errorWord)
{
  __shared__ uint32_t s_stack[kSubStack];
  __shared__ uint32_t s_size;
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  const uint32_t n = state[0];
  const uint32_t* front = state[1] ? front1 : front0;
  for (uint32_t f = blockIdx.x; f < n; f += gridDim.x)
  {
    const uint32_t root = front[f];
    const SegTree t = tree_of(r, root);
    uint32_t size = 1, budget = t.L;  // a consistent subtree has fewer nodes
    if (tid == 0) s_stack[0] = root;
    __syncthreads();
    while (size > 0)
    {
      const int room = ((int)kSubStack - kSubReserve - (int)size) / 3;
      const uint32_t take = min(size, (uint32_t)min(max(room, 1), kSubThreads));
      if (budget < take)
      {
        if (tid == 0) atomicOr(errorWord, kErrLayout);
        break;
      }
      budget -= take;
      const bool in = tid < take;
      const uint32_t j = in ? s_stack[size - 1 - tid] : 0u;
      size -= take;
      if (tid == 0) s_size = size;
      uint32_t next[4] = {0u, 0u, 0u, 0u};
      const int cnt = in ? mark_slots(t, r.mergeMode, j - t.intBase, role, next) : 0;
      const uint32_t incl = warp_inclusive((uint32_t)cnt);
      __syncthreads();  // the taken entries are read, s_size is set
      uint32_t base = 0;
      if (lane == 31 && incl) base = atomicAdd(&s_size, incl);
      base = __shfl_sync(0xFFFFFFFFu, base, 31) + incl - (uint32_t)cnt;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k < cnt && base + k < (uint32_t)kSubStack) s_stack[base + k] = next[k];
      __syncthreads();
      size = s_size;
      if (size > (uint32_t)kSubStack)  // deeper than the depth bound
      {
        if (tid == 0) atomicOr(errorWord, kErrLayout);
        break;
      }
      __syncthreads();  // s_size is read
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kThreads) k_roles(const BuildParams* __restrict__ params,
                                                    const BVHNode32* __restrict__ lr,
                                                    const uint32_t* __restrict__ runStarts, uint32_t nTris,
                                                    const uint8_t* __restrict__ depth, int mergeMode,
                                                    uint8_t* __restrict__ role)
{
  const uint32_t L = params->nLeaves;
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i + 1 < L; i += gridDim.x * kThreads)
    role[i] = node_role(lr, runStarts, L, nTris, depth[i], mergeMode, i);
}

// Exclusive scan of (role == 1) over the internal nodes: the 4-wide node index
// of each binary node that becomes one, in Karras order (the root gets 0); the
// prefix is written at every position.  n = L - 1 of params, or nGiven when
// params is null (the internal nodes of a whole batch, geometry after
// geometry).  The 4-wide nodes' positions also go to `list`, in order: the
// emission takes one per lane instead of asking every internal node.  One block per 4096 nodes, decoupled look-back as in the run
// compaction.
constexpr int      kScanItems  = 16;
constexpr uint32_t kScanTile   = kThreads * kScanItems;

__global__ void __launch_bounds__(kThreads) k_scan_roles(const BuildParams* __restrict__ params, uint32_t nGiven,
                                                         const uint8_t* __restrict__ role, uint32_t* __restrict__ index,
                                                         uint32_t* __restrict__ list, uint32_t* tileStatus, uint32_t* tileCounter, uint32_t* total,
                                                         uint32_t* errorWord)
{
  __shared__ uint32_t s_tile, s_prefix;
  __shared__ uint32_t s_warp[kThreads / 32 + 1];
  const uint32_t L = params ? params->nLeaves : 0u;
  const uint32_t n = params ? (L > 1 ? L - 1 : 0) : nGiven;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(tileCounter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tile >= tiles) return;  // the grid is sized for the worst case
  const uint32_t base = tile * kScanTile + tid * kScanItems;
  // a thread's 16 roles are one 128-bit load (the array starts at a 256-byte boundary)
  uint32_t flags = 0;
  if (base + kScanItems <= n)
  {
    const uint4 v = *reinterpret_cast<const uint4*>(role + base);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < kScanItems; k++) flags |= (((w[k >> 2] >> (8 * (k & 3))) & 0xFFu) == 1u ? 1u : 0u) << k;
  }
  else
  {
#pragma unroll
    for (int k = 0; k < kScanItems; k++) flags |= (base + k < n && role[base + k] == 1 ? 1u : 0u) << k;
  }
  const uint32_t cnt = __popc(flags);
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
    constexpr int kWarps = kThreads / 32;
    const uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
    uint32_t run = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, run, o);
      if (lane >= o) run += y;
    }
    const uint32_t sum = __shfl_sync(0xFFFFFFFFu, run, 31);
    if (lane < kWarps) s_warp[lane] = run - w;
    const uint32_t excl = bc::warp_look_back(tileStatus, tile, sum, errorWord);
    if (lane == 0)
    {
      s_prefix = excl;
      if (tile == tiles - 1) *total = excl + sum;
    }
  }
  __syncthreads();
  uint32_t pos = s_prefix + s_warp[warp] + incl - cnt;
  if (base + kScanItems <= n)
  {
    uint4* o = reinterpret_cast<uint4*>(index + base);
#pragma unroll
    for (int q = 0; q < kScanItems / 4; q++)
    {
      uint32_t v[4];
#pragma unroll
      for (int k = 0; k < 4; k++)
      {
        v[k] = pos;
        if ((flags >> (4 * q + k)) & 1u)
        {
          if (pos < n) list[pos] = base + 4 * q + k;
          pos++;
        }
      }
      o[q] = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
  else
  {
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
      if (base + k < n)
      {
        index[base + k] = pos;
        if ((flags >> k) & 1u)
        {
          if (pos < n) list[pos] = base + k;
          pos++;
        }
      }
  }
}

struct Slot
{
  float    lo[3], hi[3];
  uint32_t ref;  // node index, kLeafBit | first triangle, or kEmptyRef
};

__device__ __forceinline__ uint32_t h2_bits(__half lo, __half hi)
{
  return (uint32_t)__half_as_ushort(lo) | ((uint32_t)__half_as_ushort(hi) << 16);
}

// Smallest power-of-two exponent e with 255 * 2^e >= ext (e in [-126, 127]).
__device__ __forceinline__ int q8_exponent(float ext)
{
  if (!(ext > 0.0f)) return -126;
  int e;
  frexpf(ext / 255.0f, &e);  // ext/255 = m * 2^e, m in [0.5, 1)
  if (e < -126) e = -126;
  if (e > 127) e = 127;
  return e;
}

__device__ __forceinline__ float q8_scale(int e) { return __int_as_float((e + 127) << 23); }

// decoded bound = origin + q * 2^e (one product, exact for q < 256; one rounded add)
__device__ __forceinline__ float q8_decode(float origin, uint32_t q, float scale)
{
  return __fadd_rn(origin, __fmul_rn((float)q, scale));
}

__device__ __forceinline__ uint32_t q8_lo(float origin, float v, float scale)
{
  float qf = floorf(__fdiv_rn(__fsub_rn(v, origin), scale));
  int q = (int)fmaxf(0.0f, fminf(255.0f, qf));
  while (q > 0 && q8_decode(origin, (uint32_t)q, scale) > v) q--;
  return (uint32_t)q;
}

__device__ __forceinline__ uint32_t q8_hi(float origin, float v, float scale, bool& ok)
{
  float qf = ceilf(__fdiv_rn(__fsub_rn(v, origin), scale));
  int q = (int)fmaxf(0.0f, fminf(255.0f, qf));
  while (q < 255 && q8_decode(origin, (uint32_t)q, scale) < v) q++;
  ok = q8_decode(origin, (uint32_t)q, scale) >= v;
  return (uint32_t)q;
}

// One 4-wide node written in `format` (0 FP32, 1 FP16 rounded outward, 2
// 8-bit in a per-node frame) from its ns used slots.
__device__ __forceinline__ void write_node4(int format, void* __restrict__ nodes, uint32_t outIdx, Slot (&slot)[4],
                                            int ns, uint32_t* errorWord)
{
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k >= ns)
    {
      for (int c = 0; c < 3; c++) { slot[k].lo[c] = 0.0f; slot[k].hi[c] = 0.0f; }
      slot[k].ref = kEmptyRef;
    }
  if (format == 0)
  {
    Node4F32 o;
    o.lox = make_float4(slot[0].lo[0], slot[1].lo[0], slot[2].lo[0], slot[3].lo[0]);
    o.loy = make_float4(slot[0].lo[1], slot[1].lo[1], slot[2].lo[1], slot[3].lo[1]);
    o.loz = make_float4(slot[0].lo[2], slot[1].lo[2], slot[2].lo[2], slot[3].lo[2]);
    o.hix = make_float4(slot[0].hi[0], slot[1].hi[0], slot[2].hi[0], slot[3].hi[0]);
    o.hiy = make_float4(slot[0].hi[1], slot[1].hi[1], slot[2].hi[1], slot[3].hi[1]);
    o.hiz = make_float4(slot[0].hi[2], slot[1].hi[2], slot[2].hi[2], slot[3].hi[2]);
    o.ref = make_uint4(slot[0].ref, slot[1].ref, slot[2].ref, slot[3].ref);
    o.pad = make_uint4(0, 0, 0, 0);
    reinterpret_cast<Node4F32*>(nodes)[outIdx] = o;
  }
  else if (format == 1)
  {
    uint32_t w[12];
    for (int k = 0; k < 4; k++)
    {
      w[0 + k] = h2_bits(__float2half_rd(slot[k].lo[0]), __float2half_rd(slot[k].lo[1]));
      w[4 + k] = h2_bits(__float2half_rd(slot[k].lo[2]), __float2half_ru(slot[k].hi[0]));
      w[8 + k] = h2_bits(__float2half_ru(slot[k].hi[1]), __float2half_ru(slot[k].hi[2]));
    }
    Node4F16 o;
    o.a = make_uint4(w[0], w[1], w[2], w[3]);
    o.b = make_uint4(w[4], w[5], w[6], w[7]);
    o.c = make_uint4(w[8], w[9], w[10], w[11]);
    o.ref = make_uint4(slot[0].ref, slot[1].ref, slot[2].ref, slot[3].ref);
    reinterpret_cast<Node4F16*>(nodes)[outIdx] = o;
  }
  else
  {
    // frame: the union of the slots' boxes; per-axis power-of-two scale
    float org[3], scale[3];
    int ex[3];
    for (int c = 0; c < 3; c++)
    {
      float mn = slot[0].lo[c], mx = slot[0].hi[c];
      for (int k = 1; k < ns; k++)
      {
        mn = fminf(mn, slot[k].lo[c]);
        mx = fmaxf(mx, slot[k].hi[c]);
      }
      org[c] = mn;
      ex[c] = q8_exponent(__fsub_rn(mx, mn));
      // widen the scale until the frame's top is representable outward
      for (int guard = 0; guard < 4; guard++)
      {
        if (q8_decode(org[c], 255u, q8_scale(ex[c])) >= mx || ex[c] >= 127) break;
        ex[c]++;
      }
      scale[c] = q8_scale(ex[c]);
    }
    uint32_t qb[6] = {0, 0, 0, 0, 0, 0};  // lox, loy, loz, hix, hiy, hiz: 4 bytes each (one per slot)
    for (int k = 0; k < ns; k++)
      for (int c = 0; c < 3; c++)
      {
        bool ok = true;
        const uint32_t lo = q8_lo(org[c], slot[k].lo[c], scale[c]);
        const uint32_t hi = q8_hi(org[c], slot[k].hi[c], scale[c], ok);
        if (!ok) atomicOr(errorWord, kErrLayout);
        qb[c] |= lo << (8 * k);
        qb[3 + c] |= hi << (8 * k);
      }
    Node4Q8 o;
    o.frame = make_float4(org[0], org[1], org[2],
                          __uint_as_float((uint32_t)(ex[0] + 128) | ((uint32_t)(ex[1] + 128) << 8) |
                                          ((uint32_t)(ex[2] + 128) << 16)));
    o.q0 = make_uint4(qb[0], qb[1], qb[2], qb[3]);
    o.q1 = make_uint4(qb[4], qb[5], 0u, 0u);
    o.ref = make_uint4(slot[0].ref, slot[1].ref, slot[2].ref, slot[3].ref);
    reinterpret_cast<Node4Q8*>(nodes)[outIdx] = o;
  }
}

// The slots of the 4-wide node that binary node i (role 1) of one tree becomes:
// its grandchildren, or a child itself when that child is a leaf.  A slot is a
// leaf (kLeafBit | first triangle), a merged leaf (role 2: its runs joined, the
// 4-wide end flag cleared at the ends of the runs before the last), or the
// 4-wide node indexOf(child) of another role-1 node.  With one leaf (L == 1)
// the node holds that leaf alone.  Returns the number of used slots.
template <typename IndexOf>
__device__ __forceinline__ int node4_slots(const BVHNode32* __restrict__ lr, const uint32_t* __restrict__ lrCount,
                                           const uint32_t* __restrict__ runStarts, uint32_t L, uint32_t nTris,
                                           int collapse, const uint8_t* __restrict__ role, IndexOf indexOf, uint32_t i,
                                           TriRec* __restrict__ tris, Slot (&slot)[4])
{
  if (L == 1u)
  {
    const BVHNode32 n = lr[0];
    for (int c = 0; c < 3; c++) { slot[0].lo[c] = n.boxMin[c]; slot[0].hi[c] = n.boxMax[c]; }
    slot[0].ref = kLeafBit | runStarts[0];
    return 1;
  }
  uint32_t cand[4];
  const int nc = collapse_slots(lr, lrCount, L, collapse, i, cand);
#pragma unroll
  for (int k = 0; k < 4; k++)
  {
    if (k >= nc) break;
    const uint32_t s = cand[k];
    const BVHNode32 n = bc::load_node(lr + s);
    for (int c = 0; c < 3; c++) { slot[k].lo[c] = n.boxMin[c]; slot[k].hi[c] = n.boxMax[c]; }
    if (s + 1u >= L)
      slot[k].ref = kLeafBit | runStarts[s - (L - 1)];
    else if (role[s] == 2)
    {
      uint32_t st, en;
      node_range(lr, runStarts, L, nTris, s, st, en);
      slot[k].ref = kLeafBit | st;
      uint32_t a = s, b = s;
      while (a + 1u < L) a = lr[a].leftOffset;
      while (b + 1u < L) b = lr[b].escapeIndex;
      for (uint32_t leaf = a - (L - 1); leaf < b - (L - 1); leaf++)
      {
        const uint32_t runEnd = runStarts[leaf + 1];
        if (runEnd > st && runEnd < en)
        {
          const uint32_t w = __float_as_uint(tris[runEnd - 1].a.w);
          tris[runEnd - 1].a.w = __uint_as_float(w & ~2u);
        }
      }
    }
    else
      slot[k].ref = indexOf(s);
  }
  return nc;
}

__global__ void __launch_bounds__(kThreads) k_emit4(const BuildParams* __restrict__ params,
                                                    const BVHNode32* __restrict__ lr,
                                                    const uint32_t* __restrict__ lrCount,
                                                    const uint32_t* __restrict__ runStarts, uint32_t nTris,
                                                    int collapse, const uint8_t* __restrict__ role,
                                                    const uint32_t* __restrict__ index,
                                                    const uint32_t* __restrict__ list, int format,
                                                    void* __restrict__ nodes, uint32_t maxNodes,
                                                    TriRec* __restrict__ tris, uint32_t* errorWord)
{
  const uint32_t L = params->nLeaves;
  for (uint32_t o = blockIdx.x * kThreads + threadIdx.x; o < maxNodes; o += gridDim.x * kThreads)
  {
    const uint32_t i = L == 1u ? 0u : list[o];
    if (L != 1u && (i + 1u >= L || role[i] != 1))  // only after a failed numbering (reported through the error word)
    {
      atomicOr(errorWord, kErrLayout);
      continue;
    }
    Slot slot[4];
    const int ns = node4_slots(lr, lrCount, runStarts, L, nTris, collapse, role, [&](uint32_t c) { return index[c]; },
                               i, tris, slot);
    write_node4(format, nodes, o, slot, ns, errorWord);
  }
}

// ---------------------------------------------------------------- batches
// The same collapse for the geometries of a segmented build at once: internal
// node j of the batch is node j - intOffsets[s] of geometry s; each geometry's
// 4-wide nodes are numbered from 0 (its root) and stored at node4Off[s].
__global__ void __launch_bounds__(kThreads) k_seg4_depth_roles(Bvh4Batch b, uint32_t nInt, uint8_t* __restrict__ role)
{
  for (uint32_t j = blockIdx.x * kThreads + threadIdx.x; j < nInt; j += gridDim.x * kThreads)
  {
    const SegTree t = seg_tree(b, bc::find_segment(b.intOffsets, b.G, j));
    const uint32_t i = j - t.intBase;
    role[j] = node_role(t.lr, t.runStarts, t.L, t.nTris, node_depth(t.parent, t.L, i), b.mergeMode, i);
  }
}

// Per geometry: its 4-wide node count (role-1 nodes; 1 for a single leaf; 0
// without triangles), its first node's batch-wide rank, and the exclusive sum
// of the counts (node4Off), in one block.  out: rootRank[G], count4[G],
// node4Off[G + 1].
__global__ void __launch_bounds__(1024) k_seg4_counts(Bvh4Batch b, uint32_t nInt, const uint32_t* __restrict__ rank,
                                                      const uint32_t* __restrict__ rankTotal, uint32_t* rootRank,
                                                      uint32_t* count4, uint32_t* node4Off)
{
  __shared__ uint32_t s_part[1024];
  __shared__ uint32_t s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < b.G; base += blockDim.x)
  {
    const uint32_t s = base + threadIdx.x;
    uint32_t c = 0;
    if (s < b.G)
    {
      const uint32_t L = b.leafOffsets[s + 1] - b.leafOffsets[s];
      const uint32_t j0 = b.intOffsets[s], j1 = b.intOffsets[s + 1];
      const uint32_t r0 = j0 < nInt ? rank[j0] : *rankTotal;
      const uint32_t r1 = j1 < nInt ? rank[j1] : *rankTotal;
      c = L > 1 ? r1 - r0 : (L == 1 ? 1u : 0u);
      rootRank[s] = r0;
      count4[s] = c;
    }
    s_part[threadIdx.x] = c;
    __syncthreads();
    for (uint32_t o = 1; o < blockDim.x; o <<= 1)
    {
      const uint32_t y = threadIdx.x >= o ? s_part[threadIdx.x - o] : 0u;
      __syncthreads();
      s_part[threadIdx.x] += y;
      __syncthreads();
    }
    if (s < b.G) node4Off[s] = s_carry + s_part[threadIdx.x] - c;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry += s_part[blockDim.x - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) node4Off[b.G] = s_carry;
}

// Threads o < *rankTotal emit the 4-wide nodes of `list`; threads
// *rankTotal + s emit the lone-leaf node of geometry s when it has exactly one
// leaf.
__global__ void __launch_bounds__(kThreads) k_seg4_emit(Bvh4Batch b, uint32_t nInt, const uint8_t* __restrict__ role,
                                                        const uint32_t* __restrict__ rank,
                                                        const uint32_t* __restrict__ list,
                                                        const uint32_t* __restrict__ rankTotal,
                                                        const uint32_t* __restrict__ rootRank,
                                                        const uint32_t* __restrict__ node4Off, int format,
                                                        void* __restrict__ nodes, uint32_t* errorWord)
{
  const uint32_t n4 = min(*rankTotal, nInt);
  for (uint32_t o = blockIdx.x * kThreads + threadIdx.x; o < n4 + b.G; o += gridDim.x * kThreads)
  {
    uint32_t seg, i, j = 0;
    if (o < n4)
    {
      j = list[o];
      if (j >= nInt || role[j] != 1)
      {
        atomicOr(errorWord, kErrLayout);
        continue;
      }
      seg = bc::find_segment(b.intOffsets, b.G, j);
      i = j - b.intOffsets[seg];
    }
    else
    {
      seg = o - n4;
      if (b.leafOffsets[seg + 1] - b.leafOffsets[seg] != 1u) continue;
      i = 0;
    }
    const SegTree t = seg_tree(b, seg);
    const uint32_t r0 = rootRank[seg];
    const uint32_t local = t.L == 1u ? 0u : rank[j] - r0;
    const uint32_t outIdx = node4Off[seg] + local;
    if (outIdx >= node4Off[seg + 1])
    {
      atomicOr(errorWord, kErrLayout);
      continue;
    }
    Slot slot[4];
    const uint8_t* roleSeg = role + t.intBase;
    const uint32_t* rankSeg = rank + t.intBase;
    const int ns = node4_slots(t.lr, t.lrCount, t.runStarts, t.L, t.nTris, b.collapse, roleSeg,
                               [&](uint32_t c) { return rankSeg[c] - r0; }, i, t.tris, slot);
    write_node4(format, nodes, outIdx, slot, ns, errorWord);
  }
}

inline uint32_t grid_for(uint64_t n, int numSMs)
{
  uint64_t g = (n + kThreads - 1) / kThreads;
  const uint64_t cap = (uint64_t)numSMs * 8;
  if (g > cap) g = cap;
  return g == 0 ? 1u : (uint32_t)g;
}

}  // namespace

// Scratch: what starts at zero first (total and frontier state, 256 B; scan
// tile status; roles, N B), then the depths (N B), the node numbering (4N B;
// also a frontier list of the largest-first roles) and the other list (4N B).
namespace
{
constexpr size_t up256(size_t b) { return (b + 255) / 256 * 256; }

struct SingleScratch
{
  uint32_t *total, *state, *index, *tiles, *front2;
  uint8_t  *depth, *role;
  size_t    zeroBytes, bytes;
};
SingleScratch single_scratch(void* scratch, uint32_t N)
{
  const size_t n = N ? N : 1;
  const size_t tiles = (n + kScanTile - 1) / kScanTile;
  char* p = (char*)scratch;
  SingleScratch q;
  size_t at = 0;
  q.total = (uint32_t*)p;
  q.state = q.total + 1;
  at += 256;
  q.tiles = (uint32_t*)(p + at);
  at += up256(4 * (tiles + 8));
  q.role = (uint8_t*)(p + at);
  at += up256(n);
  q.zeroBytes = at;
  q.depth = (uint8_t*)(p + at);
  at += up256(n);
  q.index = (uint32_t*)(p + at);
  at += up256(4 * n);
  q.front2 = (uint32_t*)(p + at);
  q.bytes = at + up256(4 * n);
  return q;
}

// The largest-first roles of r's trees (at most nMost internal nodes).
cudaError_t largest_first_roles(const RoleTrees& r, uint32_t nMost, uint32_t* front0, uint32_t* front1, uint32_t* state,
                                uint8_t* role, uint32_t* errorWord, int numSMs, cudaStream_t s)
{
  k_roles_top<<<1, kTopThreads, 0, s>>>(r, front0, front1, state, role, errorWord);
  // a block per subtree: the level ends within four times the frontier's size
  // (a batch's roots may be more)
  const uint64_t most = std::min<uint64_t>(nMost, std::max<uint64_t>(4 * (uint64_t)kTopFrontier, r.params ? 0u : r.batch.G));
  const uint64_t blocks = std::min<uint64_t>(most, (uint64_t)numSMs * 8);
  k_roles_sub<<<(uint32_t)std::max<uint64_t>(blocks, 1), kSubThreads, 0, s>>>(r, front0, front1, state, role, errorWord);
  return cudaGetLastError();
}
}  // namespace

size_t bvh4_scratch_bytes(uint32_t nTris) { return single_scratch(nullptr, nTris).bytes; }

cudaError_t bvh4_plan(const Bvh4Buffers& b, int numSMs, cudaStream_t s)
{
  const uint32_t N = b.nTris;
  const SingleScratch q = single_scratch(b.scratch, N);
  const size_t nTiles = ((size_t)N + kScanTile - 1) / kScanTile;
  cudaError_t e = cudaMemsetAsync(b.scratch, 0, q.zeroBytes, s);
  if (e != cudaSuccess) return e;
  const uint32_t g = grid_for(N, numSMs);
  if (b.collapse == kCollapseLargestFirst)
  {
    RoleTrees r = {};
    r.params = b.params;
    r.one = SegTree{b.lr, b.lrCount, b.runStarts, b.parent, b.tris, 0u, N, 0u, 0u};
    r.visit = b.visit;
    r.mergeMode = b.mergeMode;
    e = largest_first_roles(r, N, q.index, q.front2, q.state, q.role, &b.params->error, numSMs, s);
    if (e != cudaSuccess) return e;
  }
  else
  {
    k_depth<<<g, kThreads, 0, s>>>(b.params, b.parent, b.visit, q.depth);
    k_roles<<<g, kThreads, 0, s>>>(b.params, b.lr, b.runStarts, N, q.depth, b.mergeMode, q.role);
  }
  k_scan_roles<<<(uint32_t)(nTiles ? nTiles : 1), kThreads, 0, s>>>(b.params, 0u, q.role, q.index, q.front2, q.tiles + 4,
                                                                      q.tiles, q.total, &b.params->error);
  return cudaMemcpyAsync(b.hostNodeCount, q.total, 4, cudaMemcpyDeviceToHost, s);
}

cudaError_t bvh4_emit(const Bvh4Buffers& b, int format, void* nodes, uint32_t maxNodes, int numSMs, cudaStream_t s)
{
  const uint32_t N = b.nTris;
  const SingleScratch q = single_scratch(b.scratch, N);
  k_emit4<<<grid_for(maxNodes, numSMs), kThreads, 0, s>>>(b.params, b.lr, b.lrCount, b.runStarts, N, b.collapse, q.role,
                                                   q.index, q.front2, format, nodes, maxNodes, b.tris, &b.params->error);
  return cudaGetLastError();
}

// Batch scratch: what starts at zero first (total and frontier state, scan
// tile status, roles), then the ranks (4 nInt B; also a frontier list),
// per-geometry rootRank, count4, node4Off (4 (3G + 1) B) and the other list.
namespace
{
struct BatchScratch
{
  uint32_t *total, *state, *rank, *rootRank, *count4, *node4Off, *tiles, *front2;
  uint8_t*  role;
  size_t    zeroBytes, bytes;
};
BatchScratch batch_scratch(void* scratch, uint32_t nInt, uint32_t G)
{
  const size_t n = nInt ? nInt : 1;
  const size_t tiles = (n + kScanTile - 1) / kScanTile;
  char* p = (char*)scratch;
  BatchScratch q;
  size_t at = 0;
  q.total = (uint32_t*)p;
  q.state = q.total + 1;
  at += 256;
  q.tiles = (uint32_t*)(p + at);
  at += up256(4 * (tiles + 8));
  q.role = (uint8_t*)(p + at);
  at += up256(n);
  q.zeroBytes = at;
  q.rank = (uint32_t*)(p + at);
  at += up256(4 * n);
  q.rootRank = (uint32_t*)(p + at);
  q.count4 = q.rootRank + G;
  q.node4Off = q.count4 + G;
  at += up256(4 * (3 * (size_t)G + 1));
  q.front2 = (uint32_t*)(p + at);
  q.bytes = at + up256(4 * n);
  return q;
}
}  // namespace

size_t bvh4_batch_scratch_bytes(uint32_t nInt, uint32_t G) { return batch_scratch(nullptr, nInt, G).bytes; }

cudaError_t bvh4_plan_batch(const Bvh4Batch& b, uint32_t nInt, void* scratch, uint32_t* hostCount4,
                            uint32_t* hostNode4Off, uint32_t* errorWord, int numSMs, cudaStream_t s)
{
  const BatchScratch q = batch_scratch(scratch, nInt, b.G);
  const size_t nTiles = ((size_t)(nInt ? nInt : 1) + kScanTile - 1) / kScanTile;
  cudaError_t e = cudaMemsetAsync(scratch, 0, q.zeroBytes, s);
  if (e != cudaSuccess) return e;
  if (nInt)
  {
    if (b.collapse == kCollapseLargestFirst)
    {
      RoleTrees r = {};
      r.batch = b;
      r.nInt = nInt;
      r.mergeMode = b.mergeMode;
      e = largest_first_roles(r, nInt, q.rank, q.front2, q.state, q.role, errorWord, numSMs, s);
      if (e != cudaSuccess) return e;
    }
    else
      k_seg4_depth_roles<<<grid_for(nInt, numSMs), kThreads, 0, s>>>(b, nInt, q.role);
    k_scan_roles<<<(uint32_t)nTiles, kThreads, 0, s>>>(nullptr, nInt, q.role, q.rank, q.front2, q.tiles + 4, q.tiles, q.total,
                                                       errorWord);
  }
  k_seg4_counts<<<1, 1024, 0, s>>>(b, nInt, q.rank, q.total, q.rootRank, q.count4, q.node4Off);
  e = cudaMemcpyAsync(hostCount4, q.count4, 4 * (size_t)b.G, cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return e;
  return cudaMemcpyAsync(hostNode4Off, q.node4Off, 4 * ((size_t)b.G + 1), cudaMemcpyDeviceToHost, s);
}

cudaError_t bvh4_emit_batch(const Bvh4Batch& b, uint32_t nInt, void* scratch, int format, void* nodes,
                            uint32_t* errorWord, int numSMs, cudaStream_t s)
{
  const BatchScratch q = batch_scratch(scratch, nInt, b.G);
  k_seg4_emit<<<grid_for((uint64_t)nInt + b.G, numSMs), kThreads, 0, s>>>(b, nInt, q.role, q.rank, q.front2, q.total, q.rootRank,
                                                                           q.node4Off, format, nodes, errorWord);
  return cudaGetLastError();
}

}  // namespace hrt
