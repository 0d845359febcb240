// Leaves, triangle records and bottom-up boxes of the LBVH, for a single geometry
// and for a segmented batch: a kernel over slices of leaves, and the walks above
// the slices in tiers.
//
// A block of k_leaf_tree owns the leaves [lo, hi) of one slice, a thread each.
//
// Leaves (kernel1D_MakeLeavesFromTriangles, core/builders/lbvh.cpp:350-384):
// leaf i is node L-1+i, its box the union of its run's triangle boxes taken in
// sorted order.  The slice's triangles are taken in chunks, a thread each: the
// record (vertex and edges, or the vertices), the sorted indices
// (AppendTreeData, core/BVH2CommonRT_host.cpp:45-64) and the box go through
// shared memory, so that records and indices leave as whole lines; every leaf
// then unites its own triangles' boxes in order.
//
// Boxes: the reference runs 32 sweeps over all internal nodes
// (core/builders/lbvh.cpp:443-489, :798-802); here each leaf walks towards the
// root and the second child to arrive at a node computes it, so every node is
// computed once from its finished children: box = (min, max) of the children
// in (left, right) order, count = children's counts + 2.  An internal node i of
// a Karras tree has i as one end of its leaf range, so the nodes whose range
// lies inside the slice are among i in [lo, hi - 1): their links, boxes and
// arrival counters are in shared memory (acquire-release at block scope).  The
// nodes whose range leaves the slice are left to k_climb.  Every node a thread
// reads was written by the thread that released the counter it acquired, or by
// an earlier kernel.
//
// What bounds it: the walks are chains of dependent steps and the leaves are
// gathers and AoS writes.  As a kernel of leaves, a thread per leaf with its own
// 48-byte stores, and one of walks with links and boxes read from L2, the
// 2M-triangle heightfield took 93 + 107 us; in one kernel 153; in this one and
// k_climb 101 + 32.
#pragma once

#include "build_common.cuh"

namespace hrt
{
namespace bc
{

constexpr uint32_t kSlice = 512;  // leaves, threads and triangles of a chunk
// k_climb: a group is kFan slices, or kFan groups of the tier below.  Each
// slice or group hands at most kEdge nodes of either list to the next tier: a
// range of leaves of a tree at most 31 levels deep is covered by 62 nodes, and
// at most 62 ancestors of its ends have an index in it and leave it.
constexpr uint32_t kFan = 32, kEdge = 64, kSlots = kFan * kEdge;
constexpr int      kClimbThreads = 1024;

constexpr uint32_t kSlotMark = 0x80000000u;  // of a slot in visit; a root's visit ends as 2
constexpr uint32_t kNone = 0xFFFFFFFFu;

// Where tier t's lists are: `producers` slices (t = 0) or groups, each with
// kEdge open nodes (outermost finished ones: {LR index, parent | kUpRight of a
// right child}), kEdge leaving nodes (LR index, the far end of its range, parent
// as above) and a word of both counts.
constexpr uint32_t kUpRight = 0x80000000u;
struct TierLists
{
  uint2*    open;
  uint32_t *leaving, *end, *up, *counts;
  uint32_t  producers;
};
__host__ __device__ inline TierLists tier_lists(uint32_t* lists, uint32_t nTris, int tier)
{
  uint32_t producers = (nTris + kSlice - 1) / kSlice;
  for (int t = 0; t < tier; t++)
  {
    lists += (5 * kEdge + 2) * (size_t)producers;
    producers = (producers + kFan - 1) / kFan;
  }
  const size_t n = kEdge * (size_t)producers;
  return {reinterpret_cast<uint2*>(lists), lists + 2 * n, lists + 3 * n, lists + 4 * n, lists + 5 * n, producers};
}
// Words of all of a build's lists.
inline size_t list_words(uint32_t nTris)
{
  size_t words = 0;
  for (uint32_t producers = (nTris + kSlice - 1) / kSlice; producers > 1; producers = (producers + kFan - 1) / kFan)
    words += (5 * kEdge + 2) * (size_t)producers;
  return words;
}

struct LeafTree
{
  const float4*   verts;
  const uint32_t* idx;
  const uint32_t* sortedTri;
  const uint32_t* runStarts;
  uint32_t        nTris;  // all of a batch's
  uint32_t        nVerts;
  BVHNode32*      lr;
  uint32_t*       lrCount;
  TriRec*         tris;
  uint32_t*       sortedIdx;
  const uint32_t* parent;
  uint32_t*       visit;
  const uint32_t* rangeEnd;
  uint32_t*       lists;  // list_words() of scratch, 8-byte aligned: tier_lists()
  uint32_t*       errorWord;
  int             vertexRecords;
  // one geometry: its leaf count
  const BuildParams* params;
  // a batch: geometry s's triangles, leaves, internal nodes and LR nodes start
  // at these offsets (local numbering within each); counts[0] = all leaves
  const uint32_t *vertOffsets, *triOffsets, *leafOffsets, *intOffsets, *nodeOffsets, *recOffsets, *counts;
  uint32_t        G;
  PairRec*        recs;  // a geometry of one leaf gets its record here; null for 4-wide layouts
};

// A parent's box from its finished child's (mn, mx) and the sibling's, in
// (left, right) order, which decides the sign of a zero.
__device__ __forceinline__ void unite(bool left, float (&mn)[3], float (&mx)[3], const float4& slo, const float4& shi)
{
  const float smn[3] = {slo.x, slo.y, slo.z}, smx[3] = {shi.x, shi.y, shi.z};
#pragma unroll
  for (int c = 0; c < 3; c++)
  {
    mn[c] = left ? lm_min(mn[c], smn[c]) : lm_min(smn[c], mn[c]);
    mx[c] = left ? lm_max(mx[c], smx[c]) : lm_max(smx[c], mx[c]);
  }
}

__device__ __forceinline__ void store_node(BVHNode32* n, const float (&mn)[3], const float (&mx)[3], uint32_t l, uint32_t r)
{
  float4* p = reinterpret_cast<float4*>(n);
  p[0] = make_float4(mn[0], mn[1], mn[2], __uint_as_float(l));
  p[1] = make_float4(mx[0], mx[1], mx[2], __uint_as_float(r));
}

template <bool SEG>
__global__ void __launch_bounds__(kSlice, 3) k_leaf_tree(LeafTree a)
{
  // chunk: records, indices, boxes of its triangles; then the slice's tree
  struct Chunk
  {
    float4   rec[3 * kSlice];
    uint32_t idx[3 * kSlice];
    float    box[6][kSlice];
    uint8_t  end[kSlice];
  };
  struct Tree
  {
    float    leaf[6][kSlice], node[6][kSlice];
    uint32_t count[kSlice], leafParent[kSlice], nodeParent[kSlice], rangeEnd[kSlice], left[kSlice], right[kSlice];
    uint32_t visit[kSlice];
  };
  __shared__ union __align__(16)
  {
    Chunk c;
    Tree  t;
  } sh;

  const uint32_t Ltot = SEG ? a.counts[0] : (a.params->nLeaves <= a.nTris ? a.params->nLeaves : 0u);
  const uint32_t lo = blockIdx.x * kSlice;
  if (lo >= Ltot) return;
  const uint32_t hi = min(lo + kSlice, Ltot);
  const uint32_t tid = threadIdx.x, g = lo + tid;
  const bool active = g < hi;
  __shared__ uint32_t s_open, s_leaving;
  const TierLists out = tier_lists(a.lists, a.nTris, 0);
  if (tid == 0) s_open = s_leaving = 0u;

  // the leaf's geometry: first leaf, triangle, LR node and internal node, leaf count
  uint32_t lb = 0, tb = 0, te = a.nTris, nb = 0, ib = 0, L = Ltot, seg = 0;
  if (SEG && active)
  {
    seg = find_segment(a.leafOffsets, a.G, g);
    lb = a.leafOffsets[seg];
    L = a.leafOffsets[seg + 1] - lb;
    tb = a.triOffsets[seg];
    te = a.triOffsets[seg + 1];
    nb = a.nodeOffsets[seg];
    ib = a.intOffsets[seg];
  }
  const uint32_t k = g - lb;  // the leaf in its geometry
  uint32_t start = 0, end = 0;
  if (active)
  {
    start = a.runStarts[g];
    end = (k + 1 < L) ? a.runStarts[g + 1] : te;
    if (k >= L || end > te || start >= end || start < tb)
    {
      atomicOr(a.errorWord, kErrLayout);
      start = end = 0;
    }
    if (end - start > 127u) atomicOr(a.errorWord, kErrLeafCount);
  }

  // the slice's triangles, in chunks
  const uint32_t first = min(a.runStarts[lo], a.nTris);
  const uint32_t last = hi < Ltot ? min(a.runStarts[hi], a.nTris) : a.nTris;
  float mn[3] = {1e10f, 1e10f, 1e10f}, mx[3] = {-1e10f, -1e10f, -1e10f};
  for (uint32_t c0 = first; c0 < last; c0 += kSlice)
  {
    const uint32_t n = min(kSlice, last - c0);
    sh.c.end[tid] = 0;
    __syncthreads();
    if (end > c0 && end - 1u - c0 < kSlice) sh.c.end[end - 1u - c0] = 1;
    __syncthreads();
    if (tid < n)
    {
      const uint32_t j = c0 + tid, tri = a.sortedTri[j];
      uint32_t vb = 0, nV = a.nVerts, t0 = 0;
      if (SEG)
      {
        const uint32_t s = find_segment(a.triOffsets, a.G, j);
        vb = a.vertOffsets[s];
        nV = a.vertOffsets[s + 1] - vb;
        t0 = a.triOffsets[s];
      }
      uint32_t ia = a.idx[3 * (size_t)tri + 0], ibx = a.idx[3 * (size_t)tri + 1], ic = a.idx[3 * (size_t)tri + 2];
      if (ia >= nV || ibx >= nV || ic >= nV)
      {
        atomicOr(a.errorWord, kErrIndexRange);
        ia = ibx = ic = 0;
      }
      const float4 A = a.verts[vb + ia], B = a.verts[vb + ibx], C = a.verts[vb + ic];
      sh.c.box[0][tid] = lm_min(A.x, lm_min(B.x, C.x));
      sh.c.box[1][tid] = lm_min(A.y, lm_min(B.y, C.y));
      sh.c.box[2][tid] = lm_min(A.z, lm_min(B.z, C.z));
      sh.c.box[3][tid] = lm_max(A.x, lm_max(B.x, C.x));
      sh.c.box[4][tid] = lm_max(A.y, lm_max(B.y, C.y));
      sh.c.box[5][tid] = lm_max(A.z, lm_max(B.z, C.z));
      // flags: bit 0 ends a binary leaf, bit 1 a 4-wide leaf (cleared later
      // where the collapse merges two leaves); the watertight test wants the
      // vertices themselves
      const uint32_t flags = sh.c.end[tid] ? 3u : 0u;
      sh.c.rec[3 * tid] = make_float4(A.x, A.y, A.z, __uint_as_float(flags));
      if (a.vertexRecords)
      {
        sh.c.rec[3 * tid + 1] = make_float4(B.x, B.y, B.z, __uint_as_float(tri - t0));
        sh.c.rec[3 * tid + 2] = make_float4(C.x, C.y, C.z, 0.0f);
      }
      else
      {
        sh.c.rec[3 * tid + 1] = make_float4(__fsub_rn(B.x, A.x), __fsub_rn(B.y, A.y), __fsub_rn(B.z, A.z),
                                            __uint_as_float(tri - t0));
        sh.c.rec[3 * tid + 2] = make_float4(__fsub_rn(C.x, A.x), __fsub_rn(C.y, A.y), __fsub_rn(C.z, A.z), 0.0f);
      }
      sh.c.idx[3 * tid] = ia;
      sh.c.idx[3 * tid + 1] = ibx;
      sh.c.idx[3 * tid + 2] = ic;
    }
    __syncthreads();
    float4* rec = reinterpret_cast<float4*>(a.tris) + 3 * (size_t)c0;
    uint32_t* idx = a.sortedIdx + 3 * (size_t)c0;
    for (uint32_t q = tid; q < 3 * n; q += kSlice)
    {
      rec[q] = sh.c.rec[q];
      idx[q] = sh.c.idx[q];
    }
    const uint32_t u0 = max(start, c0), u1 = min(end, c0 + n);
    for (uint32_t j = u0; j < u1; j++)
#pragma unroll
      for (int c = 0; c < 3; c++)
      {
        mn[c] = lm_min(mn[c], sh.c.box[c][j - c0]);
        mx[c] = lm_max(mx[c], sh.c.box[3 + c][j - c0]);
      }
    __syncthreads();
  }

  // the leaf's node, and the slice's links
  if (active)
  {
    float4* p = reinterpret_cast<float4*>(a.lr + nb + L - 1 + k);
    p[0] = make_float4(mn[0], mn[1], mn[2], __uint_as_float(pack_offset_and_size(start - tb, end - start)));
    p[1] = make_float4(mx[0], mx[1], mx[2], __uint_as_float(0xFFFFFFFFu));
    a.lrCount[nb + L - 1 + k] = 0;
#pragma unroll
    for (int c = 0; c < 3; c++)
    {
      sh.t.leaf[c][tid] = mn[c];
      sh.t.leaf[3 + c][tid] = mx[c];
    }
    sh.t.visit[tid] = 0u;
    if (L > 1)
    {
      sh.t.leafParent[tid] = a.parent[nb + L - 1 + k];
      if (k + 1 < L)
      {
        sh.t.nodeParent[tid] = k ? a.parent[nb + k] : 0u;
        sh.t.rangeEnd[tid] = a.rangeEnd[ib + k];
        sh.t.left[tid] = a.lr[nb + k].leftOffset;
        sh.t.right[tid] = a.lr[nb + k].escapeIndex;
        const uint32_t j = sh.t.rangeEnd[tid];
        if (min(k, j) + lb < lo || max(k, j) + lb >= hi)  // a node that leaves the slice
        {
          const uint32_t e = atomicAdd(&s_leaving, 1u);
          if (e < kEdge)
          {
            const size_t at = kEdge * (size_t)blockIdx.x + e;
            out.leaving[at] = nb + k;
            out.end[at] = j;
            out.up[at] = k ? sh.t.nodeParent[tid] | (a.lr[nb + sh.t.nodeParent[tid]].escapeIndex == k ? kUpRight : 0u) : 0u;
            a.visit[ib + k] = kSlotMark | (kEdge * (blockIdx.x % kFan) + e);
          }
          else
            atomicOr(a.errorWord, kErrLayout);
        }
      }
    }
    if (SEG && L == 1u && a.recs != nullptr)
    {
      PairRec r;
      r.a = make_float4(mn[0], mn[1], mn[2], mx[0]);
      r.b = make_float4(mx[1], mx[2], 0.0f, 0.0f);
      r.c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      r.d = make_uint4(kLeafBit | (start - tb), kEmptyRef, 0u, 0u);
      a.recs[a.recOffsets[seg]] = r;
    }
  }
  __syncthreads();

  // the walk; slot of a node or leaf of the slice: its index + lb - lo.  The
  // finished node's own box and count stay in registers; only the sibling's
  // are read.
  const uint32_t off = lb - lo;
  uint32_t node = active ? L - 1 + k : 0, count = 0, p = 0;
  if (node != 0) p = sh.t.leafParent[tid];
  for (int level = 0; node != 0; level++)
  {
    if (p + 1u >= L || level > kMaxDepth)  // not an internal node, or a cycle: the hierarchy is inconsistent
    {
      atomicOr(a.errorWord, kErrLayout);
      break;
    }
    const uint32_t slot = p + off;  // wraps below the slice
    bool inSlice = slot < hi - lo;
    if (inSlice)
    {
      const uint32_t j = sh.t.rangeEnd[slot];
      inSlice = min(p, j) + lb >= lo && max(p, j) + lb < hi;
    }
    if (!inSlice)
    {
      const uint32_t e = atomicAdd(&s_open, 1u);
      if (e < kEdge)
        out.open[kEdge * (size_t)blockIdx.x + e] =
            make_uint2(nb + node, p | (a.lr[nb + p].escapeIndex == node ? kUpRight : 0u));
      else atomicOr(a.errorWord, kErrLayout);
      break;
    }
    if (atomic_add_acq_rel_cta(&sh.t.visit[slot], 1u) == 0u) break;  // the sibling is not finished yet
    if (p == 0u) a.visit[ib] = 2u;  // the root finished inside the slice (a later kernel checks the counter)
    const uint32_t l = sh.t.left[slot], r = sh.t.right[slot];
    const uint32_t sib = l == node ? r : l;
    const bool leaf = sib + 1u >= L;
    // the sibling lies in the slice, whose range holds the parent's
    const uint32_t q = min((leaf ? sib - (L - 1) : sib) + off, kSlice - 1u);
    const float(*box)[kSlice] = leaf ? sh.t.leaf : sh.t.node;
    const float4 slo = make_float4(box[0][q], box[1][q], box[2][q], 0.0f);
    const float4 shi = make_float4(box[3][q], box[4][q], box[5][q], 0.0f);
    unite(l == node, mn, mx, slo, shi);
    count += (leaf ? 0u : sh.t.count[q]) + 2u;
#pragma unroll
    for (int c = 0; c < 3; c++)
    {
      sh.t.node[c][slot] = mn[c];
      sh.t.node[3 + c][slot] = mx[c];
    }
    sh.t.count[slot] = count;
    store_node(a.lr + nb + p, mn, mx, l, r);
    a.lrCount[nb + p] = count;
    node = p;
    p = sh.t.nodeParent[slot];
  }
  if (a.nTris <= kSlice) return;
  __syncthreads();
  if (tid == 0) out.counts[blockIdx.x] = min(s_open, kEdge) | min(s_leaving, kEdge) << 16;
}

// The walks on from the slices' outermost nodes, tier by tier: a block takes a
// group of kFan slices (or groups), reads the nodes that leave those into
// shared memory, a slot each (their links are static), and walks from the
// outermost finished nodes below as far as nodes whose range lies in the group.
// A level is then a chain of shared-memory accesses; a node's box goes out
// beside it.  Slot of a node: its place in the lists, which `visit` holds.
// With links, boxes and arrival counters in L2, one kernel, a level was two
// latencies and a release at device scope: 41 us for 2M triangles, 40 for
// 500,000, 24 for 15,000; so 32 (three tiers), 22 and 8.
// a slot's link: its parent's slot (below kSlots), its side there, what it is
constexpr uint32_t kLinkRight = 1u << 12, kLinkOut = 1u << 13, kLinkIn = 1u << 14, kLinkRoot = 1u << 15,
                   kLinkArrived = 1u << 16;

struct ClimbShared
{
  float    box[2][6][kSlots];  // of a slot's left and right child
  uint32_t link[kSlots], node[kSlots], up[kSlots];
};

__device__ __forceinline__ uint32_t arrive_cta(uint32_t* link)
{
  uint32_t old;
  asm volatile("atom.acq_rel.cta.shared::cta.or.b32 %0, [%1], %2;"
               : "=r"(old)
               : "r"((uint32_t)__cvta_generic_to_shared(link)), "r"(kLinkArrived)
               : "memory");
  return old;
}

template <bool SEG> __global__ void __launch_bounds__(kClimbThreads) k_climb(LeafTree a, int tier, uint64_t groupLeaves)
{
  extern __shared__ uint4 s_climb[];
  ClimbShared& sh = *reinterpret_cast<ClimbShared*>(s_climb);
  __shared__ uint32_t s_counts[kFan], s_open, s_leaving;
  const uint32_t Ltot = SEG ? a.counts[0] : (a.params->nLeaves <= a.nTris ? a.params->nLeaves : 0u);
  if (blockIdx.x * groupLeaves >= Ltot) return;
  const uint32_t tid = threadIdx.x, lo = (uint32_t)(blockIdx.x * groupLeaves);
  const TierLists in = tier_lists(a.lists, a.nTris, tier), out = tier_lists(a.lists, a.nTris, tier + 1);
  const bool last = gridDim.x == 1;
  if (tid < kFan)
  {
    const uint64_t first = lo + tid * (groupLeaves / kFan);
    s_counts[tid] = first < Ltot ? in.counts[blockIdx.x * kFan + tid] : 0u;
  }
  if (tid == 0) s_open = s_leaving = 0u;
  __syncthreads();

  // list item s: producer s % kFan, its item s / kFan; slot kEdge * producer + item
  auto slot_of = [](uint32_t s) { return kEdge * (s % kFan) + s / kFan; };
  // geometry of LR node `at`: first LR node, internal node and leaf, leaves
  auto geometry = [&](uint32_t at, uint32_t& nb, uint32_t& ib, uint32_t& lb, uint32_t& L) {
    nb = ib = lb = 0;
    L = Ltot;
    if (!SEG) return;
    const uint32_t s = find_segment(a.nodeOffsets, a.G, at);
    nb = a.nodeOffsets[s];
    ib = a.intOffsets[s];
    lb = a.leafOffsets[s];
    L = a.leafOffsets[s + 1] - lb;
  };
  // The loads go in stages over all of a thread's items, so that a stage is one
  // latency.  Item q of a list is producer c's number k.
  constexpr int kPer = kSlots / kClimbThreads;
  struct Item
  {
    uint32_t at, end, up;
  } edge[kPer], open[kPer];
#pragma unroll
  for (int q = 0; q < kPer; q++)
  {
    const uint32_t s = q * kClimbThreads + tid, c = s % kFan, k = s / kFan, n = s_counts[c];
    const size_t list = kEdge * ((size_t)blockIdx.x * kFan + c) + k;
    edge[q].at = open[q].at = kNone;
    if (k < n >> 16) edge[q] = {in.leaving[list], in.end[list], in.up[list]};
    if (k < (n & 0xFFFFu))
    {
      const uint2 v = in.open[list];
      open[q] = {v.x, 0u, v.y};
    }
  }
  // where a node goes on: its parent's slot and its side there
  auto link_up = [&](const Item& t, uint32_t ib, uint32_t lb, uint32_t L) {
    const uint32_t p = t.up & ~kUpRight;
    if (p + 1u >= L)
    {
      atomicOr(a.errorWord, kErrLayout);
      return kLinkOut;
    }
    const bool inside = p + lb >= lo && p + lb - lo < groupLeaves;
    return ((t.up & kUpRight) ? kLinkRight : 0u) | (inside ? a.visit[ib + p] & (kSlots - 1u) : kLinkOut);
  };
  uint32_t moved[kPer], from[kPer], fromLink[kPer];
#pragma unroll
  for (int q = 0; q < kPer; q++)
  {
    const Item& t = edge[q];
    uint32_t nb, ib, lb, L;
    moved[q] = kNone;
    from[q] = open[q].at;
    if (t.at != kNone)
    {
      geometry(t.at, nb, ib, lb, L);
      const uint32_t i = t.at - nb, r0 = min(i, t.end), r1 = max(i, t.end);
      uint32_t link = 0u;
      if (r0 + lb >= lo && r1 + lb - lo < groupLeaves)
      {
        link = kLinkIn | (i == 0u ? kLinkRoot : link_up(t, ib, lb, L));
        a.lrCount[t.at] = 2u * (r1 - r0);  // two for each node below
      }
      else
      {
        const uint32_t e = atomicAdd(&s_leaving, 1u);
        if (last || e >= kEdge) atomicOr(a.errorWord, kErrLayout);
        else
        {
          const size_t to = kEdge * (size_t)blockIdx.x + e;
          out.leaving[to] = t.at;
          out.end[to] = t.end;
          out.up[to] = t.up;
          moved[q] = ib + i;
          link = e;
        }
      }
      const uint32_t slot = slot_of(q * kClimbThreads + tid);
      sh.link[slot] = link;
      sh.node[slot] = t.at;
      sh.up[slot] = t.up;
    }
    if (from[q] != kNone)
    {
      geometry(from[q], nb, ib, lb, L);
      fromLink[q] = link_up(open[q], ib, lb, L);
    }
  }
  __syncthreads();  // every slot that the block needs has been read from visit
#pragma unroll
  for (int q = 0; q < kPer; q++)
    if (moved[q] != kNone)
      a.visit[moved[q]] = kSlotMark | (kEdge * (blockIdx.x % kFan) + sh.link[slot_of(q * kClimbThreads + tid)]);
#pragma unroll 1
  for (int q = 0; q < kPer; q++)
  {
    uint32_t at = kNone, link = 0, up = 0;
#pragma unroll
    for (int w = 0; w < kPer; w++)
      if (w == q)
      {
        at = from[w];
        link = fromLink[w];
        up = open[w].up;
      }
    if (at == kNone) continue;
    float4 lo4, hi4;
    load_node_cg(a.lr + at, lo4, hi4);
    float mn[3] = {lo4.x, lo4.y, lo4.z}, mx[3] = {hi4.x, hi4.y, hi4.z};
    for (int level = 0; level <= kMaxDepth; level++)
    {
      const uint32_t slot = link & (kSlots - 1u), side = (link & kLinkRight) ? 1u : 0u;
      if ((link & kLinkOut) || !(sh.link[slot] & kLinkIn))
      {
        const uint32_t e = atomicAdd(&s_open, 1u);
        if (last || e >= kEdge) atomicOr(a.errorWord, kErrLayout);
        else out.open[kEdge * (size_t)blockIdx.x + e] = make_uint2(at, up);
        break;
      }
#pragma unroll
      for (int c = 0; c < 3; c++)
      {
        sh.box[side][c][slot] = mn[c];
        sh.box[side][3 + c][slot] = mx[c];
      }
      link = arrive_cta(&sh.link[slot]);
      if (!(link & kLinkArrived)) break;  // the sibling is not finished yet
      const float4 slo = make_float4(sh.box[side ^ 1u][0][slot], sh.box[side ^ 1u][1][slot], sh.box[side ^ 1u][2][slot], 0.0f);
      const float4 shi = make_float4(sh.box[side ^ 1u][3][slot], sh.box[side ^ 1u][4][slot], sh.box[side ^ 1u][5][slot], 0.0f);
      unite(side == 0u, mn, mx, slo, shi);
      at = sh.node[slot];
      up = sh.up[slot];
#pragma unroll
      for (int c = 0; c < 3; c++)
      {
        a.lr[at].boxMin[c] = mn[c];
        a.lr[at].boxMax[c] = mx[c];
      }
      if (link & kLinkRoot)
      {
        uint32_t nb, ib, lb, L;
        geometry(at, nb, ib, lb, L);
        a.visit[ib] = 2u;
        break;
      }
    }
  }
  if (last) return;
  __syncthreads();
  if (tid == 0) out.counts[blockIdx.x] = min(s_open, kEdge) | min(s_leaving, kEdge) << 16;
}

// Leaves and boxes; a single slice leaves nothing to walk on from.
template <bool SEG> cudaError_t leaf_tree(const LeafTree& t, cudaStream_t s)
{
  uint32_t producers = (t.nTris + kSlice - 1) / kSlice;
  uint64_t leaves = kSlice;
  k_leaf_tree<SEG><<<producers, kSlice, 0, s>>>(t);
  if (producers > 1)
  {
    const cudaError_t e = cudaFuncSetAttribute(k_climb<SEG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(ClimbShared));
    if (e != cudaSuccess) return e;
  }
  for (int tier = 0; producers > 1; tier++)
  {
    producers = (producers + kFan - 1) / kFan;
    leaves *= kFan;
    k_climb<SEG><<<producers, kClimbThreads, sizeof(ClimbShared), s>>>(t, tier, leaves);
  }
  return cudaGetLastError();
}

}  // namespace bc
}  // namespace hrt
