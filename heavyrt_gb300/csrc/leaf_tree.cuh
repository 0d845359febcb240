// Leaves, triangle records and bottom-up boxes of the LBVH in one kernel, for a
// single geometry and for a segmented batch.
//
// A block owns the leaves [lo, hi) of one slice, a thread each.
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
// arrival counters are in shared memory (acquire-release at block scope).  Only
// the nodes whose range leaves the slice use the device-wide counters
// (acquire-release at device scope, children read from L2).  Every node a
// thread reads was written by the thread that released the counter it acquired.
//
// What bounds it: the walks are chains of dependent steps and the leaves are
// gathers and AoS writes.  As a kernel of leaves, a thread per leaf with its own 48-byte
// stores, and one of walks with links and boxes read from L2, the 2M-triangle
// heightfield took 93 + 107 us; in one kernel 153; in these two 97 + 41.
#pragma once

#include "build_common.cuh"

namespace hrt
{
namespace bc
{

constexpr uint32_t kSlice = 512;  // leaves, threads and triangles of a chunk

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
  uint32_t*       open;       // LR indices of the outermost finished nodes of the slices
  uint32_t*       openCount;  // zero before
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
  if (!active) return;

  // the walk; slot of a node or leaf of the slice: its index + lb - lo.  The
  // finished node's own box and count stay in registers; only the sibling's
  // are read.
  const uint32_t off = lb - lo;
  uint32_t node = L - 1 + k, count = 0, p = 0;
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
      a.open[atomicAdd(a.openCount, 1u)] = nb + node;  // one per leaf at most: the list holds them
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
}

// The walks on from the slices' outermost nodes.  A level is a chain of memory
// latencies, so the links (static) are read beside the arrival and the next
// parent beside the sibling.
template <bool SEG> __global__ void __launch_bounds__(128) k_climb(LeafTree a)
{
  const uint32_t n = *a.openCount;
  for (uint32_t e = blockIdx.x * 128 + threadIdx.x; e < n; e += gridDim.x * 128)
  {
    const uint32_t at = a.open[e];
    uint32_t nb = 0, ib = 0, L = SEG ? 0u : a.params->nLeaves;
    if (SEG)
    {
      const uint32_t s = find_segment(a.nodeOffsets, a.G, at);
      nb = a.nodeOffsets[s];
      ib = a.intOffsets[s];
      L = a.leafOffsets[s + 1] - a.leafOffsets[s];
    }
    uint32_t node = at - nb, p = a.parent[at];
    float4 lo4, hi4;
    load_node_cg(a.lr + at, lo4, hi4);
    uint32_t count = __ldcg(&a.lrCount[at]);
    float mn[3] = {lo4.x, lo4.y, lo4.z}, mx[3] = {hi4.x, hi4.y, hi4.z};
    for (int level = 0; node != 0; level++)
    {
      if (p + 1u >= L || level > kMaxDepth)
      {
        atomicOr(a.errorWord, kErrLayout);
        break;
      }
      const uint32_t l = __ldcg(&a.lr[nb + p].leftOffset), r = __ldcg(&a.lr[nb + p].escapeIndex);
      if (atomic_add_acq_rel(&a.visit[ib + p], 1u) == 0u) break;
      const uint32_t sib = l == node ? r : l;
      const uint32_t above = p != 0u ? a.parent[nb + p] : 0u;
      load_node_cg(a.lr + nb + sib, lo4, hi4);
      count += __ldcg(&a.lrCount[nb + sib]) + 2u;
      unite(l == node, mn, mx, lo4, hi4);
      store_node(a.lr + nb + p, mn, mx, l, r);
      a.lrCount[nb + p] = count;
      node = p;
      p = above;
    }
  }
}

// Blocks of k_climb: an entry or two a thread at the usual dozen per slice.
inline uint32_t climb_blocks(uint32_t nTris, int numSMs)
{
  const uint64_t want = ((uint64_t)(nTris + kSlice - 1) / kSlice * 12 + 127) / 128;
  const uint64_t most = (uint64_t)numSMs * 16;
  return (uint32_t)(want < 1 ? 1 : (want > most ? most : want));
}

}  // namespace bc
}  // namespace hrt
