// Nearest-hit / any-hit traversal of the LBVH.
//
// Each ray makes the decisions of HeavyRT's BVH2TraverseC32
// (core/BVH2CommonRT.cpp:49-141) on the same binary tree: load the two
// children of the current node, slab-test both (core/raytrace_common.h:67-80),
// descend into the nearer hit child (child 0 on equal entry distance), push
// the other, pop when neither is hit.  The leaf test is the reference's
// Moller-Trumbore with 1e-6 barycentric slack (core/BVH2CommonRT.cpp:9-47),
// written with explicit round-to-nearest intrinsics in the reference's
// evaluation order, so t/u/v match the CPU reference bit for bit.
//
// Slab distances only feed comparisons (hit tests, near-first choice, pruning
// against the current t), so the slab test takes min/max with the hardware
// fminf/fmaxf instead of the reference's std::min/std::max selects: the two
// differ only in the sign of a zero result and in one axis whose distances are
// NaN (finite rays have none, because SafeInverse keeps |1/d| <= 1e36), and
// +0 == -0 in every comparison, so every decision is unchanged.
//
// Scheduling: a persistent warp pool.  Each warp keeps one ray per lane; when
// enough lanes have finished, the warp refills them from a global ray counter
// with one atomic per warp (ballot + popc ranking), so lanes do not idle while
// the warp's longest ray finishes.  A ray's own visit order does not depend on
// the schedule.  A one-thread-per-ray grid is kept as a configuration.
//
// Memory: a node or child pair is read in 32-byte pieces, one 256-bit load
// each, a triangle as one 48-byte record (three 128-bit loads).  The stack's
// first S entries live in shared memory, interleaved by thread so a warp's
// pushes and pops hit 32 different banks; deeper entries go to a per-thread
// array in local memory (S is a launch parameter, full depth by default; the
// two-level kernels keep the whole stack in local memory by default).
//
// What bounds it (profiles/trace_kernels_cases.txt): in 8-bit and FP16 nodes
// instruction issue, 58 to 75% of cycles, at 11 to 17 of 32 threads per
// instruction, since a warp's rays part ways; in binary and FP32 nodes, where 41
// to 45% of cycles issue, the latency of nodes that miss L1 (9 to 15 stall
// cycles an issue).  DRAM moves 2 to 7% of the copy bandwidth for occlusion and
// random rays, a quarter of it for full-HD eye rays, whose rays and hits are
// half the traffic.  So the slab test runs on packed pairs of floats, picks
// entry planes by the direction's sign, and takes its min and max three at a
// time; lanes visit runs of nodes between leaves; results are written when a
// warp refills.  Against four 128-bit loads, scalar slabs and one node or leaf per
// step: 4M occlusion rays on 2M triangles, FP16 nodes 680 -> 577 us; 1M random
// rays into 1M triangles, 8-bit nodes, watertight 1,953 -> 1,475 us; full-HD
// eye rays, binary 185 -> 155 us.
//
// Triangle test: the reference's Moller-Trumbore (records {A, B-A, C-A}), or,
// for scenes built for it, the watertight test of Woop, Benthin & Wald
// (records {A, B, C}); both are template variants of the same kernels.
#pragma once

#include <cuda_fp16.h>

#include "hrt_kernels.cuh"
#include "../../include/hrt.h"

namespace hrt
{
namespace
{

// Stack bounds: the binary tree of distinct 30-bit codes is at most 30 levels
// deep (each level lengthens the common prefix), one push per level; the
// 4-wide tree halves the levels and pushes at most 3 per level.
constexpr int      kStack2 = 32;
constexpr int      kStack4 = 48;
constexpr uint32_t kNoRay = 0xFFFFFFFFu;
// Lane::cur of a lane whose ray is finished (or that has none): no reference
// of a tree has this value (leaf references stop at 2^24 triangles).
constexpr uint32_t kDone = 0xFFFFFFFEu;

// With a TLAS the instance tree's entries sit below the geometry's on the
// same stack (at most kStack2 of them: the TLAS is a binary LBVH).
template <int LAYOUT, bool TLAS = false> struct StackDepth
{
  static constexpr int value = (LAYOUT == 0 ? kStack2 : kStack4) + (TLAS ? kStack2 : 0);
};

constexpr uint32_t kTlasMode = 0xFFFFFFFEu;  // Lane::inst while the lane walks the instance tree

// Order in which a launch takes its rays.  With width > 0 the rays form
// row-major images `width` rays wide, and work item i maps to a pixel of a
// tile 4 pixels wide and 8 tall (32 consecutive work items = one warp = one
// tile, tiles row after row): neighbouring pixels trace together.  Index
// arithmetic only; each ray's result still goes to the ray's own index.  (Of
// 32 x 1, 16 x 2, 8 x 4, 8 x 8 and 4 x 8 tiles, 4 x 8 traced the 1920 x 1080
// frame's eye rays fastest.)
struct RayOrder
{
  uint32_t nWork;        // work items (>= rays; tiles that cross the image edge pad it)
  uint32_t width;        // 0: work item i is ray i
  uint32_t tilesPerRow;
  uint32_t perWarp;      // work items of a warp of the one-thread-per-ray kernels (its first lanes)
};

__device__ __forceinline__ uint32_t work_ray(const RayOrder& o, uint32_t i, uint32_t n)
{
  if (o.width == 0) return i < n ? i : kNoRay;
  const uint32_t t = i >> 5, l = i & 31u;
  const uint32_t x = (t % o.tilesPerRow) * 4u + (l & 3u);
  const uint32_t y = (t / o.tilesPerRow) * 8u + (l >> 2);
  if (x >= o.width) return kNoRay;
  const uint64_t r = (uint64_t)y * o.width + x;
  return r < n ? (uint32_t)r : kNoRay;
}

// Work item of a thread of the one-thread-per-ray kernels.
template <int THREADS> __device__ __forceinline__ uint32_t grid_work(const RayOrder& o)
{
  const uint32_t lane = threadIdx.x & 31u;
  return lane < o.perWarp ? (blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5)) * o.perWarp + lane : kNoRay;
}

template <int THREADS> __host__ __forceinline__ uint32_t grid_blocks(const RayOrder& o)
{
  const uint64_t perBlock = (uint64_t)(THREADS / 32) * o.perWarp;
  return (uint32_t)((o.nWork + perBlock - 1) / perBlock);
}

__host__ __forceinline__ RayOrder ray_order(uint32_t n, int width, int perWarp)
{
  RayOrder o{n, 0u, 0u, (uint32_t)perWarp};
  if (width <= 0 || n == 0) return o;
  const uint64_t w = (uint64_t)width;
  const uint64_t tilesPerRow = (w + 3) / 4, rows = (n + w - 1) / w;
  const uint64_t work = tilesPerRow * ((rows + 7) / 8) * 32;
  if (work > 0x7FFFFFFFull) return o;  // too much padding for 32-bit work counters: rays in order
  o.nWork = (uint32_t)work;
  o.width = (uint32_t)w;
  o.tilesPerRow = (uint32_t)tilesPerRow;
  return o;
}

// A lane's traversal stack.
//   kStackShared  the whole depth bound in shared memory, interleaved by thread
//                 (entry k of thread t at sh[k * THREADS])
//   kStackSplit   the first `shared` entries there, the rest in local memory
//   kStackLocal   all of it in local memory, which is cached in L1
constexpr int kStackShared = 0, kStackSplit = 1, kStackLocal = 2;

template <int THREADS, int STACK> struct Stack
{
  uint32_t* sh;
  uint32_t* local;  // entries from `shared` on; unused by kStackShared
  int       shared;
  __device__ __forceinline__ void put(int k, uint32_t v)
  {
    if (STACK == kStackLocal) local[k] = v;
    else if (STACK == kStackShared || k < shared) sh[k * THREADS] = v;
    else local[k - shared] = v;
  }
  __device__ __forceinline__ uint32_t get(int k) const
  {
    if (STACK == kStackLocal) return local[k];
    return (STACK == kStackShared || k < shared) ? sh[k * THREADS] : local[k - shared];
  }
  // Whether `count` entries from k on can be put without a test each.
  __device__ __forceinline__ bool fits(int k, int count) const { return STACK != kStackSplit || k + count <= shared; }
  __device__ __forceinline__ void put_fast(int k, uint32_t v)
  {
    if (STACK == kStackLocal) local[k] = v;
    else sh[k * THREADS] = v;
  }
};

// Shared-memory entries per lane for a requested short-stack size (0 or
// anything at or above the depth bound: the whole stack).
template <int DEPTH> __host__ __device__ __forceinline__ int shared_entries(int requested)
{
  return (requested <= 0 || requested >= DEPTH) ? DEPTH : requested;
}

// Instance tree (TLAS): a binary LBVH over the instances' world-space boxes,
// built like a geometry's tree from one pseudo-triangle per instance; a leaf
// is a run of sorted records whose e1.w holds the instance id.
struct Tlas
{
  const PairRec* recs;  // nullptr: no TLAS, instances are taken in order
  const TriRec*  tris;
  uint32_t       nInst;
};

struct WtRay
{
  int   kx, ky, kz;
  float sx, sy, sz;
};

__device__ __forceinline__ float pick3(float x, float y, float z, int k) { return k == 0 ? x : (k == 1 ? y : z); }

__device__ __forceinline__ void wt_setup(float dx, float dy, float dz, WtRay& w)
{
  const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
  w.kz = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
  w.kx = w.kz == 2 ? 0 : w.kz + 1;
  w.ky = w.kx == 2 ? 0 : w.kx + 1;
  const float dk = pick3(dx, dy, dz, w.kz);
  if (dk < 0.0f)
  {
    const int t = w.kx;
    w.kx = w.ky;
    w.ky = t;
  }
  w.sx = __fdiv_rn(pick3(dx, dy, dz, w.kx), dk);
  w.sy = __fdiv_rn(pick3(dx, dy, dz, w.ky), dk);
  w.sz = __frcp_rn(dk);  // correctly rounded: the value of 1.0f / dk
}

// Two floats in one 64-bit register pair, for the packed FP32 instructions of
// sm_100 (add/mul.rn.f32x2): one issue slot for two operations, each rounded
// exactly as its scalar form.
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float a, float b)
{
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}

__device__ __forceinline__ float2 unpack2(f32x2 v)
{
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
  f32x2 v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
  f32x2 v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
  f32x2 v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}

// A half (the low 16 bits of h) plus a float, converted and added in one
// instruction with one rounding.
__device__ __forceinline__ float add_h(uint32_t h, float c)
{
  float v;
  asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(v) : "h"((unsigned short)h), "f"(c));
  return v;
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
  float v;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
  return v;
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
  float v;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
  return v;
}

// A ray in the frame of the geometry being traversed.  The negated origin
// (no) and the reciprocal direction (inv) are kept as the pairs that the
// layout's packed slab test multiplies by: (x, y), (z, x), (y, z) for the
// binary records, whose boxes are stored as consecutive floats; (x, x), (y, y),
// (z, z) for the 4-wide nodes, where a pair holds one axis of two planes.
// sel[k] is the byte selector that picks the entry plane of axis k (the exit
// plane follows) from a 16-bit or 8-bit node's words: the sign of the
// direction decides it once per ray, instead of a min and a max per box.
// `w` is the watertight test's per-ray set-up; the Moller-Trumbore kernels
// never read it, so the compiler drops its computation there (as it drops sel
// in the FP32 layouts).
template <int LAYOUT> struct Ray
{
  f32x2    no[3], inv[3];
  float    tNear;
  float    dx, dy, dz;
  uint32_t sel[3];
  WtRay    w;
  __device__ __forceinline__ float nox() const { return unpack2(no[0]).x; }
  __device__ __forceinline__ float noy() const { return LAYOUT == 0 ? unpack2(no[0]).y : unpack2(no[1]).x; }
  __device__ __forceinline__ float noz() const { return LAYOUT == 0 ? unpack2(no[1]).x : unpack2(no[2]).x; }
  __device__ __forceinline__ float ix() const { return unpack2(inv[0]).x; }
  __device__ __forceinline__ float iy() const { return LAYOUT == 0 ? unpack2(inv[0]).y : unpack2(inv[1]).x; }
  __device__ __forceinline__ float iz() const { return LAYOUT == 0 ? unpack2(inv[1]).x : unpack2(inv[2]).x; }
};

// SafeInverse, core/raytrace_common.h:57-65.
__device__ __forceinline__ float safe_inv(float d)
{
  const float ooeps = 1.0e-36f;
  return __frcp_rn(fabsf(d) > ooeps ? d : copysignf(ooeps, d));  // correctly rounded, as 1.0f / d
}

template <int LAYOUT>
__device__ __forceinline__ void set_ray(Ray<LAYOUT>& r, float ox, float oy, float oz, float tNear, float dx, float dy,
                                        float dz)
{
  const float ix = safe_inv(dx), iy = safe_inv(dy), iz = safe_inv(dz);
  if (LAYOUT == 0)
  {
    r.no[0] = pack2(-ox, -oy);
    r.no[1] = pack2(-oz, -ox);
    r.no[2] = pack2(-oy, -oz);
    r.inv[0] = pack2(ix, iy);
    r.inv[1] = pack2(iz, ix);
    r.inv[2] = pack2(iy, iz);
  }
  else
  {
    r.no[0] = pack2(-ox, -ox);
    r.no[1] = pack2(-oy, -oy);
    r.no[2] = pack2(-oz, -oz);
    r.inv[0] = pack2(ix, ix);
    r.inv[1] = pack2(iy, iy);
    r.inv[2] = pack2(iz, iz);
  }
  const bool nx = __float_as_int(ix) < 0, ny = __float_as_int(iy) < 0, nz = __float_as_int(iz) < 0;
  if (LAYOUT == 2)
  {
    // halves of (lo.x, lo.y), (lo.z, hi.x), (hi.y, hi.z): (entry, exit) of an
    // axis from the two words that hold its planes
    r.sel[0] = nx ? 0x1076u : 0x7610u;
    r.sel[1] = ny ? 0x3254u : 0x5432u;
    r.sel[2] = nz ? 0x1076u : 0x7610u;
  }
  else if (LAYOUT == 3)
  {
    // the whole word of the four lower or of the four upper bounds
    r.sel[0] = nx ? 0x7654u : 0x3210u;
    r.sel[1] = ny ? 0x7654u : 0x3210u;
    r.sel[2] = nz ? 0x7654u : 0x3210u;
  }
  r.tNear = tNear;
  r.dx = dx;
  r.dy = dy;
  r.dz = dz;
  wt_setup(dx, dy, dz, r.w);
}

// A 32-byte ray or hit record: one 256-bit access when the record is 32-byte
// aligned (sm_100 and later), else two 128-bit ones.  A warp's 32 records are
// then one contiguous kilobyte per instruction, which matters most for arrays
// read and written in place over the host link.
__device__ __forceinline__ void load_record(const float4* __restrict__ p, float4& a, float4& b)
{
  if ((reinterpret_cast<uintptr_t>(p) & 31u) == 0u)
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
  else
  {
    a = __ldg(p);
    b = __ldg(p + 1);
  }
}

__device__ __forceinline__ void store_record(float4* p, const float4& a, const float4& b)
{
  if ((reinterpret_cast<uintptr_t>(p) & 31u) == 0u)
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
  else
  {
    p[0] = a;
    p[1] = b;
  }
}

struct Hit
{
  float    t, u, v;
  uint32_t prim, inst;  // sorted triangle, instance index (0xFFFFFFFF: no hit)
};

// matmul4x3 / matmul3x3 (core/raytrace_common.h:82-90) with the column sum
// order ((m0*x + m1*y) + m2*z) + m3*w.
__device__ __forceinline__ float row_dot(const float* m, float x, float y, float z, float w)
{
  return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], x), __fmul_rn(m[1], y)), __fmul_rn(m[2], z)), __fmul_rn(m[3], w));
}

template <int LAYOUT>
__device__ __forceinline__ void make_ray(const InstanceDesc& d, const float4& po, const float4& di, Ray<LAYOUT>& r)
{
  if (d.identity)
    set_ray(r, po.x, po.y, po.z, po.w, di.x, di.y, di.z);
  else
    set_ray(r, row_dot(d.inv + 0, po.x, po.y, po.z, 1.0f), row_dot(d.inv + 4, po.x, po.y, po.z, 1.0f),
            row_dot(d.inv + 8, po.x, po.y, po.z, 1.0f), po.w, row_dot(d.inv + 0, di.x, di.y, di.z, 0.0f),
            row_dot(d.inv + 4, di.x, di.y, di.z, 0.0f), row_dot(d.inv + 8, di.x, di.y, di.z, 0.0f));
}

// Moller-Trumbore leaf test over the leaf starting at sorted triangle j
// (IntersectAllPrimitivesInLeaf, core/BVH2CommonRT.cpp:9-47); the leaf ends at
// the record whose flags have ENDBIT set (1: binary leaf, 2: 4-wide leaf).
// Returns true when ANY and a triangle was accepted.
template <bool ANY, bool COUNT, uint32_t ENDBIT, int LAYOUT>
__device__ __forceinline__ bool leaf_test(const TriRec* __restrict__ tris, uint32_t j, const Ray<LAYOUT>& r, Hit& h,
                                          uint32_t instIndex, uint64_t& nTris)
{
  while (true)
  {
    const float4* q = reinterpret_cast<const float4*>(tris + j);
    const float4 A = __ldg(q + 0);
    const float4 e1 = __ldg(q + 1);
    const float4 e2 = __ldg(q + 2);
    if (COUNT) nTris++;
    // pvec = cross(dir, e2), tvec = pos - A, qvec = cross(tvec, e1)
    const float px = __fsub_rn(__fmul_rn(r.dy, e2.z), __fmul_rn(r.dz, e2.y));
    const float py = __fsub_rn(__fmul_rn(r.dz, e2.x), __fmul_rn(r.dx, e2.z));
    const float pz = __fsub_rn(__fmul_rn(r.dx, e2.y), __fmul_rn(r.dy, e2.x));
    const float tx = __fsub_rn(-r.nox(), A.x);
    const float ty = __fsub_rn(-r.noy(), A.y);
    const float tz = __fsub_rn(-r.noz(), A.z);
    const float qx = __fsub_rn(__fmul_rn(ty, e1.z), __fmul_rn(tz, e1.y));
    const float qy = __fsub_rn(__fmul_rn(tz, e1.x), __fmul_rn(tx, e1.z));
    const float qz = __fsub_rn(__fmul_rn(tx, e1.y), __fmul_rn(ty, e1.x));
    const float det = __fadd_rn(__fadd_rn(__fmul_rn(e1.x, px), __fmul_rn(e1.y, py)), __fmul_rn(e1.z, pz));
    const float invDet = __frcp_rn(det);  // correctly rounded: the value of 1.0f / det
    const float v = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(tx, px), __fmul_rn(ty, py)), __fmul_rn(tz, pz)), invDet);
    const float u = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(qx, r.dx), __fmul_rn(qy, r.dy)), __fmul_rn(qz, r.dz)), invDet);
    const float t = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(e2.x, qx), __fmul_rn(e2.y, qy)), __fmul_rn(e2.z, qz)), invDet);
    // 1.0f + 1e-6f rounds to 1 + 2^-20 in binary32
    if (v >= -1e-6f && u >= -1e-6f && __fadd_rn(u, v) <= 0x1.00001p+0f && t > r.tNear && t < h.t)
    {
      h.t = t;
      h.u = u;
      h.v = v;
      h.prim = j;
      h.inst = instIndex;
      if (ANY) return true;
    }
    if (__float_as_uint(A.w) & ENDBIT) return false;  // last triangle of the leaf
    j++;
  }
}

// ------------------------------------------------------- watertight triangle test
// Woop, Benthin & Wald, "Watertight Ray/Triangle Intersection", JCGT 2(1),
// 2013: the ray's dominant axis becomes z (kx, ky keep the winding), the
// triangle is translated to the ray origin and sheared so that the ray runs
// along +z, and the signs of the three 2D edge functions at the origin decide
// the hit (both windings accepted).  The paper re-evaluates an edge function
// in double precision when it comes out zero; here each one is Kahan's
// difference of products (the rounding error of one product recovered by an
// FMA), whose relative error stays below 2 ulp, so its sign is exact in FP32
// and the test needs no FP64.  An edge shared by two triangles then gets
// exactly opposite signs on both sides: no ray passes between them.  Records
// hold the vertices {A, B, C} (w: flags, triangle id, 0).  Outputs match the
// Moller-Trumbore fields: u = the weight of C, v = the weight of B.
// a*b - c*d with the rounding error of c*d restored (Kahan).
__device__ __forceinline__ float diff_of_products(float a, float b, float c, float d)
{
  const float w = __fmul_rn(c, d);
  const float e = __fmaf_rn(-c, d, w);
  const float f = __fmaf_rn(a, b, -w);
  return __fadd_rn(f, e);
}

template <bool ANY, bool COUNT, uint32_t ENDBIT, int LAYOUT>
__device__ __forceinline__ bool leaf_test_wt(const TriRec* __restrict__ tris, uint32_t j, const Ray<LAYOUT>& r, Hit& h,
                                             uint32_t instIndex, uint64_t& nTris)
{
  const WtRay& w = r.w;
  while (true)
  {
    const float4* q = reinterpret_cast<const float4*>(tris + j);
    const float4 A = __ldg(q + 0);
    const float4 B = __ldg(q + 1);
    const float4 Cv = __ldg(q + 2);
    if (COUNT) nTris++;
    const float a0 = __fadd_rn(A.x, r.nox()), a1 = __fadd_rn(A.y, r.noy()), a2 = __fadd_rn(A.z, r.noz());
    const float b0 = __fadd_rn(B.x, r.nox()), b1 = __fadd_rn(B.y, r.noy()), b2 = __fadd_rn(B.z, r.noz());
    const float c0 = __fadd_rn(Cv.x, r.nox()), c1 = __fadd_rn(Cv.y, r.noy()), c2 = __fadd_rn(Cv.z, r.noz());
    const float az = pick3(a0, a1, a2, w.kz), bz = pick3(b0, b1, b2, w.kz), cz = pick3(c0, c1, c2, w.kz);
    const float ax = __fsub_rn(pick3(a0, a1, a2, w.kx), __fmul_rn(w.sx, az));
    const float ay = __fsub_rn(pick3(a0, a1, a2, w.ky), __fmul_rn(w.sy, az));
    const float bx = __fsub_rn(pick3(b0, b1, b2, w.kx), __fmul_rn(w.sx, bz));
    const float by = __fsub_rn(pick3(b0, b1, b2, w.ky), __fmul_rn(w.sy, bz));
    const float cx = __fsub_rn(pick3(c0, c1, c2, w.kx), __fmul_rn(w.sx, cz));
    const float cy = __fsub_rn(pick3(c0, c1, c2, w.ky), __fmul_rn(w.sy, cz));
    const float U = diff_of_products(cx, by, cy, bx);
    const float V = diff_of_products(ax, cy, ay, cx);
    const float W = diff_of_products(bx, ay, by, ax);
    const bool outside = (U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f);
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (!outside && det != 0.0f)
    {
      const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, __fmul_rn(w.sz, az)), __fmul_rn(V, __fmul_rn(w.sz, bz))),
                                __fmul_rn(W, __fmul_rn(w.sz, cz)));
      const float inv = __frcp_rn(det);
      const float t = __fmul_rn(T, inv);
      if (t > r.tNear && t < h.t)
      {
        h.t = t;
        h.u = __fmul_rn(W, inv);
        h.v = __fmul_rn(V, inv);
        h.prim = j;
        h.inst = instIndex;
        if (ANY) return true;
      }
    }
    if (__float_as_uint(A.w) & ENDBIT) return false;  // last triangle of the leaf
    j++;
  }
}

// The scene's triangle test: 0 Moller-Trumbore (the reference's), 1 watertight.
template <int TRI, bool ANY, bool COUNT, uint32_t ENDBIT, int LAYOUT>
__device__ __forceinline__ bool test_leaf(const TriRec* __restrict__ tris, uint32_t j, const Ray<LAYOUT>& r, Hit& h,
                                          uint32_t instIndex, uint64_t& nTris)
{
  if constexpr (TRI == 1) return leaf_test_wt<ANY, COUNT, ENDBIT>(tris, j, r, h, instIndex, nTris);
  else return leaf_test<ANY, COUNT, ENDBIT>(tris, j, r, h, instIndex, nTris);
}

// ---------------------------------------------------------------- 4-wide nodes
// A 32-byte piece of a node or pair record: one 256-bit read-only load.  The
// node arrays start at an allocation's boundary and their records are 64 or
// 128 bytes, so the pieces are aligned.
__device__ __forceinline__ void load_piece(const void* p, f32x2 (&v)[4])
{
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
}

__device__ __forceinline__ void load_piece(const void* p, uint32_t (&v)[8])
{
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "l"(p));
}

// Entry and exit distances of the four child boxes (RayBoxIntersection2,
// core/raytrace_common.h:67-80: the differences, products and their rounding
// are the reference's; min and max as explained above) and the child
// references.
//
// Where the entry plane is picked by the direction's sign: with 1/d > 0 the
// product of the lower plane is the smaller one, since subtraction and
// multiplication round monotonically, so picking is the min and max of the two
// products (up to the sign of a zero).
__device__ __forceinline__ void slabs4(const Ray<1>& r, const Node4F32* __restrict__ n, float (&tn)[4], float (&tf)[4],
                                       uint4& ref)
{
  const char* p = reinterpret_cast<const char*>(n);
  f32x2 a[4], b[4], c[4];  // lo.x lo.y | lo.z hi.x | hi.y hi.z, each of the children (0, 1), (2, 3)
  load_piece(p, a);
  load_piece(p + 32, b);
  load_piece(p + 64, c);
  ref = __ldg(reinterpret_cast<const uint4*>(p + 96));
#pragma unroll
  for (int q = 0; q < 2; q++)
  {
    const float2 lx = unpack2(mul2(r.inv[0], add2(a[q], r.no[0]))), hx = unpack2(mul2(r.inv[0], add2(b[2 + q], r.no[0])));
    const float2 ly = unpack2(mul2(r.inv[1], add2(a[2 + q], r.no[1]))), hy = unpack2(mul2(r.inv[1], add2(c[q], r.no[1])));
    const float2 lz = unpack2(mul2(r.inv[2], add2(b[q], r.no[2]))), hz = unpack2(mul2(r.inv[2], add2(c[2 + q], r.no[2])));
    tn[2 * q] = max3(fminf(lx.x, hx.x), fminf(ly.x, hy.x), fminf(lz.x, hz.x));
    tf[2 * q] = min3(fmaxf(lx.x, hx.x), fmaxf(ly.x, hy.x), fmaxf(lz.x, hz.x));
    tn[2 * q + 1] = max3(fminf(lx.y, hx.y), fminf(ly.y, hy.y), fminf(lz.y, hz.y));
    tf[2 * q + 1] = min3(fmaxf(lx.y, hx.y), fmaxf(ly.y, hy.y), fmaxf(lz.y, hz.y));
  }
}

// FP16: a byte permute gathers (entry, exit) of one axis of a child into one
// word; each half is converted and subtracted in one mixed-precision add
// (against a conversion and half a packed add: 3 to 5% less time on nearest
// hits of 500,000 random rays into 500,000 triangles).
__device__ __forceinline__ void slabs4(const Ray<2>& r, const Node4F16* __restrict__ n, float (&tn)[4], float (&tf)[4],
                                       uint4& ref)
{
  const char* p = reinterpret_cast<const char*>(n);
  uint32_t u[8], v[8];
  load_piece(p, u);
  load_piece(p + 32, v);
  ref = make_uint4(v[4], v[5], v[6], v[7]);
#pragma unroll
  for (int k = 0; k < 4; k++)
  {
    const uint32_t X = __byte_perm(u[k], u[4 + k], r.sel[0]);
    const uint32_t Y = __byte_perm(u[k], v[k], r.sel[1]);
    const uint32_t Z = __byte_perm(u[4 + k], v[k], r.sel[2]);
    const float2 x = unpack2(mul2(r.inv[0], pack2(add_h(X & 0xFFFF, r.nox()), add_h(X >> 16, r.nox()))));
    const float2 y = unpack2(mul2(r.inv[1], pack2(add_h(Y & 0xFFFF, r.noy()), add_h(Y >> 16, r.noy()))));
    const float2 z = unpack2(mul2(r.inv[2], pack2(add_h(Z & 0xFFFF, r.noz()), add_h(Z >> 16, r.noz()))));
    tn[k] = max3(x.x, y.x, z.x);
    tf[k] = min3(x.y, y.y, z.y);
  }
}

// Bytes q and q + 1 of w as floats: the byte in the mantissa of 2^23, minus
// 2^23 (both exact).
template <int Q> __device__ __forceinline__ f32x2 bytes2(uint32_t w)
{
  const f32x2 v = pack2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | Q)),
                        __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | (Q + 1))));
  return add2(v, pack2(-8388608.0f, -8388608.0f));
}

// 8-bit: the entry planes' word of each axis is picked whole (four children),
// then bound = origin + q * 2^e (the product is exact, so one fused add
// rounds like the encoder's add).
__device__ __forceinline__ void slabs4(const Ray<3>& r, const Node4Q8* __restrict__ n, float (&tn)[4], float (&tf)[4],
                                       uint4& ref)
{
  const char* p = reinterpret_cast<const char*>(n);
  uint32_t u[8], v[8];  // frame (4), lo.x lo.y lo.z hi.x | hi.y hi.z - -, refs (4)
  load_piece(p, u);
  load_piece(p + 32, v);
  ref = make_uint4(v[4], v[5], v[6], v[7]);
  const uint32_t lo[3] = {u[4], u[5], u[6]}, hi[3] = {u[7], v[0], v[1]};
  float2 t0[3][2], t1[3][2];  // [axis][children (0, 1) / (2, 3)] entry, exit
#pragma unroll
  for (int c = 0; c < 3; c++)
  {
    const float sc = __uint_as_float((((u[3] >> (8 * c)) & 0xFFu) - 1u) << 23);
    const f32x2 sc2 = pack2(sc, sc), org = pack2(__uint_as_float(u[c]), __uint_as_float(u[c]));
    const uint32_t en = __byte_perm(lo[c], hi[c], r.sel[c]), ex = __byte_perm(hi[c], lo[c], r.sel[c]);
    t0[c][0] = unpack2(mul2(r.inv[c], add2(fma2(bytes2<0>(en), sc2, org), r.no[c])));
    t0[c][1] = unpack2(mul2(r.inv[c], add2(fma2(bytes2<2>(en), sc2, org), r.no[c])));
    t1[c][0] = unpack2(mul2(r.inv[c], add2(fma2(bytes2<0>(ex), sc2, org), r.no[c])));
    t1[c][1] = unpack2(mul2(r.inv[c], add2(fma2(bytes2<2>(ex), sc2, org), r.no[c])));
  }
#pragma unroll
  for (int q = 0; q < 2; q++)
  {
    tn[2 * q] = max3(t0[0][q].x, t0[1][q].x, t0[2][q].x);
    tf[2 * q] = min3(t1[0][q].x, t1[1][q].x, t1[2][q].x);
    tn[2 * q + 1] = max3(t0[0][q].y, t0[1][q].y, t0[2][q].y);
    tf[2 * q + 1] = min3(t1[0][q].y, t1[1][q].y, t1[2][q].y);
  }
}

template <int LAYOUT> struct Node4Type;
template <> struct Node4Type<1> { using type = Node4F32; };
template <> struct Node4Type<2> { using type = Node4F16; };
template <> struct Node4Type<3> { using type = Node4Q8; };

__device__ __forceinline__ void cswap(float& ka, uint32_t& va, float& kb, uint32_t& vb)
{
  const bool s = kb < ka;
  const float tk = s ? kb : ka;
  const uint32_t tv = s ? vb : va;
  kb = s ? ka : kb;
  vb = s ? va : vb;
  ka = tk;
  va = tv;
}

// Per-lane traversal state.
template <int LAYOUT> struct Lane
{
  Ray<LAYOUT> r;
  Hit      h;
  float4   po, di;    // the ray as given (world space)
  uint32_t ray;       // ray index or kNoRay
  uint32_t inst;      // current instance
  const void*   nodes;  // the current instance's records (binary) or 4-wide nodes
  const TriRec* tris;   // the current instance's triangle records
  uint32_t cur;       // current record / leaf reference
  int      top;       // stack depth
  int      base;      // stack depth at which the current instance's traversal began
  uint32_t tnext;     // next record of the current TLAS leaf run, or kNoRay
  bool     stale;     // r is not the world-space ray (an instance was entered)
  uint32_t budget;    // steps left for this ray
};

// Upper bound on the steps of one ray: far above any real traversal (a ray
// visits each node at most once per instance); reaching it means a broken
// tree, and the ray ends as a miss with kErrStepBudget instead of looping.
constexpr uint32_t kStepBudget = 1u << 24;

// The first lane to run out of budget records its state after the error word:
// [1] = 1 (taken), [2] ray, [3] current ref, [4] stack depth.
template <typename LaneT>
__device__ __forceinline__ bool out_of_budget(LaneT& L, uint32_t* errorWord)
{
  if (L.budget-- != 0u) return false;
  atomicOr(errorWord, kErrStepBudget);
  if (atomicCAS(errorWord + 1, 0u, 1u) == 0u)
  {
    errorWord[2] = L.ray;
    errorWord[3] = L.cur;
    errorWord[4] = (uint32_t)L.top;
  }
  return true;
}

// Makes instance k the lane's current instance: its ray, and its node and
// triangle arrays held in registers for the steps that follow.
template <int LAYOUT>
__device__ __forceinline__ void enter_instance(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, uint32_t k)
{
  const InstanceDesc& d = inst[k];
  L.inst = k;
  make_ray(d, L.po, L.di, L.r);
  L.nodes = LAYOUT == 0 ? static_cast<const void*>(d.recs) : d.nodes4;
  L.tris = d.tris;
  L.cur = 0;  // record / node 0 = the root
}

// Advances the lane's instance cursor to the next instance with triangles,
// starting at `from`; prepares the ray for it.  Returns false when none is left.
template <int LAYOUT>
__device__ __forceinline__ bool begin_instance(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, uint32_t nInst,
                                               uint32_t from)
{
  for (uint32_t k = from; k < nInst; k++)
    if (inst[k].valid)
    {
      enter_instance<LAYOUT>(L, inst, k);
      L.top = 0;
      L.base = 0;
      return true;
    }
  return false;
}

template <int LAYOUT> struct EndBit
{
  static constexpr uint32_t value = LAYOUT == 0 ? 1u : 2u;  // flag bit that ends a leaf of this layout
};

// min and max of which either gives NaN when an operand is NaN.
__device__ __forceinline__ float max_or_nan(float a, float b)
{
  float v;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(v) : "f"(a), "f"(b));
  return v;
}

__device__ __forceinline__ float min_or_nan(float a, float b)
{
  float v;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(v) : "f"(a), "f"(b));
  return v;
}

// A box is entered when its interval meets the ray's: tn <= tf, tf >= tNear,
// tn <= t (core/raytrace_common.h:67-80).  Taken as one comparison of the
// clamped ends, which also asks tNear <= t: without that no triangle can be
// accepted (a ray whose tFar lies before its tNear ends at the root), so only
// the counting kernels, whose visits are the reference's, compare one by one.
// Each of those comparisons fails on a NaN, and so does this one: the ends keep
// a NaN operand (a ray without a number for its origin, tNear or t ends at the
// root; with a min and max that drop it, it walked the whole tree).
template <bool COUNT> __device__ __forceinline__ bool box_hit(float tn, float tf, float tNear, float t)
{
  if (COUNT) return tn <= tf && tf >= tNear && tn <= t;
  return max_or_nan(tn, tNear) <= min_or_nan(tf, t);
}

// Visits the internal node L.cur: tests its children, continues with the
// nearest hit child (child 0 on equal entry distance) and pushes the others,
// farthest first.  Returns 1 when no child is hit (the caller pops), 0
// otherwise, -1 when the stack bound would be exceeded (reported).
// One child pair of a binary tree: BVH2TraverseC32's decisions
// (core/BVH2CommonRT.cpp:88-113).
template <bool COUNT, int THREADS, int DEPTH, int STACK, int LAYOUT, typename LaneT>
__device__ __forceinline__ int visit_pair(LaneT& L, const Ray<LAYOUT>& r, const PairRec* __restrict__ recs,
                                          Stack<THREADS, STACK>& st, uint64_t& nPairs, uint32_t* errorWord)
{
  const char* p = reinterpret_cast<const char*>(recs + L.cur);
  f32x2 a[4], b[4];  // L.min L.max R.min | R.max refs, six floats a box
  load_piece(p, a);
  load_piece(p + 32, b);
  if (COUNT) nPairs++;
  float t0n, t0f, t1n, t1f;
  if constexpr (LAYOUT == 0)
  {
    const float2 p0 = unpack2(mul2(r.inv[0], add2(a[0], r.no[0]))), p1 = unpack2(mul2(r.inv[1], add2(a[1], r.no[1]))),
                 p2 = unpack2(mul2(r.inv[2], add2(a[2], r.no[2])));
    t0n = max3(fminf(p0.x, p1.y), fminf(p0.y, p2.x), fminf(p1.x, p2.y));
    t0f = min3(fmaxf(p0.x, p1.y), fmaxf(p0.y, p2.x), fmaxf(p1.x, p2.y));
    const float2 q0 = unpack2(mul2(r.inv[0], add2(a[3], r.no[0]))), q1 = unpack2(mul2(r.inv[1], add2(b[0], r.no[1]))),
                 q2 = unpack2(mul2(r.inv[2], add2(b[1], r.no[2])));
    t1n = max3(fminf(q0.x, q1.y), fminf(q0.y, q2.x), fminf(q1.x, q2.y));
    t1f = min3(fmaxf(q0.x, q1.y), fmaxf(q0.y, q2.x), fmaxf(q1.x, q2.y));
  }
  else
  {
    // the same from a ray kept for 4-wide nodes: the pairs are (min, max) of an axis
    const float2 m0 = unpack2(a[0]), m1 = unpack2(a[1]), m2 = unpack2(a[2]);
    const float2 n0 = unpack2(a[3]), n1 = unpack2(b[0]), n2 = unpack2(b[1]);
    const float2 x0 = unpack2(mul2(r.inv[0], add2(pack2(m0.x, m1.y), r.no[0]))),
                 y0 = unpack2(mul2(r.inv[1], add2(pack2(m0.y, m2.x), r.no[1]))),
                 z0 = unpack2(mul2(r.inv[2], add2(pack2(m1.x, m2.y), r.no[2])));
    t0n = max3(fminf(x0.x, x0.y), fminf(y0.x, y0.y), fminf(z0.x, z0.y));
    t0f = min3(fmaxf(x0.x, x0.y), fmaxf(y0.x, y0.y), fmaxf(z0.x, z0.y));
    const float2 x1 = unpack2(mul2(r.inv[0], add2(pack2(n0.x, n1.y), r.no[0]))),
                 y1 = unpack2(mul2(r.inv[1], add2(pack2(n0.y, n2.x), r.no[1]))),
                 z1 = unpack2(mul2(r.inv[2], add2(pack2(n1.x, n2.y), r.no[2])));
    t1n = max3(fminf(x1.x, x1.y), fminf(y1.x, y1.y), fminf(z1.x, z1.y));
    t1f = min3(fmaxf(x1.x, x1.y), fmaxf(y1.x, y1.y), fmaxf(z1.x, z1.y));
  }
  const float2 ref = unpack2(b[2]);
  const uint32_t ref0 = __float_as_uint(ref.x), ref1 = __float_as_uint(ref.y);
  const bool h0 = box_hit<COUNT>(t0n, t0f, r.tNear, L.h.t);
  const bool h1 = box_hit<COUNT>(t1n, t1f, r.tNear, L.h.t);
  if (!h0 && !h1) return 1;
  const bool first0 = h0 && (!h1 || t0n <= t1n);
  L.cur = first0 ? ref0 : ref1;
  if (h0 && h1)
  {
    if (L.top >= DEPTH)
    {
      atomicOr(errorWord, kErrStack);
      return -1;
    }
    st.put(L.top, first0 ? ref1 : ref0);
    L.top++;
  }
  return 0;
}

template <int LAYOUT, bool ANY, bool COUNT, int THREADS, int DEPTH, int STACK, typename LaneT>
__device__ __forceinline__ int visit_node(LaneT& L, Stack<THREADS, STACK>& st, uint64_t& nPairs, uint32_t* errorWord)
{
  if constexpr (LAYOUT != 0)
  {
    // 4-wide node: HeavyRT's BVH4 order (core/BVH4CommonRT.cpp:49-246).  An
    // unused slot (kEmptyRef; its box is a point: 0, or the corner of an 8-bit
    // node's frame) may pass the test for a ray through that point.  For any
    // hits it then counts as a leaf without triangles.  Nearest hits leave it
    // out: the network that sorts the children is not stable, so one key more
    // can swap children of equal entry distance, and with them the triangle
    // that a ray through a shared edge reports.  Slot 1 may be unused only in
    // the node of a lone leaf, where nothing can be swapped.
    using N = typename Node4Type<LAYOUT>::type;
    float key[4], tf[4];
    uint4 r4;
    slabs4(L.r, reinterpret_cast<const N*>(L.nodes) + L.cur, key, tf, r4);
    if (COUNT) nPairs++;
    uint32_t ref[4] = {r4.x, r4.y, r4.z, r4.w};
    bool hit[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      hit[k] = box_hit<COUNT>(key[k], tf[k], L.r.tNear, L.h.t) && (ANY || k < 2 || ref[k] != kEmptyRef);
    // at most three pushes; near the stack's bound they are counted first
    if (L.top > DEPTH - 3 && L.top + (int)hit[0] + (int)hit[1] + (int)hit[2] + (int)hit[3] - 1 > DEPTH)
    {
      int used = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) used += hit[k] && ref[k] != kEmptyRef;
      if (L.top + used - 1 > DEPTH)
      {
        atomicOr(errorWord, kErrStack);
        return -1;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) hit[k] = hit[k] && ref[k] != kEmptyRef;
    }
    if constexpr (ANY)
    {
      // any hit: the answer does not depend on the visit order, so the hit
      // children are taken in slot order without sorting; what is pushed
      // follows from the hits alone (2M occlusion rays, FP16 nodes 383 -> 375
      // us against asking each reference; leaves before nodes 407)
      const bool any1 = hit[0], any2 = any1 || hit[1], any3 = any2 || hit[2];
      if (!any3 && !hit[3]) return 1;
      if (st.fits(L.top, 3))
      {
        if (hit[3] && any3) st.put_fast(L.top++, ref[3]);
        if (hit[2] && any2) st.put_fast(L.top++, ref[2]);
        if (hit[1] && any1) st.put_fast(L.top++, ref[1]);
      }
      else
      {
        if (hit[3] && any3) st.put(L.top++, ref[3]);
        if (hit[2] && any2) st.put(L.top++, ref[2]);
        if (hit[1] && any1) st.put(L.top++, ref[1]);
      }
      L.cur = hit[0] ? ref[0] : hit[1] ? ref[1] : hit[2] ? ref[2] : ref[3];
      return 0;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) key[k] = hit[k] ? key[k] : INFINITY;
    cswap(key[0], ref[0], key[1], ref[1]);
    cswap(key[2], ref[2], key[3], ref[3]);
    cswap(key[0], ref[0], key[2], ref[2]);
    cswap(key[1], ref[1], key[3], ref[3]);
    cswap(key[1], ref[1], key[2], ref[2]);
    if (key[0] == INFINITY) return 1;
    L.cur = ref[0];
    if (st.fits(L.top, 3))
    {
#pragma unroll
      for (int k = 3; k >= 1; k--)
        if (key[k] < INFINITY) st.put_fast(L.top++, ref[k]);
    }
    else
    {
#pragma unroll
      for (int k = 3; k >= 1; k--)
        if (key[k] < INFINITY) st.put(L.top++, ref[k]);
    }
    return 0;
  }
  else
    return visit_pair<COUNT, THREADS, DEPTH, STACK, LAYOUT>(L, L.r, reinterpret_cast<const PairRec*>(L.nodes), st,
                                                            nPairs, errorWord);
}

// Ray of the lane in world space (the instance tree is not transformed).
template <int LAYOUT> __device__ __forceinline__ void world_ray(Lane<LAYOUT>& L)
{
  set_ray(L.r, L.po.x, L.po.y, L.po.z, L.po.w, L.di.x, L.di.y, L.di.z);
}

template <int LAYOUT> __device__ __forceinline__ void tlas_begin(Lane<LAYOUT>& L)
{
  L.inst = kTlasMode;
  world_ray(L);
  L.cur = 0;
  L.top = 0;
  L.base = 0;
  L.tnext = kNoRay;
  L.stale = false;
}

// Node visits that a lane may make in one advance before its leaf.  A warp
// whose lanes alternate freely between nodes and leaves runs both paths in
// nearly every step, the leaf path for a few lanes only; a run of nodes first
// gathers more lanes at leaves, but lanes that reach a leaf early wait.  Binary
// leaves are rare (one visit in twenty), so the run is long; any-hit rays end
// at a leaf, so theirs is short.  Measured, us: one node and one leaf at most
// per step against this: 4M occlusion rays, FP16 nodes 632 -> 580 (runs of 3
// and 4: 597, 628); 1M random rays, 8-bit nodes 1,646 -> 1,482 (runs of 2 and
// 4: 1,587, 1,530); full-HD eye rays, binary 255 -> 215 (a run of 4: 217).
// Watertight any hits are faster at 3 in 4-wide trees (1M random rays, 20,000
// triangles, 8-bit nodes 617 -> 583, FP16 506 -> 479), and one thread per ray
// in binary ones at 2 (100,000 rays, 20,000 and 500,000 triangles 165 and 438
// us at 6, 141 and 349 at 2, 153 and 364 at 1; in the pool 6 and 2 are even).
template <int LAYOUT, int TRI, bool ANY, bool GRID> struct NodeRun
{
  static constexpr bool wt = TRI == 1 && ANY;
  static constexpr int  value = LAYOUT == 0 ? (wt && GRID ? 2 : 6) : (ANY && !wt ? 2 : 3);
};

// Stride of the pools' step loops.  It changes nothing but the registers that
// the compiler finds (500,000 random rays, binary, watertight: 784 us at 1,
// 694 at the run's length; FP16 nodes, Moller-Trumbore: 501 at 1, 523).
template <int LAYOUT> struct PoolStep
{
  static constexpr int value = LAYOUT == 0 ? 6 : 1;
};

// One advance of a lane that walks its instances in order: nodes, then a leaf
// when it holds one.  Returns true when the lane's ray is finished.
template <bool GRID, int LAYOUT, int TRI, bool ANY, bool COUNT, int THREADS, int STACK>
__device__ __forceinline__ bool step(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, uint32_t nInst,
                                     Stack<THREADS, STACK>& st, uint64_t& nPairs, uint64_t& nTris, uint32_t* errorWord)
{
  constexpr int DEPTH = StackDepth<LAYOUT, false>::value;
  auto leave = [&]() {
    if (L.top == 0) return !begin_instance<LAYOUT>(L, inst, nInst, L.inst + 1);
    L.top--;
    L.cur = st.get(L.top);
    return false;
  };
#pragma unroll 1
  for (int k = 0; k < NodeRun<LAYOUT, TRI, ANY, GRID>::value; k++)
  {
    if ((L.cur & kLeafBit) != 0u) break;
    const int r = visit_node<LAYOUT, ANY, COUNT, THREADS, DEPTH, STACK>(L, st, nPairs, errorWord);
    if (r < 0) return true;
    if (r == 1 && leave()) return true;
  }
  if ((L.cur & kLeafBit) != 0u)
  {
    if (L.cur != kEmptyRef &&
        test_leaf<TRI, ANY, COUNT, EndBit<LAYOUT>::value>(L.tris, L.cur & ~kLeafBit, L.r, L.h, L.inst, nTris))
      return true;  // any-hit found
    return leave();
  }
  return false;
}

// The instance tree's walk: what a lane does next.
//   tree   visit a pair of instance boxes
//   enter  take the next instance of a leaf of the tree (L.cur = kLeafBit |
//          its record), or put the ray back into world space (L.stale)
//   node, leaf   of the instance entered
// Pops the stack to an entry of the instance tree, or ends the ray.
template <int LAYOUT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_pop(Lane<LAYOUT>& L, const Stack<THREADS, STACK>& st)
{
  if (L.top == 0) L.cur = kDone;
  else
  {
    L.top--;
    L.cur = st.get(L.top);
  }
}

// Leaves the current instance: the next record of the tree's leaf, or the tree.
template <int LAYOUT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_leave(Lane<LAYOUT>& L, const Stack<THREADS, STACK>& st)
{
  L.inst = kTlasMode;
  if (L.tnext != kNoRay) L.cur = kLeafBit | L.tnext;
  else tlas_pop(L, st);
}

template <int LAYOUT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_enter(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, const Tlas& tl,
                                           const Stack<THREADS, STACK>& st)
{
  if ((L.cur & kLeafBit) == 0u)
  {
    world_ray(L);
    L.stale = false;
    return;
  }
  if (L.cur == kEmptyRef)
  {
    tlas_pop(L, st);
    return;
  }
  const uint32_t j = L.cur & ~kLeafBit;
  const float4* q = reinterpret_cast<const float4*>(tl.tris + j);
  const uint32_t flags = __float_as_uint(__ldg(q).w);
  const uint32_t k = __float_as_uint(__ldg(q + 1).w);
  L.tnext = (flags & 1u) ? kNoRay : j + 1;
  if (k < tl.nInst && inst[k].valid)
  {
    enter_instance<LAYOUT>(L, inst, k);
    L.base = L.top;
    L.stale = true;
  }
  else
    tlas_leave(L, st);
}

// Visits that a lane may make in one phase (921,600 rays, 240 instances, FP32
// nodes: (1, 2), (2, 1), (2, 2), (4, 2), (2, 4) node and tree visits 1,239,
// 1,219, 1,193, 1,177, 1,169 us).
constexpr int kTlasNodeRun = 2, kTlasTreeRun = 4;
// The same for a lane that walks without a vote, one thread per ray and in the
// pool (63,000 rays into 100 instances, FP16 nodes, one thread per ray, (node,
// tree) runs of (1, 1), (2, 1), (3, 1), (4, 2), (6, 6): 737, 683, 673, 755, 757
// us; 170,000 rays in the pool 972, 1,005, 1,091, 950, 994).
constexpr int kGridNodeRun = 3, kGridTreeRun = 1, kAloneNodeRun = 4, kAloneTreeRun = 2;

// The walk of a two-level tree has four kinds of work.  tlas_walk_* do the one
// that the lane waits for (as `state` of it says).
struct TlasState
{
  bool tree, enter, node, leaf;
};
template <int LAYOUT> __device__ __forceinline__ TlasState tlas_state(const Lane<LAYOUT>& L)
{
  const bool live = L.cur != kDone, inTree = L.inst == kTlasMode, leaf = (L.cur & kLeafBit) != 0u;
  const bool enter = live && inTree && (leaf || L.stale);
  return {live && inTree && !enter, enter, live && !inTree && !leaf, live && !inTree && leaf};
}

template <int RUN, int LAYOUT, bool ANY, bool COUNT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_walk_nodes(Lane<LAYOUT>& L, Stack<THREADS, STACK>& st, uint64_t& nPairs,
                                                uint32_t* errorWord)
{
  constexpr int DEPTH = StackDepth<LAYOUT, true>::value;
  if (out_of_budget(L, errorWord)) L.cur = kDone;
#pragma unroll 1
  for (int k = 0; k < RUN && (L.cur & kLeafBit) == 0u; k++)
  {
    const int r = visit_node<LAYOUT, ANY, COUNT, THREADS, DEPTH, STACK>(L, st, nPairs, errorWord);
    if (r < 0) L.cur = kDone;
    else if (r == 1)
    {
      if (L.top > L.base)
      {
        L.top--;
        L.cur = st.get(L.top);
      }
      else
      {
        tlas_leave(L, st);
        break;
      }
    }
  }
}

template <int RUN, int LAYOUT, bool COUNT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_walk_tree(Lane<LAYOUT>& L, const Tlas& tl, Stack<THREADS, STACK>& st,
                                               uint64_t& nPairs, uint32_t* errorWord)
{
  constexpr int DEPTH = StackDepth<LAYOUT, true>::value;
  if (out_of_budget(L, errorWord)) L.cur = kDone;
#pragma unroll 1
  for (int k = 0; k < RUN && (L.cur & kLeafBit) == 0u; k++)
  {
    const int r = visit_pair<COUNT, THREADS, DEPTH, STACK, LAYOUT>(L, L.r, tl.recs, st, nPairs, errorWord);
    if (r < 0) L.cur = kDone;
    else if (r == 1) tlas_pop(L, st);
  }
}

template <int LAYOUT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_walk_enter(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, const Tlas& tl,
                                                const Stack<THREADS, STACK>& st, uint32_t* errorWord)
{
  if (out_of_budget(L, errorWord)) L.cur = kDone;
  else tlas_enter<LAYOUT, THREADS, STACK>(L, inst, tl, st);
}

template <int LAYOUT, int TRI, bool ANY, bool COUNT, int THREADS, int STACK>
__device__ __forceinline__ void tlas_walk_leaf(Lane<LAYOUT>& L, const Stack<THREADS, STACK>& st, uint64_t& nTris,
                                               uint32_t* errorWord)
{
  if (out_of_budget(L, errorWord) ||
      (L.cur != kEmptyRef &&
       test_leaf<TRI, ANY, COUNT, EndBit<LAYOUT>::value>(L.tris, L.cur & ~kLeafBit, L.r, L.h, L.inst, nTris)))
    L.cur = kDone;
  else if (L.top > L.base)
  {
    L.top--;
    L.cur = st.get(L.top);
  }
  else
    tlas_leave(L, st);
}

// Up to `phases` phases of a warp over its lanes' rays, all 32 lanes calling
// together: in each phase the warp does the kind of work that most of its lanes
// wait for, and the others wait.  A lane's own order of visits does not depend
// on the votes; every phase advances at least one lane.  A finished lane has
// L.cur = kDone.  (921,600 rays into 240 instances: 6.8 threads per instruction
// and 1,320 us with every lane stepping at once, 13.0 and 1,190 us by vote.)
template <int LAYOUT, int TRI, bool ANY, bool COUNT, int THREADS, int STACK>
__device__ __forceinline__ void run_phases(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, const Tlas& tl,
                                           Stack<THREADS, STACK>& st, uint64_t& nPairs, uint64_t& nTris,
                                           uint32_t* errorWord, int phases)
{
  for (int s = 0; s < phases; s++)
  {
    const TlasState a = tlas_state(L);
    const int nEnter = __popc(__ballot_sync(0xFFFFFFFFu, a.enter)), nTree = __popc(__ballot_sync(0xFFFFFFFFu, a.tree));
    const int nNode = __popc(__ballot_sync(0xFFFFFFFFu, a.node)), nLeaf = __popc(__ballot_sync(0xFFFFFFFFu, a.leaf));
    const int most = max(max(nEnter, nTree), max(nNode, nLeaf));
    if (most == 0) return;
    if (nNode == most)
    {
      if (a.node) tlas_walk_nodes<kTlasNodeRun, LAYOUT, ANY, COUNT>(L, st, nPairs, errorWord);
    }
    else if (nTree == most)
    {
      if (a.tree) tlas_walk_tree<kTlasTreeRun, LAYOUT, COUNT>(L, tl, st, nPairs, errorWord);
    }
    else if (nEnter == most)
    {
      if (a.enter) tlas_walk_enter(L, inst, tl, st, errorWord);
    }
    else if (a.leaf)
      tlas_walk_leaf<LAYOUT, TRI, ANY, COUNT>(L, st, nTris, errorWord);
  }
}

// Up to `steps` steps of a lane's walk with no vote, a run of each kind of work
// that it comes to.  A batch that does not fill the machine is bound by its
// slowest warps' chains, and lanes that wait for a vote make them longer
// (63,000 rays into 100 instances, nearest and any hits: binary 1,012 and 563
// us by vote, 857 and 408 so; FP16 nodes 758, 368; 674, 318).
template <int NODES, int PAIRS, int LAYOUT, int TRI, bool ANY, bool COUNT, int THREADS, int STACK>
__device__ __forceinline__ void run_alone(Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, const Tlas& tl,
                                          Stack<THREADS, STACK>& st, uint64_t& nPairs, uint64_t& nTris,
                                          uint32_t* errorWord, int steps)
{
  for (int k = 0; k < steps && L.cur != kDone; k++)
  {
    if (tlas_state(L).tree) tlas_walk_tree<PAIRS, LAYOUT, COUNT>(L, tl, st, nPairs, errorWord);
    if (tlas_state(L).enter) tlas_walk_enter(L, inst, tl, st, errorWord);
    if (tlas_state(L).node) tlas_walk_nodes<NODES, LAYOUT, ANY, COUNT>(L, st, nPairs, errorWord);
    if (tlas_state(L).leaf) tlas_walk_leaf<LAYOUT, TRI, ANY, COUNT>(L, st, nTris, errorWord);
  }
}

// The hit holds the instance's index; its instance and geometry ids are read
// once, here.
template <bool ANY, int LAYOUT>
__device__ __forceinline__ void write_result(const Lane<LAYOUT>& L, const InstanceDesc* __restrict__ inst, void* out)
{
  const bool hit = L.h.prim != 0xFFFFFFFFu;
  if (ANY)
    reinterpret_cast<uint8_t*>(out)[L.ray] = hit ? 1 : 0;
  else
  {
    const uint32_t instId = hit ? inst[L.h.inst].instId : 0xFFFFFFFFu;
    const uint32_t geomId = hit ? inst[L.h.inst].geomId : 0xFFFFFFFFu;
    store_record(reinterpret_cast<float4*>(reinterpret_cast<hrt_hit*>(out) + L.ray),
                 make_float4(L.h.t, __uint_as_float(L.h.prim), __uint_as_float(instId), __uint_as_float(geomId)),
                 make_float4(L.h.u, L.h.v, 0.0f, 0.0f));
  }
}

// A segmented query: ray i is traced against the one instance of its segment
// (rayOffsets[0..nSeg] ascending, ray i in segment k when rayOffsets[k] <= i <
// rayOffsets[k+1]); an instance id out of range leaves the ray a miss.
struct Segments
{
  const uint32_t* rayOffsets;
  const uint32_t* segInst;
  uint32_t        nSeg;
  uint32_t        nInst;
  const float4* const* segRays;  // segment k's rays, where they lie apart; nullptr: ray i at rays[2 i]
};

__device__ __forceinline__ uint32_t segment_of(uint32_t i, const Segments& sg)
{
  uint32_t lo = 0, hi = sg.nSeg;
  while (hi - lo > 1)
  {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(sg.rayOffsets + mid) <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <int LAYOUT>
__device__ __forceinline__ void start_ray(Lane<LAYOUT>& L, uint32_t i, const float4* __restrict__ rays)
{
  L.ray = i;
  load_record(rays + 2 * (size_t)i, L.po, L.di);
  L.h.t = L.di.w;
  L.h.u = L.h.v = 0.0f;
  L.h.prim = L.h.inst = 0xFFFFFFFFu;
  L.budget = kStepBudget;
}

template <bool COUNT>
__device__ __forceinline__ void flush_counters(uint64_t nPairs, uint64_t nTris, unsigned long long* counters)
{
  if (!COUNT) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    nPairs += __shfl_down_sync(0xFFFFFFFFu, nPairs, o);
    nTris += __shfl_down_sync(0xFFFFFFFFu, nTris, o);
  }
  if ((threadIdx.x & 31) == 0)
  {
    atomicAdd(&counters[0], (unsigned long long)nPairs);
    atomicAdd(&counters[1], (unsigned long long)nTris);
  }
}

// Persistent warp pool.  Lanes make `steps` advances or phases between refills; a warp refills when at least
// `refill` lanes are idle (or all are).  The two-level kernels are held to six
// blocks of 128 threads an SM (80 registers; 921,600 rays, 240 instances: 1,136
// us unbounded, 1,113 at 6, 1,185 at 7, 1,275 at 8 blocks).
template <int LAYOUT, int TRI, bool ANY, int THREADS, bool TLAS, int STACK>
__global__ void __launch_bounds__(THREADS, TLAS ? 768 / THREADS : 0) k_trace_pool(const float4* __restrict__ rays, uint32_t n,
                                                        const InstanceDesc* __restrict__ inst, uint32_t nInst, Tlas tl,
                                                        void* out, uint32_t* errorWord, unsigned int* rayCounter,
                                                        int steps, int refill, int alone, int stackShared,
                                                        RayOrder order)
{
  extern __shared__ uint32_t s_stack[];  // stackShared * THREADS entries
  uint32_t local[STACK != kStackShared ? StackDepth<LAYOUT, TLAS>::value : 1];
  Stack<THREADS, STACK> st{s_stack + threadIdx.x, local, stackShared};
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t ltMask = (1u << lane) - 1u;
  uint64_t none = 0;
  Lane<LAYOUT> L;
  constexpr int kStep = PoolStep<LAYOUT>::value;
  L.ray = kNoRay;
  L.cur = kDone;
  bool exhausted = false;
  while (true)
  {
    // idle lanes write their finished rays' results together, then take new rays
    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, L.cur == kDone);
    const bool all = idle == 0xFFFFFFFFu;
    if (all || (!exhausted && __popc(idle) >= refill))
    {
      if (L.cur == kDone && L.ray != kNoRay) write_result<ANY>(L, inst, out);
      if (all && exhausted) break;
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(rayCounter, (unsigned int)__popc(idle));
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base + (uint32_t)__popc(idle) >= order.nWork) exhausted = true;
      if (L.cur == kDone)
      {
        const uint32_t w = base + __popc(idle & ltMask);
        const uint32_t i = w < order.nWork ? work_ray(order, w, n) : kNoRay;
        L.ray = kNoRay;
        if (i != kNoRay)
        {
          start_ray(L, i, rays);
          bool live = true;
          if (TLAS) tlas_begin(L);
          else live = begin_instance<LAYOUT>(L, inst, nInst, 0);
          if (!live) L.cur = kDone;
        }
      }
    }
    if (TLAS && alone)
      run_alone<kAloneNodeRun, kAloneTreeRun, LAYOUT, TRI, ANY, false, THREADS, STACK>(L, inst, tl, st, none, none, errorWord, steps);
    else if (TLAS)
      run_phases<LAYOUT, TRI, ANY, false, THREADS, STACK>(L, inst, tl, st, none, none, errorWord, steps);
    else if (L.cur != kDone)
    {
      for (int s = 0; s < steps * kStep; s += kStep)
      {
        if (out_of_budget(L, errorWord) ||
            step<false, LAYOUT, TRI, ANY, false, THREADS, STACK>(L, inst, nInst, st, none, none, errorWord))
        {
          L.cur = kDone;
          break;
        }
      }
    }
  }
}

// One thread per ray.
template <int LAYOUT, int TRI, bool ANY, bool COUNT, int THREADS, bool TLAS, int STACK>
__global__ void __launch_bounds__(THREADS) k_trace_grid(const float4* __restrict__ rays, uint32_t n,
                                                        const InstanceDesc* __restrict__ inst, uint32_t nInst, Tlas tl,
                                                        void* out, unsigned long long* counters, uint32_t* errorWord,
                                                        int stackShared, RayOrder order)
{
  extern __shared__ uint32_t s_stack[];  // stackShared * THREADS entries
  uint32_t local[STACK != kStackShared ? StackDepth<LAYOUT, TLAS>::value : 1];
  Stack<THREADS, STACK> st{s_stack + threadIdx.x, local, stackShared};
  uint64_t nPairs = 0, nTris = 0;
  const uint32_t w = grid_work<THREADS>(order);
  const uint32_t i = w < order.nWork ? work_ray(order, w, n) : kNoRay;
  Lane<LAYOUT> L;
  L.cur = kDone;
  if (i != kNoRay)
  {
    start_ray(L, i, rays);
    if (TLAS) tlas_begin(L);
    else if (begin_instance<LAYOUT>(L, inst, nInst, 0))
      while (!out_of_budget(L, errorWord) &&
             !step<true, LAYOUT, TRI, ANY, COUNT, THREADS, STACK>(L, inst, nInst, st, nPairs, nTris, errorWord)) {}
  }
  if (TLAS) run_alone<kGridNodeRun, kGridTreeRun, LAYOUT, TRI, ANY, COUNT, THREADS, STACK>(L, inst, tl, st, nPairs, nTris, errorWord, 0x7FFFFFFF);
  if (i != kNoRay) write_result<ANY>(L, inst, out);
  flush_counters<COUNT>(nPairs, nTris, counters);
}

// ------------------------------------------------ one instance per ray
// A ray that is traced against one instance only needs none of the walk over
// instances: it is set up once and leaves after its last pop.  The lane keeps
// less state, so the kernel holds fewer registers and more warps fit on an SM;
// each ray's decisions are those of the general kernel.  Either the whole
// launch has the one untransformed geometry of its scene (SEG = false: the
// arrays and ids are kernel parameters and the ray is used as given), or every
// ray has the instance of its segment (SEG = true).
struct OneSource
{
  const void*         nodes;  // SEG = false
  const TriRec*       tris;
  uint32_t            instId, geomId;
  const InstanceDesc* inst;  // SEG = true
  Segments            sg;
};

template <int LAYOUT> struct Lane1
{
  Ray<LAYOUT>   r;
  Hit           h;
  uint32_t      ray;     // ray index or kNoRay
  uint32_t      cur;     // current node / leaf reference
  int           top;     // stack depth
  uint32_t      budget;  // steps left for this ray
  const void*   nodes;   // the geometry's binary records or 4-wide nodes
  const TriRec* tris;
  uint32_t      inst;    // instance of the ray's segment (SEG)
};

template <bool SEG, int LAYOUT>
__device__ __forceinline__ void start_ray_one(Lane1<LAYOUT>& L, uint32_t i, const float4* __restrict__ rays,
                                              const OneSource& src)
{
  float4 po, di;
  uint32_t seg = 0;
  const float4* at = rays + 2 * (size_t)i;
  if (SEG)
  {
    seg = segment_of(i, src.sg);
    if (src.sg.segRays != nullptr) at = src.sg.segRays[seg] + 2 * (size_t)(i - __ldg(src.sg.rayOffsets + seg));
  }
  load_record(at, po, di);
  L.ray = i;
  L.h.t = di.w;
  L.h.u = L.h.v = 0.0f;
  L.h.prim = L.h.inst = 0xFFFFFFFFu;
  L.cur = 0;
  L.top = 0;
  L.budget = kStepBudget;
  if (!SEG)
  {
    set_ray(L.r, po.x, po.y, po.z, po.w, di.x, di.y, di.z);
    return;
  }
  const uint32_t k = __ldg(src.sg.segInst + seg);
  L.inst = k;
  if (k < src.sg.nInst && src.inst[k].valid)
  {
    const InstanceDesc& d = src.inst[k];
    make_ray(d, po, di, L.r);
    L.nodes = LAYOUT == 0 ? static_cast<const void*>(d.recs) : d.nodes4;
    L.tris = d.tris;
  }
  else
    L.cur = kDone;
}

// One advance of the single-instance kernel (nodes, then a leaf when the lane
// holds one); true when the ray is finished.
template <bool GRID, int LAYOUT, int TRI, bool ANY, int THREADS, int STACK>
__device__ __forceinline__ bool step_one(Lane1<LAYOUT>& L, Stack<THREADS, STACK>& st, uint32_t* errorWord)
{
  constexpr int DEPTH = StackDepth<LAYOUT, false>::value;
  uint64_t none = 0;
#pragma unroll 1
  for (int k = 0; k < NodeRun<LAYOUT, TRI, ANY, GRID>::value; k++)
  {
    if ((L.cur & kLeafBit) != 0u) break;
    const int r = visit_node<LAYOUT, ANY, false, THREADS, DEPTH, STACK>(L, st, none, errorWord);
    if (r < 0) return true;
    if (r == 1)
    {
      if (L.top == 0) return true;
      L.top--;
      L.cur = st.get(L.top);
    }
  }
  if ((L.cur & kLeafBit) != 0u)
  {
    if (L.cur != kEmptyRef &&
        test_leaf<TRI, ANY, false, EndBit<LAYOUT>::value>(L.tris, L.cur & ~kLeafBit, L.r, L.h, 0u, none))
      return true;  // any-hit found
    if (L.top == 0) return true;
    L.top--;
    L.cur = st.get(L.top);
  }
  return false;
}

template <bool ANY, bool SEG, int LAYOUT>
__device__ __forceinline__ void write_result_one(const Lane1<LAYOUT>& L, const OneSource& src, void* out)
{
  const bool hit = L.h.prim != 0xFFFFFFFFu;
  const uint32_t instId = !ANY && SEG && hit ? src.inst[L.inst].instId : src.instId;
  const uint32_t geomId = !ANY && SEG && hit ? src.inst[L.inst].geomId : src.geomId;
  if (ANY)
    reinterpret_cast<uint8_t*>(out)[L.ray] = hit ? 1 : 0;
  else
  {
    store_record(reinterpret_cast<float4*>(reinterpret_cast<hrt_hit*>(out) + L.ray),
                 make_float4(L.h.t, __uint_as_float(L.h.prim), __uint_as_float(hit ? instId : 0xFFFFFFFFu),
                             __uint_as_float(hit ? geomId : 0xFFFFFFFFu)),
                 make_float4(L.h.u, L.h.v, 0.0f, 0.0f));
  }
}

// Persistent warp pool over one instance (the refill rule of k_trace_pool).
template <int LAYOUT, int TRI, bool ANY, int THREADS, int STACK, bool SEG>
__global__ void __launch_bounds__(THREADS) k_trace_one(const float4* __restrict__ rays, uint32_t n, OneSource src,
                                                       void* out, uint32_t* errorWord, unsigned int* rayCounter,
                                                       int steps, int refill, int stackShared, RayOrder order)
{
  extern __shared__ uint32_t s_stack[];  // stackShared * THREADS entries
  uint32_t local[STACK != kStackShared ? StackDepth<LAYOUT, false>::value : 1];
  Stack<THREADS, STACK> st{s_stack + threadIdx.x, local, stackShared};
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t ltMask = (1u << lane) - 1u;
  Lane1<LAYOUT> L;
  L.ray = kNoRay;
  L.cur = kDone;
  L.nodes = src.nodes;
  L.tris = src.tris;
  constexpr int kStep = PoolStep<LAYOUT>::value;
  bool exhausted = false;
  while (true)
  {
    // idle lanes write their finished rays' results together, then take new rays
    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, L.cur == kDone);
    const bool all = idle == 0xFFFFFFFFu;
    if (all || (!exhausted && __popc(idle) >= refill))
    {
      if (L.cur == kDone && L.ray != kNoRay) write_result_one<ANY, SEG>(L, src, out);
      if (all && exhausted) break;
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(rayCounter, (unsigned int)__popc(idle));
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base + (uint32_t)__popc(idle) >= order.nWork) exhausted = true;
      if (L.cur == kDone)
      {
        const uint32_t w = base + __popc(idle & ltMask);
        const uint32_t i = w < order.nWork ? work_ray(order, w, n) : kNoRay;
        L.ray = kNoRay;
        if (i != kNoRay) start_ray_one<SEG>(L, i, rays, src);
      }
    }
    if (L.cur != kDone)
    {
      for (int s = 0; s < steps * kStep; s += kStep)
      {
        if (out_of_budget(L, errorWord) || step_one<false, LAYOUT, TRI, ANY, THREADS, STACK>(L, st, errorWord))
        {
          L.cur = kDone;
          break;
        }
      }
    }
  }
}

// One thread per ray over one instance: a warp's 32 consecutive rays end
// together, so their results go out as one contiguous kilobyte (results
// written in place over the host link want this).
template <int LAYOUT, int TRI, bool ANY, int THREADS, int STACK, bool SEG>
__global__ void __launch_bounds__(THREADS)
    k_trace_one_grid(const float4* __restrict__ rays, uint32_t n, OneSource src, void* out, uint32_t* errorWord,
                     int stackShared, RayOrder order)
{
  extern __shared__ uint32_t s_stack[];  // stackShared * THREADS entries
  uint32_t local[STACK != kStackShared ? StackDepth<LAYOUT, false>::value : 1];
  Stack<THREADS, STACK> st{s_stack + threadIdx.x, local, stackShared};
  const uint32_t w = grid_work<THREADS>(order);
  const uint32_t i = w < order.nWork ? work_ray(order, w, n) : kNoRay;
  if (i == kNoRay) return;
  Lane1<LAYOUT> L;
  L.nodes = src.nodes;
  L.tris = src.tris;
  start_ray_one<SEG>(L, i, rays, src);
  if (L.cur != kDone)
    while (!out_of_budget(L, errorWord) && !step_one<true, LAYOUT, TRI, ANY, THREADS, STACK>(L, st, errorWord)) {}
  write_result_one<ANY, SEG>(L, src, out);
}

// Dynamic shared memory of a traversal kernel: `shared` stack entries per
// thread; above 48 KB a block needs the opt-in attribute.
template <typename K> cudaError_t allow_smem(K kernel, size_t smem)
{
  if (smem <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <int LAYOUT, int TRI, bool ANY, int THREADS, int STACK, bool SEG>
cudaError_t launch_one(const TraceArgs& a, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  const uint32_t n = (uint32_t)a.n;
  const int shared = STACK == kStackLocal ? 0 : shared_entries<StackDepth<LAYOUT, false>::value>(c.stackEntries);
  const size_t smem = sizeof(uint32_t) * (size_t)shared * THREADS;
  const RayOrder order = ray_order(n, c.imageWidth, c.raysPerWarp);
  OneSource src = {};
  if (SEG)
  {
    src.inst = a.inst;
    src.sg = Segments{a.rayOffsets, a.segInst, a.nSeg, a.nInst, a.segRays};
    src.instId = src.geomId = 0xFFFFFFFFu;  // of a miss
  }
  else
  {
    const InstanceDesc& d = *a.one;
    src.nodes = LAYOUT == 0 ? static_cast<const void*>(d.recs) : d.nodes4;
    src.tris = d.tris;
    src.instId = d.instId;
    src.geomId = d.geomId;
  }
  // launch configuration, with the L2 access-policy window when one is asked for
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t lc = {};
  lc.blockDim = dim3(THREADS);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  if (!SEG && a.persistBytes)
  {
    attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
    attr[0].val.accessPolicyWindow.base_ptr = const_cast<void*>(a.persistBase);
    attr[0].val.accessPolicyWindow.num_bytes = a.persistBytes;
    attr[0].val.accessPolicyWindow.hitRatio = a.persistHitRatio;
    attr[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    lc.attrs = attr;
    lc.numAttrs = 1;
  }
  if (!c.persistent)
  {
    cudaError_t e = allow_smem(k_trace_one_grid<LAYOUT, TRI, ANY, THREADS, STACK, SEG>, smem);
    if (e != cudaSuccess) return e;
    lc.gridDim = dim3(grid_blocks<THREADS>(order));
    return cudaLaunchKernelEx(&lc, k_trace_one_grid<LAYOUT, TRI, ANY, THREADS, STACK, SEG>, a.rays, n, src, a.hits,
                              a.errorWord, shared, order);
  }
  cudaError_t e = allow_smem(k_trace_one<LAYOUT, TRI, ANY, THREADS, STACK, SEG>, smem);
  if (e != cudaSuccess) return e;
  int perSM = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_trace_one<LAYOUT, TRI, ANY, THREADS, STACK, SEG>, THREADS,
                                                    smem);
  if (e != cudaSuccess) return e;
  if (perSM < 1) perSM = 1;
  uint64_t blocks = (uint64_t)numSMs * perSM;
  const uint64_t need = ((uint64_t)order.nWork + THREADS - 1) / THREADS;
  if (blocks > need) blocks = need;
  e = cudaMemsetAsync(a.rayCounter, 0, sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  lc.gridDim = dim3((uint32_t)blocks);
  return cudaLaunchKernelEx(&lc, k_trace_one<LAYOUT, TRI, ANY, THREADS, STACK, SEG>, a.rays, n, src, a.hits,
                            a.errorWord, a.rayCounter, c.stepsPerRefill, c.refillLanes, shared, order);
}

// The short-stack variant only when the requested size leaves part of the
// depth bound to local memory.
template <int LAYOUT, int TRI, bool ANY, int THREADS, bool SEG>
cudaError_t launch_one_any_stack(const TraceArgs& a, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  constexpr int DEPTH = StackDepth<LAYOUT, false>::value;
  return shared_entries<DEPTH>(c.stackEntries) < DEPTH
             ? launch_one<LAYOUT, TRI, ANY, THREADS, kStackSplit, SEG>(a, c, numSMs, s)
             : launch_one<LAYOUT, TRI, ANY, THREADS, kStackShared, SEG>(a, c, numSMs, s);
}

template <int LAYOUT, int TRI, bool SEG>
cudaError_t trace_one(const TraceArgs& a, int kind, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  switch (c.threadsPerBlock)
  {
    case 64:
      return kind == 0 ? launch_one_any_stack<LAYOUT, TRI, false, 64, SEG>(a, c, numSMs, s)
                       : launch_one_any_stack<LAYOUT, TRI, true, 64, SEG>(a, c, numSMs, s);
    case 256:
      return kind == 0 ? launch_one_any_stack<LAYOUT, TRI, false, 256, SEG>(a, c, numSMs, s)
                       : launch_one_any_stack<LAYOUT, TRI, true, 256, SEG>(a, c, numSMs, s);
    default:
      return kind == 0 ? launch_one_any_stack<LAYOUT, TRI, false, 128, SEG>(a, c, numSMs, s)
                       : launch_one_any_stack<LAYOUT, TRI, true, 128, SEG>(a, c, numSMs, s);
  }
}

template <int LAYOUT, int TRI, bool ANY, bool COUNT, int THREADS, bool TLAS, int STACK>
cudaError_t launch(const TraceArgs& a, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  const uint32_t n = (uint32_t)a.n;
  const Tlas tl{a.tlasRecs, a.tlasTris, a.nInst};
  const int shared = STACK == kStackLocal ? 0
                     : STACK == kStackSplit ? shared_entries<StackDepth<LAYOUT, TLAS>::value>(c.stackEntries)
                                            : StackDepth<LAYOUT, TLAS>::value;
  const size_t smem = sizeof(uint32_t) * (size_t)shared * THREADS;
  const RayOrder order = ray_order(n, c.imageWidth, c.raysPerWarp);
  if constexpr (!COUNT)
  {
    if (c.persistent)
    {
      cudaError_t e = allow_smem(k_trace_pool<LAYOUT, TRI, ANY, THREADS, TLAS, STACK>, smem);
      if (e != cudaSuccess) return e;
      int perSM = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_trace_pool<LAYOUT, TRI, ANY, THREADS, TLAS, STACK>,
                                                        THREADS, smem);
      if (e != cudaSuccess) return e;
      if (perSM < 1) perSM = 1;
      uint64_t blocks = (uint64_t)numSMs * perSM;
      const uint64_t need = ((uint64_t)order.nWork + THREADS - 1) / THREADS;
      if (blocks > need) blocks = need;
      e = cudaMemsetAsync(a.rayCounter, 0, sizeof(unsigned int), s);
      if (e != cudaSuccess) return e;
      k_trace_pool<LAYOUT, TRI, ANY, THREADS, TLAS, STACK><<<(uint32_t)blocks, THREADS, smem, s>>>(
          a.rays, n, a.inst, a.nInst, tl, a.hits, a.errorWord, a.rayCounter, c.stepsPerRefill, c.refillLanes, c.alone,
          shared, order);
      return cudaGetLastError();
    }
  }
  cudaError_t e = allow_smem(k_trace_grid<LAYOUT, TRI, ANY, COUNT, THREADS, TLAS, STACK>, smem);
  if (e != cudaSuccess) return e;
  const uint32_t blocks = grid_blocks<THREADS>(order);
  k_trace_grid<LAYOUT, TRI, ANY, COUNT, THREADS, TLAS, STACK><<<blocks, THREADS, smem, s>>>(
      a.rays, n, a.inst, a.nInst, tl, a.hits, a.counters, a.errorWord, shared, order);
  return cudaGetLastError();
}

// An instance tree's stack is all in local memory unless the caller set a shape,
// and all in shared memory when that shape asks for the whole of it: the split
// variant's, whose shared part is then the whole.
template <int LAYOUT, int TRI, bool ANY, int THREADS, bool TLAS>
cudaError_t launch_any_stack(const TraceArgs& a, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  constexpr int DEPTH = StackDepth<LAYOUT, TLAS>::value;
  return shared_entries<DEPTH>(c.stackEntries) < DEPTH || (TLAS && c.given)
             ? launch<LAYOUT, TRI, ANY, false, THREADS, TLAS, kStackSplit>(a, c, numSMs, s)
             : launch<LAYOUT, TRI, ANY, false, THREADS, TLAS, TLAS ? kStackLocal : kStackShared>(a, c, numSMs, s);
}

template <int LAYOUT, int TRI, bool TLAS>
cudaError_t trace_tlas(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  // counting runs: the whole stack in shared memory (the counts do not depend on it)
  if (counting)
    return kind == 0 ? launch<LAYOUT, TRI, false, true, 128, TLAS, kStackShared>(a, c, numSMs, s)
                     : launch<LAYOUT, TRI, true, true, 128, TLAS, kStackShared>(a, c, numSMs, s);
  switch (c.threadsPerBlock)
  {
    case 64:
      return kind == 0 ? launch_any_stack<LAYOUT, TRI, false, 64, TLAS>(a, c, numSMs, s)
                       : launch_any_stack<LAYOUT, TRI, true, 64, TLAS>(a, c, numSMs, s);
    case 256:
      return kind == 0 ? launch_any_stack<LAYOUT, TRI, false, 256, TLAS>(a, c, numSMs, s)
                       : launch_any_stack<LAYOUT, TRI, true, 256, TLAS>(a, c, numSMs, s);
    default:
      return kind == 0 ? launch_any_stack<LAYOUT, TRI, false, 128, TLAS>(a, c, numSMs, s)
                       : launch_any_stack<LAYOUT, TRI, true, 128, TLAS>(a, c, numSMs, s);
  }
}

// Counting runs use the one-thread-per-ray grid at 128 threads (the counts do
// not depend on the schedule) and have no segments.  Segmented queries and a
// scene of one untransformed instance use the one-instance kernels, a scene with
// an instance tree the two-level ones.
template <int LAYOUT, int TRI>
cudaError_t trace_layout(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s)
{
  if (a.rayOffsets != nullptr)
    return counting ? cudaErrorInvalidValue : trace_one<LAYOUT, TRI, true>(a, kind, c, numSMs, s);
  if (a.one != nullptr && !counting && a.tlasRecs == nullptr)
    return trace_one<LAYOUT, TRI, false>(a, kind, c, numSMs, s);
  if (a.tlasRecs != nullptr)
    return trace_tlas<LAYOUT, TRI, true>(a, kind, counting, c, numSMs, s);
  return trace_tlas<LAYOUT, TRI, false>(a, kind, counting, c, numSMs, s);
}

}  // namespace

// Per-layout entry points, one translation unit each (trace_l*.cu).
cudaError_t trace_l0(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_l1(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_l2(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_l3(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
// The same with the watertight triangle test (trace_w*.cu).
cudaError_t trace_w0(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w1(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w2(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w3(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);

}  // namespace hrt
