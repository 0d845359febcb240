// Traversal dispatch: validates the batch and calls the layout's kernels
// (trace_impl.cuh; one translation unit per layout and triangle test,
// trace_l0..3.cu for Moller-Trumbore, trace_w0..3.cu for the watertight test).
#include "hrt_kernels.cuh"

namespace hrt
{
cudaError_t trace_l0(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_l1(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_l2(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_l3(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w0(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w1(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w2(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);
cudaError_t trace_w3(const TraceArgs& a, int kind, int counting, const TraceConfig& c, int numSMs, cudaStream_t s);

namespace
{

// Warps an SM that a small batch is spread over, and that hold a batch at once.
constexpr int kSpreadWarps = 13, kResidentWarps = 36;
// Unless the caller set a shape: idle lanes at which a warp refills, and
// advances (phases of an instance tree's walk) between its looks at them.
constexpr int kRefillLanes = 8, kAdvances = 8, kTreePhases = 32, kTreeSteps = 4;
// The same on an instance tree, and (4-wide nodes) on a transformed instance or
// several in turn, whose lanes hold more registers; the batch on a tree (in
// warps of 32 rays an SM) from which nearest hits go by vote.
constexpr int kTreeResidentWarps = 24, kGeneralResidentWarps = 18, kVoteWarps = 128;

// The shape of one launch.  A shape that the caller set is kept, but for a pool
// in a batch so small that it is spread over warps (below): a pool of any block
// and stack size holds such a batch at once and would refill nothing, so it goes
// one thread per ray, with the block and the stack that were set (1,000 rays, a
// pool of 128 threads 82 us, so 49; FP16 nodes, any hits).
//
// A batch that does not fill the GPU's warps is bound by the slowest warp's
// chain of dependent instructions, and a warp of 32 rays that part ways runs
// all their chains: such a batch is spread, the fewest rays a warp (a power of
// two) for which 13 warps an SM suffice, one thread per ray.  Random rays into
// a soup, us, 32 rays a warp against the spread: 96 rays into 2,003 triangles
// 41 -> 27 (binary), 34 -> 20 (FP16 nodes); 1,000 rays into 20,000 triangles
// 90 -> 62, 72 -> 45; 8,000 rays into 100,000 triangles 155 -> 125, 127 -> 103
// (at 4 rays a warp; at 1: 143, 143); 30,000 rays 169 -> 156, 134 -> 127 (at
// 16; at 8: 161, 158); 100,000 rays are faster at 32 (210 against 260 at 16).
// A batch whose rays are all resident at once gains nothing from the pool and
// goes without its counter and the memset before it (100,000 rays 210 -> 208,
// FP16 nodes 180 -> 170); 262,144 eye rays are faster in the pool (binary 157
// against 172).
//
// The refills: incoherent rays want idle lanes filled early (500,000
// random rays, 8-bit nodes: 652 us at 24 lanes, 555 at 8; FP16 582 -> 520),
// and coherent ones do not care (full-HD eye rays 156 against 157).  Looks after
// 4, 8, 16 advances: 2M occlusion rays, FP16 nodes 391, 378, 419 us, 500,000
// random rays 496, 497, 509; after 16 and 32 phases, 240 instances 1,161, 1,154.
//
// On an instance tree lanes wait for the warp's vote only in large batches
// (trace_impl.cuh).  Nearest hits, 8 and 100 instances, us, pool without a vote
// against with it: binary, 170,000 rays 913, 1,091 against 1,002, 1,221; 400,000
// 1,642, 1,627 against 1,684, 1,709; 900,000 3,282, 2,927 against 3,191, 2,864;
// FP16 nodes 798, 914 against 847, 1,051; 1,435, 1,408 against 1,437, 1,486;
// 2,832, 2,533 against 2,709, 2,439.  Any hits are faster without at every size
// (binary, 900,000 rays 1,452 and 1,126 against 1,532 and 1,226), 8-bit nodes by
// vote (129,600 eye rays, 60 instances 266 against 332).  One thread per ray, no
// vote, while all rays are resident (100,000 rays, 100 instances, binary 924,
// in the pool 927; FP16 764, 798; 10,000 rays 555, 681); 170,000 rays are faster
// in the pool (1,091 against 1,340).  One transformed instance, binary: 150,000
// rays 159 us in the pool, 203 one thread per ray; 90,000, watertight, 165, 157.
// Eight in turn, FP32 nodes, watertight: 100,000 rays 626, 852.
TraceConfig launch_shape(const TraceArgs& a, const TraceConfig& c, int kind, int layout, int numSMs)
{
  TraceConfig s = c;
  const bool tree = a.tlasRecs != nullptr && a.rayOffsets == nullptr;
  s.alone = tree && layout != 3 && (kind == 1 || a.n <= (uint64_t)numSMs * kVoteWarps * 32);
  if (!c.given)
  {
    if (s.refillLanes > kRefillLanes) s.refillLanes = kRefillLanes;
    s.stepsPerRefill = !tree ? kAdvances : s.alone ? kTreeSteps : kTreePhases;
  }
  int perWarp = 32;
  while (perWarp > 1 && a.n <= (uint64_t)numSMs * kSpreadWarps * (perWarp / 2)) perWarp /= 2;
  const int resident = !tree && (a.one || a.rayOffsets) ? kResidentWarps
                       : tree || layout == 0            ? kTreeResidentWarps
                                                        : kGeneralResidentWarps;
  if (!c.given && a.n <= (uint64_t)numSMs * resident * 32)
  {
    s.persistent = 0;
    s.threadsPerBlock = 64;
  }
  if (trace_spreads(a.n, numSMs)) s.persistent = 0;
  if (!s.persistent) s.raysPerWarp = perWarp;
  return s;
}

}  // namespace

bool trace_spreads(uint64_t n, int numSMs) { return n <= (uint64_t)numSMs * kSpreadWarps * 16; }

cudaError_t trace(const TraceArgs& a, int kind, int counting, int layout, const TraceConfig& config, int numSMs,
                  cudaStream_t s)
{
  if (a.n == 0) return cudaSuccess;
  if (a.n > 0x7FFFFFFFull) return cudaErrorInvalidValue;  // the pool's counter may overshoot n by a few warps
  const TraceConfig c = counting ? config : launch_shape(a, config, kind, layout, numSMs);
  if (a.triTest == 1)
    switch (layout)
    {
      case 0: return trace_w0(a, kind, counting, c, numSMs, s);
      case 1: return trace_w1(a, kind, counting, c, numSMs, s);
      case 2: return trace_w2(a, kind, counting, c, numSMs, s);
      case 3: return trace_w3(a, kind, counting, c, numSMs, s);
      default: return cudaErrorInvalidValue;
    }
  if (a.triTest != 0) return cudaErrorInvalidValue;
  switch (layout)
  {
    case 0: return trace_l0(a, kind, counting, c, numSMs, s);
    case 1: return trace_l1(a, kind, counting, c, numSMs, s);
    case 2: return trace_l2(a, kind, counting, c, numSMs, s);
    case 3: return trace_l3(a, kind, counting, c, numSMs, s);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace hrt
