// Ray-query traversal kernels: closest hit and any hit over the four-wide
// nodes, or over the paired-child node records (trees without wide nodes,
// statistics), Wald or Kensler-Shirley triangles.
//
// Visit order follows DynBVH::intersectNode (Model/Groups/DynBVH.cc:274-404):
// the child on the near side of the node's split axis first for closest
// hit (dir[axis] > 0 ? left : right), the RTSAH-cheaper child first for any
// hit (isLeftCheaper).  A child whose box was hit but which is visited
// later is pushed with its entry distance; at pop time it is skipped unless
// entry <= current minT, which is exactly the reference's re-test of that
// box at visit time (the box's exit side was already checked at push).
//
// Two launch forms:
//   * one thread per ray (grid covers the batch);
//   * persistent: a grid sized to fill the GPU once, each warp fetching new
//     rays with one atomicAdd per refill when `refill` or more of its lanes
//     are idle (warp-ballot work stealing).
// The traversal stack lives in shared memory, one column per thread, sized to
// the tree's depth so it can never overflow.
#include <cuda_runtime.h>

#include "rq_wide.cuh"

namespace rq {

// Wide walk: lanes of a warp that wait at a leaf, or have ended, before the
// others stop descending.  Random rays, bound by L1 wavefronts, want the leaves
// batched (any hit 507 / 427 / 404 us at 8 / 16 / 24 for 3 M; closest hits at 12 /
// 16 / 20: 359 / 333 / 326 us for 3 M over 8 k triangles), sparse camera rays,
// bound by issue slots, the idle lanes short (closest 150 / 157 / 158 us for
// 777,777 over 410 k).  Any-hit rays end at their first hit and lose nothing at
// 20; closest hits stay at 12 for the camera's sake.  A vote that follows what
// the warp sees is not built.
constexpr int kClosestVote = 12, kAnyVote = 20;

// Registers of both forms: left alone the compiler takes 64 for closest Wald hits
// and spills (777,777 random rays over 295 k triangles 171 us, 160 at 72).  At 64
// without spills batches of millions gain 2-4% (3 M camera rays over 8 k triangles
// 145 -> 140 us) and small ones, bound by latency, lose 3-8% (100 k over 295 k
// 33.9 -> 35.9 us); Kensler-Shirley rays lose 6% (777,777 camera rays 134 -> 143).
constexpr int kTraceRegisters = 72;

template <class Walk, bool ANY>
__global__ void __maxnreg__(kTraceRegisters)
    trace_kernel(const __grid_constant__ DevScene S, RayArgs a) {
  extern __shared__ int2 smem_stack[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  Walk walk;
  walk.init(smem_stack);
  Ray r;
  Hit h;
  int ref = kDone;
  if (i < a.n) {
    load_ray(a, i, r);
    walk.start(S, r, ANY, h, ref);
  }
  while (__any_sync(0xffffffffu, ref != kDone))
    walk.step(S, r, h, ANY, ref != kDone, ANY ? kAnyVote : kClosestVote, ref, ANY);
  if (i < a.n) store_hit(a, i, h);
}

// Persistent form: each lane keeps one ray in flight; after every step the
// warp counts its idle lanes with a ballot and, once `refill` or more are
// idle (or none is busy), one lane claims that many ray indices with a single
// atomicAdd and the idle lanes take them.
template <class Walk, bool ANY>
__global__ void __maxnreg__(kTraceRegisters)
    trace_persistent_kernel(const __grid_constant__ DevScene S, RayArgs a, int* counter,
                            int refill) {
  extern __shared__ int2 smem_stack[];
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  Walk walk;
  walk.init(smem_stack);
  int idx = -1;  // ray in flight, -1 = idle
  bool exhausted = false;
  Ray r;
  Hit h;
  int ref = kDone;
  for (;;) {
    const bool idle = (idx < 0) && !exhausted;
    const unsigned m = __ballot_sync(0xffffffffu, idle);
    const unsigned busy = __ballot_sync(0xffffffffu, idx >= 0);
    if (m != 0u && (__popc(m) >= refill || busy == 0u)) {
      const int leader = __ffs(m) - 1;
      int base = 0;
      if ((int)lane == leader) base = atomicAdd(counter, __popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (idle) {
        const int mine = base + __popc(m & lt_mask);
        if (mine < a.n) {
          idx = mine;
          load_ray(a, idx, r);
          walk.start(S, r, ANY, h, ref);
        } else {
          exhausted = true;
        }
      }
    }
    if (__all_sync(0xffffffffu, exhausted)) break;
    walk.step(S, r, h, ANY, idx >= 0 && ref != kDone, ANY ? kAnyVote : kClosestVote, ref, ANY);
    if (idx >= 0 && ref == kDone) {
      store_hit(a, idx, h);
      idx = -1;
    }
  }
}

// The kernel of a query over this scene: the wide walk where the tree has
// wide nodes.
template <class Walk>
static const void* trace_fn(bool any, bool persistent) {
  if (persistent)
    return any ? (const void*)trace_persistent_kernel<Walk, true>
               : (const void*)trace_persistent_kernel<Walk, false>;
  return any ? (const void*)trace_kernel<Walk, true> : (const void*)trace_kernel<Walk, false>;
}

static const void* trace_fn(const DevScene& S, bool any, bool persistent) {
  if (S.tri_kind == kWald)
    return S.wide ? trace_fn<WideWalk<kWald>>(any, persistent)
                  : trace_fn<BinaryWalk<kWald, false, 0>>(any, persistent);
  return S.wide ? trace_fn<WideWalk<kKS>>(any, persistent)
                : trace_fn<BinaryWalk<kKS, false, 0>>(any, persistent);
}

cudaError_t launch_trace(const DevScene& S, const RayArgs& a, bool anyhit,
                         const LaunchPlan& plan, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const void* f = trace_fn(S, anyhit, plan.persistent);
  const size_t smem = stack_bytes(S.depth, plan.block_threads, S.wide != nullptr);
  const int grid = plan.persistent ? plan.grid
                                   : (a.n + plan.block_threads - 1) / plan.block_threads;
  void* args[] = {(void*)&S, (void*)&a, (void*)&plan.counter, (void*)&plan.refill};
  return cudaLaunchKernel(f, dim3(grid), dim3(plan.block_threads), args, smem, st);
}

// Occupancy-derived resident blocks per SM.
int max_blocks_per_sm(const DevScene& S, bool anyhit, bool persistent, int block_threads) {
  int nb = 0;
  const void* f = trace_fn(S, anyhit, persistent);
  const size_t smem = stack_bytes(S.depth, block_threads, S.wide != nullptr);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, block_threads,
                                                    smem) != cudaSuccess)
    return 1;
  return nb > 0 ? nb : 1;
}

}  // namespace rq
