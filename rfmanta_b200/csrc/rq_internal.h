// Internal declarations shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "rq_device.cuh"

namespace rq {

// Device pointers of one ray batch (SoA) and its outputs.
struct RayArgs {
  int n;
  const float* org;  // 3 rows: org[c * stride + i]
  const float* dir;  // 3 rows
  const float* tmax; // n
  float* t;
  int32_t* prim;
  float* u;
  float* v;
  int stride = 0;    // elements between the rows of org/dir; 0 = n
};

struct LaunchPlan {
  int block_threads;
  int grid;         // persistent grid size
  int refill;       // idle lanes before a warp refills
  bool persistent;
  int* counter;     // device ray counter (persistent form), zeroed per launch
};

// Bytes of traversal stack per block: of the binary walk 8 per pending entry
// not kept in registers (at least one); of the wide walk 4, for at most three
// refs per two levels, the end mark and one entry past the top.
inline size_t stack_bytes(int depth, int block, bool wide, int regs = 0) {
  const int binary = depth - regs > 1 ? depth - regs : 1;
  return wide ? (size_t)((depth + 1) / 2 * 3 + 2) * block * sizeof(int)
              : (size_t)binary * block * 2 * sizeof(int);
}

cudaError_t launch_trace(const DevScene& S, const RayArgs& a, bool anyhit,
                         const LaunchPlan& plan, cudaStream_t st);

int max_blocks_per_sm(const DevScene& S, bool anyhit, bool persistent, int block_threads);

// Writes the 48-byte triangle records in leaf order (perm[k] = original
// triangle id; bit 31 of perm[k] marks the last triangle of a leaf).
cudaError_t launch_tri_setup(int tri_kind, const float* d_verts,
                             const uint32_t* d_idx, const int32_t* d_perm,
                             int n, float4* d_tris, cudaStream_t st);

// Ordered stream compaction (rq_path.cu): the indices i < n with flags[i]
// != 0, in increasing order, into qout, and their count into *total_out;
// tile_counts holds flag_compaction_tiles(n) ints of scratch.
int flag_compaction_tiles(int n);
cudaError_t launch_flag_compaction(const uint8_t* flags, int n, int* tile_counts, int* total_out,
                                   int* qout, cudaStream_t st);

// cudaMalloc, with rq_fail_allocation's failures.
cudaError_t device_alloc(void** p, size_t bytes);
template <class T>
bool device_array(T** p, size_t n) {
  return device_alloc(reinterpret_cast<void**>(p), (n ? n : 1) * sizeof(T)) == cudaSuccess;
}

// Whether the stream is being recorded into a CUDA graph.
bool recording(cudaStream_t st);

// Device memory that frames recorded into a caller's CUDA graph may hold: given
// up by an owner that replaces it, such memory is kept until the owner goes (at
// most one block per recording), other memory is freed.
struct Kept {
  std::vector<void*> blocks;
  void give_up(void* p, bool& recorded) {
    if (recorded && p)
      blocks.push_back(p);
    else
      cudaFree(p);
    recorded = false;
  }
  ~Kept() {
    for (void* p : blocks) cudaFree(p);
  }
};

void set_error(const std::string& msg);

}  // namespace rq
