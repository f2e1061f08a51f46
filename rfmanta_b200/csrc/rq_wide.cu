// Makes the four-wide nodes of a scene's tree (rq_wide.cuh) from its node
// records, one thread per record: the node of record r folds r and its two
// child records and holds the (up to four) grandchildren, a child that is a
// leaf taking the first of its side's two slots.  Nodes are numbered like the
// records, so every thread works alone and the walk, which only follows
// grandchildren, touches every other level's.  Folding fixed pairs of levels
// costs 1% more visits than choosing the largest children (measured on the
// benchmark's scenes) and needs no order between the threads.
//
// 96 bytes, 32-byte aligned, read as three 256-bit loads:
//   words 0-2   centre of the node's cube / its size
//   word 3      1 / size of the cube
//   words 4-7   refs of the four slots (kDone: empty)
//   words 8-13  box centres x01 x23 y01 y23 z01 z23 (packed 16-bit pairs)
//   words 14-19 half extents, the same order, padded (rq_wide.cuh)
//   word 20     a byte per folded record (r, first side, second side): one-hot
//               of its axis, 3 higher where the side in front is the right one
// The sides, and the slots within a side, are in any-hit order (the cheaper
// child, isLeftCheaper, in front).
//
// The thread also stores the boxes of r's leaf children (leaf_box) and
// checks what the walk relies on: finite, nested boxes.  After an update that
// failed on the device nothing is made, and a ref outside the tree is not
// followed: records that a failed update never wrote hold anything.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "rq_scene.h"
#include "rq_wide.cuh"

namespace rq {

namespace {

struct RecBox {
  float lo[3], hi[3];
};

__device__ __forceinline__ void record_boxes(const float4* p, RecBox& l, RecBox& r) {
  const float4 q0 = p[0], q1 = p[1], q2 = p[2];
  l = RecBox{{q0.x, q0.y, q0.z}, {q0.w, q1.x, q1.y}};
  r = RecBox{{q1.z, q1.w, q2.x}, {q2.y, q2.z, q2.w}};
}

__device__ __forceinline__ bool inside(const RecBox& a, const RecBox& b) {
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) ok = ok && a.lo[c] >= b.lo[c] && a.hi[c] <= b.hi[c];
  return ok;
}

__device__ __forceinline__ uint32_t pair_bits(__half a, __half b) {
  return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
}

__global__ void __launch_bounds__(128)
    wide_nodes_kernel(const float4* __restrict__ recs, int n, const int* n_dev, const int* error,
                      int n_tris, uint32_t* wide, float4* leaf_box, int* bad) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (n_dev) n = min(n, *n_dev);
  if (r >= n) return;
  if (error && *error != 0) {
    *bad = 1;
    return;
  }
  // largest coordinate of the scene, for the smallest cube
  RecBox rl, rr;
  record_boxes(recs, rl, rr);
  float big = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c)
    big = fmaxf(big, fmaxf(fmaxf(fabsf(rl.lo[c]), fabsf(rl.hi[c])),
                           fmaxf(fabsf(rr.lo[c]), fabsf(rr.hi[c]))));
  const float4* p = recs + 4 * (size_t)r;
  const int4 q3 = reinterpret_cast<const int4*>(p)[3];
  RecBox side[2];
  record_boxes(p, side[0], side[1]);
  bool ok = true;
  float lo[3], hi[3], ext = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lo[c] = fminf(side[0].lo[c], side[1].lo[c]);
    hi[c] = fmaxf(side[0].hi[c], side[1].hi[c]);
    ext = fmaxf(ext, hi[c] - lo[c]);
#pragma unroll
    for (int k = 0; k < 2; ++k)
      ok = ok && side[k].lo[c] <= side[k].hi[c] && fabsf(side[k].lo[c]) < 1e15f &&
           fabsf(side[k].hi[c]) < 1e15f;
  }
  const float size = fmaxf(ext, big * kWideMinCube);
  const float gs = __frcp_rn(size);
  float pb[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) pb[c] = (0.5f * lo[c] + 0.5f * hi[c]) * gs;
  RecBox box[4];
  int ref[4] = {kDone, kDone, kDone, kDone};
  const auto order = [](int meta) {  // its byte of word 20
    return 1u << ((meta & 3) + ((meta >> 2) & 1 ? 0 : 3));
  };
  unsigned meta = order(q3.z);
  const bool left = (q3.z >> 2) & 1;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const bool is_left = (k == 0) == left;
    const int c = is_left ? q3.x : q3.y;
    const RecBox b = side[is_left ? 0 : 1];
    if (c < 0 ? ~c >= n_tris : c >= n) {
      ok = false;
    } else if (c < 0) {
      ref[2 * k] = c;
      box[2 * k] = b;
      leaf_box[2 * (size_t)(~c)] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.hi[0]);
      leaf_box[2 * (size_t)(~c) + 1] = make_float4(b.hi[1], b.hi[2], 0.f, 0.f);
    } else {
      const float4* s = recs + 4 * (size_t)c;
      const int4 t3 = reinterpret_cast<const int4*>(s)[3];
      RecBox x, y;
      record_boxes(s, x, y);
      const bool x_first = (t3.z >> 2) & 1;
      box[2 * k] = x_first ? x : y;
      box[2 * k + 1] = x_first ? y : x;
      ref[2 * k] = x_first ? t3.x : t3.y;
      ref[2 * k + 1] = x_first ? t3.y : t3.x;
      ok = ok && inside(x, b) && inside(y, b);
      meta |= order(t3.z) << (8 + 8 * k);
    }
  }
  if (!ok || !(big > 1e-15f)) *bad = 1;
  uint32_t w[24];
#pragma unroll
  for (int c = 0; c < 3; ++c) w[c] = __float_as_uint(pb[c]);
  w[3] = __float_as_uint(gs);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[4 + k] = (uint32_t)ref[k];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    __half ce[4], he[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (ref[k] == kDone) {
        ce[k] = he[k] = __float2half(0.f);
        continue;
      }
      // exact in double: products of two floats, and sums of near magnitudes
      const double a = (double)box[k].lo[c] * gs - pb[c], b = (double)box[k].hi[c] * gs - pb[c];
      ce[k] = __float2half((float)(0.5 * (a + b)));
      const double m = (double)__half2float(ce[k]);
      he[k] = __float2half_ru(__double2float_ru(fmax(b - m, m - a) + (double)kWidePad));
    }
    w[8 + 2 * c] = pair_bits(ce[0], ce[1]);
    w[9 + 2 * c] = pair_bits(ce[2], ce[3]);
    w[14 + 2 * c] = pair_bits(he[0], he[1]);
    w[15 + 2 * c] = pair_bits(he[2], he[3]);
  }
  w[20] = meta;
  w[21] = w[22] = w[23] = 0u;
  uint4* out = reinterpret_cast<uint4*>(wide + 24 * (size_t)r);
#pragma unroll
  for (int k = 0; k < 6; ++k)
    out[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
}

}  // namespace

// Launches the kernel over the scene's first n records, or the first
// min(n, *n_dev) of an update whose *error is 0 (on the legacy stream, where
// trees are made), with n_tris triangles in their leaves; *d_bad is set to 1
// where the tree cannot be walked wide.
cudaError_t Scene::make_wide(int n, int n_tris, int* d_bad, const int* n_dev, const int* error) {
  if (n <= 0) return cudaSuccess;
  wide_nodes_kernel<<<(n + 127) / 128, 128>>>(d_nodes, n, n_dev, error, n_tris, d_wide,
                                              d_leaf_box, d_bad);
  return cudaGetLastError();
}

}  // namespace rq
