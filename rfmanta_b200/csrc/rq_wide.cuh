// Four-wide traversal of the binary tree, with the binary walk's results.
//
// A wide node holds the (up to four) grandchildren of a node record in
// 96 bytes: their boxes as 16-bit centre and half extent in the node's own
// cube, padded outwards, their refs, and the three split axes (layout in
// rq_wide.cu).  One visit replaces two to three dependent record visits and
// tests four boxes with packed 16-bit arithmetic.
//
// Why the results are the binary walk's, bit for bit:
//   * the four children are taken in the binary walk's order, which each of
//     the three folded records fixes by its axis and the ray's direction
//     signs (closest hit) or its isLeftCheaper flag (any hit: the order of the
//     slots themselves, so kernels of any-hit rays alone swap nothing);
//   * a 16-bit box only decides what is skipped, and it contains the exact
//     box by more than all rounding errors (bound below), so no leaf that the
//     binary walk tests is skipped;
//   * a leaf's exact box test (box_test, the current minT) is made before a
//     hit in it is accepted.  Node boxes are nested (checked when the wide
//     nodes are made) and rounding is monotonic, so every record above a leaf
//     whose exact box is hit was hit too, with a minT at least as large: the
//     leaf's own test stands for the whole chain.
//
// Error bound.  In units of the node's cube (boxes within 0.565 of its centre,
// padding included) the reference point is the ray's closest point to the
// cube's centre.  A ray that meets the cube has it within 0.98, and within 0.78
// along one axis, so a plane lies within 1.34 of it.  With u = 2^-11 (half
// rounding), a plane's time carries errors, as positions along its axis, of
// 0.78 u (offset) + 0.5 u (slope) + 1.34 u (centre) + 0.53 u (extent) + 1.34 u
// (sum) = 4.5 u = 2.2e-3 < kWidePad, by which the node's boxes are larger.
// The 32-bit roundings - the origin in cube units (one multiply-add, so relative
// to the distance, not to the coordinate: the boxes are placed in double around
// the rounded centre), the slope, and two of the exact test - are 4 * 2^-24 of
// the time to the plane, at most 7 against a bound (minT); both planes of a
// comparison together, 8 * 2^-24 of the time to the cube: kWide32 of it is added
// to every exit time.  So the padding grows with the ray's own distance and
// costs nothing near by, wherever the scene lies and however fine it is.  Times
// against 0 and minT carry 2^-8 cubes more.
//
// What it is for: the binary walk is bound by issue slots (52-57% issued, 10-15
// of 32 lanes) and by the dependent record loads (13 to 31 visits a ray), and on
// random rays by L1 wavefronts (79% busy).  The wide walk makes 1.7 times fewer
// visits, reads a node in three loads for a record's four, and votes: a warp
// stops descending once enough lanes wait at leaves, so leaves are tested by
// more lanes together.  Measured against the binary walk: 777,777 camera rays
// 234 -> 134 us, 2^20 random closest hits 239 -> 194 us, 3 M random occlusion
// rays 581 -> 385 us, the 512x512 Whitted frame 211 -> 133 us, the 1280x720x16
// path frame 11.35 -> 7.24 ms (in one pass, rq_pathhost.cu).  Dense coherent
// closest hits, two to four visits a ray, lose by their longer setup: 3 M camera
// rays over 8 k / 295 k triangles 122 -> 145, 174 -> 203 us.  Eight-wide nodes
// would save a third more visits but cost as many instructions a ray (more order
// to keep) and more L1 wavefronts; 8-bit boxes halve the bytes but need twice the
// padding.
//
// Rays along an axis plane (a direction component of zero, or below 2^-kWideFlat of
// the largest) are flat on that axis: their offset along it does not change, and
// the slabs are tested with the slope kWideSlope (wide_visit<true>).  Where the
// inverse is infinite and the origin lies on a plane of the hit leaf's box, the
// exact tests of the boxes above it are not implied by the leaf's (0 * inf is NaN,
// which bounds nothing): such a ray starts again on the exact walk, with what it
// has found.
//
// Other rays outside the bounds (slopes between kWideSlope and flat, an origin
// more than kWideOrigin half sizes from the scene's centre, no finite direction)
// take the exact binary walk over the node records (exact_visit), in the same loop
// and on the same stack column: refs alone, since a popped record's children are
// tested against the minT of then.
#pragma once

#include <cuda_fp16.h>

#include "rq_traverse.cuh"

namespace rq {

constexpr float kWidePad = 2.5e-3f;
constexpr float kWide32 = 5e-7f;        // 8.4 * 2^-24
constexpr float kWideSlope = 16384.f;   // |d|max / |d_k| is below
constexpr int kWideFlat = 48;
// Distance of an origin from the scene's centre in (largest) half sizes.  The
// bound above needs kWideOrigin / kWideMinCube * kWide32 to stay a half number,
// and a flat ray's real change of offset, 2^-kWideFlat of the distance in cubes,
// to stay below kWidePad.  Camera rays from 400 / 1,000 / 1,900 sizes away on 295
// k and 410 k triangles: 65 / 66 / 68 and 135 / 148 / 161 us (the exact walk: 72,
// 74 and 193, 189 at the last two).
constexpr float kWideOrigin = 4096.f;
// Smallest cube over the scene's largest |coordinate|: 32 roundings of it, so
// that the rounded centre is within 2/32 of the box's.
constexpr float kWideMinCube = 1.f / (1 << 19);
// Deeper trees (chains, from files) keep the walk over the records.
constexpr int kWideMaxDepth = 64;

// What a wide visit needs of a ray beside the Ray itself.
struct WideRay {
  float A[3];         // |d|max / d_k
  float w[3];         // -(d_k / |d|max) / sum (d_k / |d|max)^2
  __half2 a2[3];      // A, both halves
  __half2 p2[3];      // |A|, both halves
  __half2 n2[3];      // -|A|
  float dm;           // |d|max
  unsigned side;      // per folded record's byte: bit k: d_k > 0, bit 3 + k: not
                      // (closest hit); all set: any hit.  kRayFlat, kRayExact
};
constexpr unsigned kRayFlat = 1u << 24, kRayExact = 1u << 25;

// Prepares a ray but for its origin; false when it must take the exact walk.
__device__ __forceinline__ bool wide_setup(const Ray& r, bool any, WideRay& w) {
  const float ax = fabsf(r.d[0]), ay = fabsf(r.d[1]), az = fabsf(r.d[2]);
  w.dm = fmaxf(fmaxf(ax, ay), az);
  bool ok = w.dm > 1e-15f && w.dm < 1e15f && !(r.minT != r.minT), flat = false;
  const float rd = __fdividef(1.f, w.dm);
  float g[3], sum = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w.A[c] = w.dm * r.inv[c];
    if (fabsf(w.A[c]) > (float)(1LL << kWideFlat)) {
      flat = true;
      w.A[c] = kWideSlope;
    } else {
      ok = ok && fabsf(w.A[c]) < kWideSlope;
    }
    g[c] = r.d[c] * rd;
    sum = __fmaf_rn(g[c], g[c], sum);
    w.a2[c] = __float2half2_rn(w.A[c]);
    w.p2[c] = __habs2(w.a2[c]);
    w.n2[c] = __hneg2(w.p2[c]);
  }
  const float k = __fdividef(-1.f, sum);
#pragma unroll
  for (int c = 0; c < 3; ++c) w.w[c] = g[c] * k;
  const unsigned up =
      (r.d[0] > 0.f ? 1u : 0u) | (r.d[1] > 0.f ? 2u : 0u) | (r.d[2] > 0.f ? 4u : 0u);
  w.side = 0x010101u * (any ? 0x3fu : up | (~up & 7u) << 3) | (flat ? kRayFlat : 0u);
  return ok;
}

// Whether a tree takes rays from this origin over its wide nodes.
__device__ __forceinline__ bool wide_origin(const DevScene& S, const float* o) {
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) ok = ok && o[c] >= S.wide_lo[c] && o[c] <= S.wide_hi[c];
  return ok;
}

// Node visits between two votes: 2 against 1 saves the loop's overhead (camera
// rays 131.6 -> 128.3 us, random any hit 408 -> 401 us, 24 batches 629 -> 614
// us); at 3 the path stages lose 5% to idle lanes.
constexpr int kWideVisits = 2;

struct Words8 {
  uint32_t x[8];
};
__device__ __forceinline__ Words8 load_words8(const void* p) {
  Words8 r;
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r.x[0]), "=r"(r.x[1]), "=r"(r.x[2]), "=r"(r.x[3]), "=r"(r.x[4]), "=r"(r.x[5]),
        "=r"(r.x[6]), "=r"(r.x[7])
      : "l"(p));
  return r;
}
__device__ __forceinline__ __half2 as_half2(uint32_t x) {
  __half2 h;
  memcpy(&h, &x, 4);
  return h;
}
__device__ __forceinline__ uint32_t as_word(__half2 h) {
  uint32_t x;
  memcpy(&x, &h, 4);
  return x;
}

// refs a, b where the packed comparison near <= far holds, else kDone
__device__ __forceinline__ void keep_hit(__half2 near, __half2 far, int& a, int& b) {
  asm("{\n\t.reg .pred p, q;\n\tsetp.le.f16x2 p|q, %2, %3;\n\t"
      "selp.b32 %0, %0, 0x7fffffff, p;\n\tselp.b32 %1, %1, 0x7fffffff, q;\n\t}"
      : "+r"(a), "+r"(b)
      : "r"(as_word(near)), "r"(as_word(far)));
}

// A lane's stack of refs in shared memory: `top` is the shared-memory address
// of the next entry, entries `step` bytes apart (one column per thread).
struct WideStack {
  uint32_t base, top, step;
  __device__ __forceinline__ void init(int* column, int stride) {
    base = (uint32_t)__cvta_generic_to_shared(column);
    step = (uint32_t)stride * 4u;
    top = base;
  }
  // empties it down to its end mark, which the last pop returns
  __device__ __forceinline__ void reset() {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(base), "r"(kDone) : "memory");
    top = base + step;
  }
  __device__ __forceinline__ int pop() {
    int r;
    top -= step;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(top) : "memory");
    return r;
  }
  // stores x beyond the top and keeps it there unless it is kDone
  __device__ __forceinline__ void push_hit(int x) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tst.shared.u32 [%0], %1;\n\t"
        "setp.ne.s32 p, %1, 0x7fffffff;\n\t@p add.u32 %0, %0, %2;\n\t}"
        : "+r"(top)
        : "r"(x), "r"(step)
        : "memory");
  }
};

// One wide node: the children hit are pushed, last to visit first, and the
// top of the stack (a child, or an older ref when none was hit) is popped.
// slots: an any-hit ray, known where the code is compiled - its order is the
// slots' own.  FLAT: the ray may be flat on some axis (told by its slope there).
template <bool FLAT>
__device__ __forceinline__ void wide_visit(const DevScene& S, const Ray& r, const WideRay& w,
                                           bool slots, int& ref, WideStack& st) {
  const char* p = reinterpret_cast<const char*>(S.wide) + 96 * (size_t)ref;
  const Words8 u0 = load_words8(p), u1 = load_words8(p + 32), u2 = load_words8(p + 64);
  const float gs = __uint_as_float(u0.x[3]);
  float o[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) o[c] = __fmaf_rn(r.o[c], gs, -__uint_as_float(u0.x[c]));
  // time of the point closest to the cube's centre, in cube units
  const float tm = __fmaf_rn(o[0], w.w[0], __fmaf_rn(o[1], w.w[1], o[2] * w.w[2]));
  const __half2 lo =
      __float2half2_rn(__fmaf_rn(kTEpsilon * w.dm, gs, -1.f / 256 - tm));
  const __half2 hi = __float2half2_rn(__fmaf_rn(r.minT * w.dm, gs, 1.f / 256 - tm));
  const __half2 far = __float2half2_rn(fabsf(tm) * kWide32);
  __half2 near01 = lo, near23 = lo, far01 = hi, far23 = hi;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float at = FLAT && w.A[c] == kWideSlope ? 0.f : tm;
    const __half2 b = __float2half2_rn(__fmaf_rn(-o[c], w.A[c], -at));
    const __half2 c01 = as_half2(c == 0 ? u1.x[0] : c == 1 ? u1.x[2] : u1.x[4]);
    const __half2 c23 = as_half2(c == 0 ? u1.x[1] : c == 1 ? u1.x[3] : u1.x[5]);
    const __half2 h01 = as_half2(c == 0 ? u1.x[6] : c == 1 ? u2.x[0] : u2.x[2]);
    const __half2 h23 = as_half2(c == 0 ? u1.x[7] : c == 1 ? u2.x[1] : u2.x[3]);
    const __half2 t01 = __hfma2(c01, w.a2[c], b), t23 = __hfma2(c23, w.a2[c], b);
    near01 = __hmax2(near01, __hfma2(h01, w.n2[c], t01));
    near23 = __hmax2(near23, __hfma2(h23, w.n2[c], t23));
    far01 = __hmin2(far01, __hfma2(h01, w.p2[c], t01));
    far23 = __hmin2(far23, __hfma2(h23, w.p2[c], t23));
  }
  int r0 = (int)u0.x[4], r1 = (int)u0.x[5], r2 = (int)u0.x[6], r3 = (int)u0.x[7];
  keep_hit(near01, __hadd2(far01, far), r0, r1);
  keep_hit(near23, __hadd2(far23, far), r2, r3);
  if (slots) {
    st.push_hit(r3);
    st.push_hit(r2);
    st.push_hit(r1);
    st.push_hit(r0);
  } else {
    // the binary order: within each side, then the sides
    const unsigned m = u2.x[4] & w.side;
    const bool f0 = (m & 0xffu) != 0u, f1 = (m & 0xff00u) != 0u, f2 = (m & 0xff0000u) != 0u;
    const int a0 = f1 ? r0 : r1, a1 = f1 ? r1 : r0;
    const int b0 = f2 ? r2 : r3, b1 = f2 ? r3 : r2;
    st.push_hit(f0 ? b1 : a1);
    st.push_hit(f0 ? b0 : a0);
    st.push_hit(f0 ? a1 : b1);
    st.push_hit(f0 ? a0 : b0);
  }
  ref = st.pop();
}

// A leaf's triangles; the first accepted hit is preceded by the leaf's exact
// box test with the minT the leaf was entered with.  Pops the next ref.
template <int KIND, bool FLAT>
__device__ __forceinline__ void wide_leaf(const DevScene& S, Ray& r, unsigned& side, Hit& h,
                                          bool any, int& ref, WideStack& st) {
  const int first = ~ref;
  const float4* p = S.tris + 3 * (size_t)first;
  bool in_box = false;
  for (int pos = first;; ++pos) {
    bool last;
    const float t_in = r.minT;
    Hit n;
    const bool hit = tri_test<KIND>(r, p, n, last);
    if (hit) {
      if (!in_box) {
        const Words8 b = load_words8(S.leaf_box + 2 * (size_t)first);
        const float t_hit = r.minT;
        r.minT = t_in;
        float te;
        in_box = box_test(r, __uint_as_float(b.x[0]), __uint_as_float(b.x[1]),
                          __uint_as_float(b.x[2]), __uint_as_float(b.x[3]),
                          __uint_as_float(b.x[4]), __uint_as_float(b.x[5]), te);
        if (!in_box) break;
        if (FLAT && (side & (kRayFlat | kRayExact)) == kRayFlat) {
          bool on = false;
#pragma unroll
          for (int c = 0; c < 3; ++c)
            on = on || (fabsf(r.inv[c]) == INFINITY && (r.o[c] == __uint_as_float(b.x[c]) ||
                                                        r.o[c] == __uint_as_float(b.x[3 + c])));
          if (on) {  // again from the root record (its root box was hit)
            side |= kRayExact;
            ref = 0;
            st.reset();
            return;
          }
        }
        r.minT = t_hit;
      }
      h = n;
      h.pos = pos;
      if (any) {
        ref = kDone;
        return;
      }
    }
    if (last) break;
    p += 3;
  }
  ref = st.pop();
}

// One node record, with the exact tests, for rays outside the wide bounds.
__device__ __forceinline__ void exact_visit(const DevScene& S, const Ray& r, bool fast, bool any,
                                            int& ref, WideStack& st) {
  const float4* p = S.nodes + 4 * (size_t)ref;
  const float4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
  const int4 q3 = __ldg(reinterpret_cast<const int4*>(p + 3));
  float tl, tr;
  bool hl, hr;
  box_pair(r, fast, q0, q1, q2, hl, hr, tl, tr);
  if (hl && hr) {
    const bool left_first = any ? ((q3.z >> 2) & 1) != 0 : pick3(r.d, q3.z & 3) > 0.f;
    st.push_hit(left_first ? q3.y : q3.x);
    ref = left_first ? q3.x : q3.y;
  } else {
    ref = hl ? q3.x : hr ? q3.y : st.pop();
  }
}

// A lane's exact visits to its next leaf or its end, as the binary walk's step.
__device__ __forceinline__ void exact_descend(const DevScene& S, const Ray& r, bool any, int& ref,
                                              WideStack& st) {
  const bool fast = inv_finite(r);
  while ((unsigned)ref < (unsigned)kDone) exact_visit(S, r, fast, any, ref, st);
}

// A ray's start: root box and walk.  ref = kDone when the ray is finished.  The
// column's first entry is the end mark that the last pop returns.
__device__ __forceinline__ void wide_start(const DevScene& S, Ray& r, bool any, WideRay& w,
                                           Hit& h, int& ref, WideStack& st) {
  int sp;
  start_ray(S, r, h, ref, sp);
  if (ref == kDone) return;
  if (!(wide_setup(r, any, w) && wide_origin(S, r.o))) w.side |= kRayExact;
  st.reset();
}

// The exact walk of a tree to its end, from `ref` on.  A call: inlined with its
// loops in the two-level reflection kernel it took the frame from 4.2 to 5.0 ms.
template <int KIND, bool ANY>
__device__ __noinline__ Hit exact_trace(const float4* nodes, const float4* tris,
                                        const float4* leaf_box, int ref, Ray r, Hit h,
                                        WideStack st) {
  DevScene S;
  S.nodes = nodes;
  for (;;) {
    exact_descend(S, r, ANY, ref, st);
    if (ref == kDone) return h;
    const float4 a = __ldg(leaf_box + 2 * (size_t)(~ref));
    const float4 b = __ldg(leaf_box + 2 * (size_t)(~ref) + 1);
    float te;
    if (box_test(r, a.x, a.y, a.z, a.w, b.x, b.y, te)) {
      const float4* p = tris + 3 * (size_t)(~ref);
      for (bool last = false; !last; p += 3) {
        const bool hit = tri_test<KIND>(r, p, h, last);
        if (hit) h.pos = (int)((p - tris) / 3);
        if (ANY && hit) return h;
      }
    }
    ref = st.pop();
  }
}

// One lane's walk of a tree to its end, for kernels that trace a ray at a time,
// its direction prepared (dir_ok: wide_setup's result).  FLAT: flat rays over the
// wide nodes too; the frame kernels, whose pinhole and shadow rays are hardly ever
// flat, send them to the exact walk and save the code.
template <int KIND, bool ANY, bool FLAT>
__device__ __forceinline__ void wide_trace(const DevScene& S, Ray& r, const WideRay& w,
                                           bool dir_ok, Hit& h, int ref, WideStack& st) {
  if (ref == kDone) return;
  st.reset();
  unsigned side = w.side;
  if (dir_ok && (FLAT || !(side & kRayFlat)) && wide_origin(S, r.o)) {
    DevScene L;
    L.wide = S.wide;
    L.tris = S.tris;
    L.leaf_box = S.leaf_box;
    do {
      while ((unsigned)ref < (unsigned)kDone) wide_visit<FLAT>(L, r, w, ANY, ref, st);
      if (ref < 0) wide_leaf<KIND, FLAT>(L, r, side, h, ANY, ref, st);
    } while (ref != kDone && !(FLAT && (side & kRayExact)));
    if (ref == kDone) return;
  }
  h = exact_trace<KIND, ANY>(S.nodes, S.tris, S.leaf_box, ref, r, h, st);
  if (h.id >= 0) r.minT = h.t;
}

// Node visits of a whole warp until `vote` of its live lanes wait at a leaf
// or at their end.
template <bool FLAT>
__device__ __forceinline__ void wide_descend(const DevScene& S, const Ray& r, const WideRay& w,
                                             bool live, int vote, bool slots, int& ref,
                                             WideStack& st) {
  const int stop = max(0, __popc(__ballot_sync(0xffffffffu, live)) - vote);
  while (__popc(__ballot_sync(0xffffffffu, live && (unsigned)ref < (unsigned)kDone)) > stop) {
#pragma unroll
    for (int k = 0; k < kWideVisits; ++k)
      if (live && (unsigned)ref < (unsigned)kDone) wide_visit<FLAT>(S, r, w, slots, ref, st);
  }
}

// Flat rays are parallel as a rule and reach their leaves together: 3 M vertical
// rays over 295 k triangles 271 -> 237 us against the caller's 12.
constexpr int kFlatVote = 24;

// wide_descend, then the leaves waiting.  Called by all 32 lanes.  A warp with
// flat or exact rays takes loops of its own: the exact lanes go to their next
// leaf first.
template <int KIND>
__device__ __forceinline__ void wide_step(const DevScene& S, Ray& r, WideRay& w, Hit& h,
                                          bool any, bool live, int vote, bool slots,
                                          int& ref, WideStack& st) {
  if (__any_sync(0xffffffffu, live && w.side >= kRayFlat)) {
    const bool exact = live && (w.side & kRayExact) != 0u;
    if (exact) exact_descend(S, r, any, ref, st);
    __syncwarp();
    wide_descend<true>(S, r, w, live && !exact, max(vote, kFlatVote), slots, ref, st);
  } else {
    wide_descend<false>(S, r, w, live, vote, slots, ref, st);
  }
  if (live && ref < 0) wide_leaf<KIND, true>(S, r, w.side, h, any, ref, st);
}

// The two walks behind one interface, for kernels whose warps keep one ray per
// lane in flight: init once, start per ray (ref = kDone when it is finished
// already), step by the whole warp with `live` where ref != kDone (slots: every
// ray is an any-hit ray, said where the code is compiled).

// Binary walk over the node records, R stack entries in registers; a step of
// a lane runs to its next leaf and through it.
template <int KIND_, bool STATS_, int R>
struct BinaryWalk {
  static constexpr int KIND = KIND_;
  static constexpr bool STATS = STATS_, WIDE = false;
  RegStack<R> st;
  Counts cnt;
  __device__ __forceinline__ void init(void* smem) {
    st.init(static_cast<int2*>(smem) + threadIdx.x, blockDim.x);
  }
  __device__ __forceinline__ void start(const DevScene& S, Ray& r, bool any, Hit& h, int& ref) {
    start_ray(S, r, h, ref, st.sp);
    st.nreg = 0;
    if (STATS) cnt.boxes += 1;
  }
  __device__ __forceinline__ void step(const DevScene& S, Ray& r, Hit& h, bool any, bool live,
                                       int vote, int& ref, bool slots = false) {
    if (live) step_dyn<KIND, R, STATS>(S, r, h, ref, st, any, &cnt);
  }
};

// Wide walk; needs S.wide.
template <int KIND_>
struct WideWalk {
  static constexpr int KIND = KIND_;
  static constexpr bool STATS = false, WIDE = true;
  WideStack st;
  WideRay w;
  Counts cnt;  // stays zero
  __device__ __forceinline__ void init(void* smem) {
    st.init(static_cast<int*>(smem) + threadIdx.x, blockDim.x);
  }
  __device__ __forceinline__ void start(const DevScene& S, Ray& r, bool any, Hit& h, int& ref) {
    wide_start(S, r, any, w, h, ref, st);
  }
  __device__ __forceinline__ void step(const DevScene& S, Ray& r, Hit& h, bool any, bool live,
                                       int vote, int& ref, bool slots = false) {
    wide_step<KIND>(S, r, w, h, any, live, vote, slots, ref, st);
  }
};

// The pointers a walk's steps follow, copied from a scene table in shared
// memory.
template <class Walk>
__device__ __forceinline__ DevScene walk_scene(const DevScene& s) {
  DevScene S;
  S.tris = s.tris;
  S.nodes = s.nodes;
  if (Walk::WIDE) {
    S.wide = s.wide;
    S.leaf_box = s.leaf_box;
  }
  return S;
}

}  // namespace rq
