// CUDA kernels of the nBounce path-tracing pass for sm_103a.
//
// The reference runs one WGSL invocation per pixel that loops over bounces with the whole
// traversal inline (pathtracing.wgsl:161-260).  Here the pass is a wavefront:
//   raygen      one path per (pixel, sample) of a batch: Cranley-Patterson-rotated Sobol
//               jitter and generate_ray (pathtracing.wgsl:27-41, 245-255), queued in 8x8
//               pixel tiles
//   trace       persistent warps take 32 rays at a time with one atomic and walk 8-wide
//               quantised trees (raytracing_sw.wgsl:176-319): BLASes collapsed from the
//               reference's, a TLAS over tight world boxes of the instances (large instances
//               split at their BLAS root).  One node load (80 bytes) tests eight child boxes; hit
//               children are pushed in distance order so the nearest is visited next, then the
//               node's hit leaf triangles are tested
//   shade       hit attributes (raytracing_sw.wgsl:138-173), env/emission termination, lobe
//               choice, VNDF / cosine sampling, Russian roulette (pathtracing.wgsl:161-241);
//               each block appends its survivors to the next bounce's queue grouped by
//               direction bin (one atomic per block)
//   paths       queues too short to fill the GPU: 8 lanes per path run it to its end, traversal and
//               shading, in one launch (nb_group.cuh)
//   accumulate  running mean over the batch's samples in sample order (pathtracing.wgsl:258)
// so traversal runs in a lean kernel and the path state lives in HBM.  A wave can hold paths
// of several jobs (render requests): tables of segments, jobs and scenes ride in the kernel
// parameters and each path finds its job through its path id.
//
// The traversal finds the reference's closest hit: quantised BLAS boxes contain the reference
// boxes, TLAS boxes contain each instance's geometry, triangles are tested with the
// reference's Moller-Trumbore arithmetic, and a hit replaces the current one only when
// strictly closer.  Visiting order differs from the
// reference (8-wide nodes, BLAS nodes pruned by the running closest hit where the reference
// restarts each BLAS from NO_HIT, raytracing_sw.wgsl:255), so among triangles at exactly the
// same distance another one may win: the documented near-tie class.

#include <algorithm>
#include <cstdint>

#include "nb_device.cuh"
#include "nb_launch.h"
#include "nb_mlp.cuh"

namespace nbd {

using nb::JobParams;
using nb::kMaxBounceSlots;
using nb::PathBatch;
using nb::Segment;
using nb::ShadowQueue;
using nb::WaveTables;

constexpr int kStackSize = 64;
constexpr uint32_t kIterationCap = 1u << 22;
constexpr uint32_t kInstanceBit = 0x80000000u;

__device__ __forceinline__ float4 ld4(const float4* p) { return __ldg(p); }
__device__ __forceinline__ uint32_t f2u(float x) { return __float_as_uint(x); }
// A 32-byte sector in one load (32-byte aligned).
struct F8 {
  float4 a, b;
};
__device__ __forceinline__ F8 ld8(const float4* p) {
  F8 v;
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.a.w), "=f"(v.b.x), "=f"(v.b.y), "=f"(v.b.z), "=f"(v.b.w)
      : "l"(p));
  return v;
}

// The first sector of a WideNode.  Its integers are loaded as integers: of a loaded float's bits
// the compiler may make a float negation where the sign bit is added, and that changes a NaN's bits.
struct NodeHead {
  V3 p;
  uint32_t bits, child_base, leaf_base;
  float step_x, step_y;
  __device__ __forceinline__ float step_z() const { return __uint_as_float(bits & 0x7F800000u); }
};
__device__ __forceinline__ NodeHead load_head(const float4* node) {
  NodeHead h;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(h.p.x), "=f"(h.p.y), "=f"(h.p.z), "=r"(h.bits), "=r"(h.child_base), "=r"(h.leaf_base), "=f"(h.step_x), "=f"(h.step_y)
      : "l"(node));
  return h;
}

// Direction reciprocal for box tests only: components below 2e-20 in magnitude are nudged to
// +-2e-20 so that every plane distance stays finite (triangle tests use the true direction).
// The hardware's approximate reciprocal (relative error <= 2^-23, no slow path) instead of a
// correctly rounded division: the box test's per-axis margins cover the extra rounding (see
// trace_step), and the correctly rounded division cost 2.2 ms of the benchmark frame's traversal.
__device__ __forceinline__ float safe_rcp(float d) {
  const float m = 2e-20f;
  const float x = fabsf(d) < m ? copysignf(m, d) : d;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct Hit {
  float t, u, v;
  uint32_t tri, inst;
};

// Two floats in a register pair and arithmetic on both: one instruction for two IEEE operations,
// each rounded as the scalar one.
struct F2 {
  uint64_t r;
};
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v.r) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ F2 pack2(uint32_t lo, uint32_t hi) {
  F2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v.r) : "r"(lo), "r"(hi));
  return v;
}
__device__ __forceinline__ float2 unpack2(F2 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v.r));
  return f;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v.r) : "l"(a.r), "l"(b.r), "l"(c.r));
  return v;
}
// The product is taken as fma(a, b, -0), the same value and sign: a packed multiplication that meets
// a packed addition is contracted into one FMA even with -fmad=false (and so is one whose -0 the
// compiler can see, hence the constant bank), which would change the hit's bits.
__constant__ float2 kNegZero2 = {-0.0f, -0.0f};
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return fma2(a, b, pack2(kNegZero2.x, kNegZero2.y)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v.r) : "l"(a.r), "l"(b.r));
  return v;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 v;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v.r) : "l"(a.r), "l"(b.r));
  return v;
}
// A plane byte q as the float offset + q: a byte product added to the offset's bits.  The products run
// beside the ALU pipe, which bounds the traversal of camera rays (75% of its peak, the FMA pipes 25%):
// against byte permutes on that pipe, and the maximum of three and the hit test on it too, 1920x1080 at
// 64 spp 101.3 -> 93.9 ms, camera rays on the 1M-triangle soup 2.52 -> 2.33.
// Near planes have offset 2^15, bits 0x47000000 + (q << 8) by a product of 16-bit weights held in
// registers.  Their rounding is part of the answer: a child's entry distance decides the order of
// overlapping children and with it which of two triangles at the same distance is found, and the group
// kernels (GroupTrace) have the same offset, so that a hit does not depend on the size of the call.  Far planes
// only decide whether a box is opened, with a margin (trace_step) for any rounding.  For closest hits
// they have offset 2^16, bits 0x47800000 + (q << 7), whose weight fits a byte, an immediate: 1920x1080 at
// 64 spp 91.1 -> 89.4 ms, camera rays 2.29 -> 2.28.  (Near planes that way too: 88.2 and 2.25, but another
// triangle for one in 170,000 rays on coincident surfaces.)  Any-hit queries take 2^15 for both: scattered
// rays 3.57 ms, with 2^16 for the far planes 3.62.
template <bool kAny>
struct Planes {
  static constexpr float kOffset = 32768.0f;
  static __device__ __forceinline__ uint32_t decode(uint32_t w, int k) {
    const uint32_t weight = (k & 1) ? 0x01000000u : 0x100u;
    return (k & 2) ? __dp2a_hi(weight, w, 0x47000000u) : __dp2a_lo(weight, w, 0x47000000u);
  }
  // byte k of a near and a far word
  static __device__ __forceinline__ F2 pair(uint32_t n, uint32_t f, int k) {
    return pack2(decode(n, k), kAny ? decode(f, k) : __dp4a(f, 0x80u << (8 * k), 0x47800000u));
  }
  // the far planes' constant from c, the one with offset 2^15, and the near planes' margin d
  static __device__ __forceinline__ float far(float a, float c, float d) {
    return kAny ? c + d : fmaf(-32768.0f, a, fmaf(2.0f, d, c));
  }
};
// maximum and minimum of three, as fmaxf and fminf of two treat NaN
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
struct V3x2 {
  F2 x, y, z;
};
__device__ __forceinline__ V3x2 both(V3 v) { return V3x2{pack2(v.x, v.x), pack2(v.y, v.y), pack2(v.z, v.z)}; }
__device__ __forceinline__ V3x2 operator-(V3x2 a, V3x2 b) { return V3x2{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F2 dot(V3x2 a, V3x2 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3x2 cross(V3x2 a, V3x2 b) {
  return V3x2{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// Moller-Trumbore (raytracing_sw.wgsl:51-78) on the two triangles of a leaf slot at once
// (GpuTriPair): the operations and roundings of the two tests one after the other.  Calls
// hit(t, u, v, triangle) for the first if it is closer than t_max, then for the second if it is
// closer than that.  The records' loads are issued together and the arithmetic is packed, so a slot
// costs one round trip and about 90 instructions instead of two and 130.
template <class OnHit>
__device__ __forceinline__ void triangle_pair_test(V3 ro, V3 rd, const float4* p, float t_max, OnHit hit) {
  const F8 s0 = ld8(p), s1 = ld8(p + 2);
  const float4 p0 = s0.a, p1 = s0.b, p2 = s1.a, p3 = s1.b, p4 = ld4(p + 4);
  const V3x2 v0{pack2(p0.x, p0.y), pack2(p0.z, p0.w), pack2(p1.x, p1.y)};
  const V3x2 e1{pack2(p1.z, p1.w), pack2(p2.x, p2.y), pack2(p2.z, p2.w)};
  const V3x2 e2{pack2(p3.x, p3.y), pack2(p3.z, p3.w), pack2(p4.x, p4.y)};
  const V3x2 d = both(rd);
  const V3x2 hv = cross(d, e2);
  const F2 det2 = dot(e1, hv);
  const float2 det = unpack2(det2);
  const bool back0 = det.x < kEps, back1 = det.y < kEps;
  if (back0 && back1) return;
  // a det that counts is >= kEps; 1 / det correctly rounded, as the reference arithmetic divides
  float2 inv{rcp_newton(det.x), rcp_newton(det.y)};
  if (!(fmaxf(det.x, det.y) < kRcpNewtonMax)) inv = make_float2(1.0f / det.x, 1.0f / det.y);
  const F2 inv2 = pack2(inv.x, inv.y);
  const V3x2 sv = both(ro) - v0;
  const F2 u2 = inv2 * dot(sv, hv);
  const V3x2 q = cross(sv, e1);
  const F2 v2 = inv2 * dot(d, q);
  const float2 u = unpack2(u2), v = unpack2(v2), uv = unpack2(u2 + v2);
  const bool out0 = back0 || u.x < 0.0f || u.x > 1.0f || v.x < 0.0f || uv.x > 1.0f;
  const bool out1 = back1 || u.y < 0.0f || u.y > 1.0f || v.y < 0.0f || uv.y > 1.0f;
  if (out0 && out1) return;
  const float2 t = unpack2(inv2 * dot(e2, q));
  if (!out0 && !(t.x < kBias) && t.x < t_max) {
    t_max = t.x;
    hit(t.x, u.x, v.x, f2u(p4.z));
  }
  if (!out1 && !(t.y < kBias) && t.y < t_max) hit(t.y, u.y, v.y, f2u(p4.w));
}

// Traversal state of one ray: the world ray, the current ray (world, or instance-local inside
// a BLAS), the distance of the closest hit so far and the depth of the stack both levels share.
// The stack itself is a separate per-thread array, so that these scalars stay in registers;
// the rest of the hit record (u, v, triangle, instance), written only when a closer hit is
// found, lives in two extra slots at the end of that array (kHitSlot), and the world ray's
// reciprocal direction is recomputed when a BLAS is left - both to keep the state within the
// register budget (kRefillBlocks, kChunkBlocks).
constexpr int kHitSlot = kStackSize;  // stack[kHitSlot] = (u, v), stack[kHitSlot + 1] = (tri, inst)
struct TraceState {
  V3 wo, wd;
  V3 ro, rd, rinv;
  float t_hit;
  float next_d;                  // have_node: distance of the pending node
  int sp, blas_base;
  uint32_t cur_inst, node, iter, status;
  uint32_t leaf_mask, leaf_base; // slots of the last node still to test: slot k is record leaf_base + k
  bool in_blas, have_node;
};

__device__ __forceinline__ void trace_begin(TraceState& t, uint2* stack, const DevScene& s, const V3 wo,
                                            const V3 wd) {
  t.t_hit = kNoHit;
  stack[kHitSlot] = make_uint2(0u, 0u);
  stack[kHitSlot + 1] = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
  t.status = 0;
  t.wo = wo;
  t.wd = wd;
  t.ro = wo;
  t.rd = wd;
  t.rinv = V3{safe_rcp(wd.x), safe_rcp(wd.y), safe_rcp(wd.z)};
  t.sp = 0;
  t.blas_base = 0;
  t.in_blas = false;
  t.cur_inst = 0;
  t.node = 0;  // the TLAS root
  // no TLAS, or a ray with a NaN or infinite component: nothing to hit (every slab and
  // triangle comparison of the reference fails on NaN; the box test below relies on it)
  const float fin = fabsf(wo.x) + fabsf(wo.y) + fabsf(wo.z) + fabsf(wd.x) + fabsf(wd.y) + fabsf(wd.z);
  t.have_node = s.has_tlas != 0u && fin <= 3.4028235e38f;
  t.next_d = 0.0f;
  t.leaf_mask = t.leaf_base = 0;
  t.iter = 0;
}

// Where trace_step reads the world ray and its box-test reciprocal when it enters or leaves an
// instance.  A per-warp array in shared memory, component-major so that the 32 lanes' loads hit
// distinct banks, kWorldFloats floats: origin, direction, reciprocal direction x 32 lanes.
//   WorldShared  all three in shared memory: keeps six registers free in the lane-refill
//                kernels, whose register budget is tightest;
//   WorldMixed   origin and direction in registers, the reciprocal in shared memory (the
//                camera-ray kernel, which enters and leaves instances at most steps);
//   WorldRegs    origin and direction in registers, the reciprocal recomputed (caller rays
//                without refill).
// Keeping the reciprocal instead of recomputing it when a BLAS is left measured 2.3 ms faster
// traversal on the benchmark frame.
constexpr int kWorldFloats = 9 * 32;
constexpr int kTraceWarps = 4;  // every traversal kernel runs blocks of 128 threads
constexpr int kTraceThreads = 32 * kTraceWarps;
// Blocks per SM of the traversal kernels: with lane refill 7 (72 registers), whole-warp chunks 6 (80), of
// closest-hit queries 7 (kQueryBlocks).  Camera grids of 2048x2048 with 6 / 7: closest hits on soups of 1M, 200K and 20K
// triangles 2.28 / 2.23, 2.07 / 2.03 and 0.72 / 0.71 ms, on the instanced scene 1.35 / 1.32; any hits
// 2.02 / 2.03, 2.04 / 2.06, 0.74 / 0.75 and 1.11 / 1.14, and a render's camera rays with 7 no faster than with
// 6.  1920x1080 at 64 spp and scattered any hit, refill and chunk blocks 8+7: 103.5 and 4.79 ms, 7+6: 90.9
// and 3.59, 6+5: 94.4 and 3.77.
constexpr int kRefillBlocks = 7, kChunkBlocks = 6, kQueryBlocks = 7;
struct WorldRegs {
  const TraceState& t;
  __device__ __forceinline__ V3 o() const { return t.wo; }
  __device__ __forceinline__ V3 d() const { return t.wd; }
  __device__ __forceinline__ V3 inv() const { return V3{safe_rcp(t.wd.x), safe_rcp(t.wd.y), safe_rcp(t.wd.z)}; }
};
// a warp's reciprocal directions: kInvFloats floats, component-major
constexpr int kInvFloats = 3 * 32;
__device__ __forceinline__ V3 world_inv(const float* w) {
  const uint32_t l = threadIdx.x & 31u;
  return V3{w[l], w[32 + l], w[64 + l]};
}
__device__ __forceinline__ void set_world_inv(float* w, V3 r) {
  const uint32_t l = threadIdx.x & 31u;
  w[l] = r.x; w[32 + l] = r.y; w[64 + l] = r.z;
}
struct WorldMixed {
  const TraceState& t;
  const float* w;  // kInvFloats
  __device__ __forceinline__ V3 o() const { return t.wo; }
  __device__ __forceinline__ V3 d() const { return t.wd; }
  __device__ __forceinline__ V3 inv() const { return world_inv(w); }
};
struct WorldShared {
  float* w;
  __device__ __forceinline__ V3 o() const {
    const uint32_t l = threadIdx.x & 31u;
    return V3{w[l], w[32 + l], w[64 + l]};
  }
  __device__ __forceinline__ V3 d() const {
    const uint32_t l = threadIdx.x & 31u;
    return V3{w[96 + l], w[128 + l], w[160 + l]};
  }
  __device__ __forceinline__ V3 inv() const { return world_inv(w + 192); }
  __device__ __forceinline__ void set(V3 o, V3 d) const {
    const uint32_t l = threadIdx.x & 31u;
    w[l] = o.x; w[32 + l] = o.y; w[64 + l] = o.z;
    w[96 + l] = d.x; w[128 + l] = d.y; w[160 + l] = d.z;
  }
  __device__ __forceinline__ void set_inv(V3 r) const { set_world_inv(w + 192, r); }
};

// Where a ray's stack entries lie.  LocalStack: all in thread-local memory (whole-warp chunks: a
// warp's rays are at nearly the same depth, 92% of the loads hit L1, and a node step is then often the
// same single hit child for all lanes, which needs no sort).  SharedStack (lane refill): the first
// kSharedEntries in shared memory, entry-major (conflict-free at any mix of depths), deeper ones in
// local memory.  Scattered rays' local stacks miss L1 (16% hits on the 1M-triangle soup, half on the
// benchmark frame's bounce 1), and a pop then waits for L2 before the node's own load can start.  8 /
// 12 / 16 / 20 entries: scattered any hit on the soup 5.15 / 4.78 / 4.60 / 4.58 ms (all local 5.02),
// 1920x1080 at 64 spp 110.3 / 106.5 / 106.6 / 107.0 (110.4).  Without the single-child branch the
// scattered rays take 4.51 ms (camera rays, which keep it, 2.53 instead of 2.60).
constexpr int kSharedEntries = 16;
struct LocalStack {
  static constexpr bool kScattered = false;
  static constexpr int kFast = kStackSize, kStride = 1;
  uint2* local;
  __device__ __forceinline__ uint2* fast(int top) const { return local + top; }
  __device__ __forceinline__ uint2 get(int i) const { return local[i]; }
  __device__ __forceinline__ void put(int i, uint2 e) const { local[i] = e; }
};
struct SharedStack {
  static constexpr bool kScattered = true;
  static constexpr int kFast = kSharedEntries, kStride = kTraceThreads;
  uint2* local;
  uint2* sh;  // this thread's column
  __device__ __forceinline__ uint2* fast(int top) const { return sh + top * kStride; }
  __device__ __forceinline__ uint2 get(int i) const { return i < kFast ? sh[i * kStride] : local[i]; }
  __device__ __forceinline__ void put(int i, uint2 e) const {
    if (i < kFast) sh[i * kStride] = e;
    else local[i] = e;
  }
};

// Lane refill: a step goes on to its lanes' further leaf slots only while this many lanes have one.  The
// others keep theirs for the next step, where they share the pass with the leaves that other lanes
// reach meanwhile; testing every slot at once, most passes ran with two or three lanes.  1 (all slots) /
// 3 / 6 / 9 / 12 lanes / one pass per step: scattered any hit on the 1M-triangle soup 4.52 / 4.00 / 3.82
// / 3.82 / 3.83 / 3.75 ms, closest (1M rays) 1.54 / 1.42 / 1.37 / 1.37 / 1.38 / 1.40, 1920x1080 at
// 64 spp 105.5 / 101.6 / 101.6 / 101.7 / 101.6 / 103.0, 1013x571 at 3 spp with NEE 3.66 / 3.59 / 3.58 /
// 3.59 / 3.59 / 3.69.  Whole-warp chunks test all slots: their lanes reach the same leaves together
// (camera rays on the soup 2.53, with one pass per step 2.97).
constexpr int kLeafLanes = 6;

// Work counters of the instrumented traversal (kCount instantiations only): what the device
// layout fetches per ray - 80 bytes of the wide nodes of the TLAS and the BLASes, the triangles of
// leaf slots (80 bytes for one or two), 64-byte instance records - and the 8-byte stack entries pushed (each later popped);
// and how the lanes of a warp share the node steps: warp steps (lanes that test a node
// together count one step, recorded by the lowest of them) with their lanes, and of those the
// steps in which some lane tests leaf triangles, with the lanes that do and the largest
// triangle count among them (the warp's iterations of the leaf loop).
struct TraceCount {
  uint32_t tlas_nodes = 0, blas_nodes = 0, tris = 0, insts = 0, pushes = 0;
  uint32_t warp_steps = 0, lane_steps = 0, leaf_steps = 0, leaf_lanes = 0, leaf_trips = 0;
};
__device__ __forceinline__ bool lowest_active(uint32_t mask) {
  return (threadIdx.x & 31u) == (uint32_t)(__ffs(mask) - 1);
}

// Bound by instruction issue, latency and divergence: the schedulers issue in 71% of cycles for camera rays
// (ALU pipe 59% of its peak, 20 of 32 lanes active) and 73% for secondary rays (55%, 16 of 32; the
// benchmark scene at 480x270, 64 spp).  Run twice, the leaf tests
// add 16% to the 1080p frame (51% to scattered rays in the soup), the sort 4%, the pushes 2%.  What it costs per warp
// step is its instructions, most of them not in the box tests: a slot's triangles are tested two at a
// time (triangle_pair_test), the box tests take a child's near and far plane of an axis in one packed
// FMA, and a hit child's stack entry is one addition (the slot is the offset) stored at a fixed place below
// the batch's top.  Against one triangle at a time,
// slot metadata and a branch per pushed child, at the same sizes as above: 1920x1080 at 64 spp 116.6 ->
// 110.4 ms, camera rays on the soup 2.67 -> 2.53, scattered any hit 5.42 -> 5.02, closest (1M rays)
// 1.94 -> 1.71 ms.
//
// One traversal step: pop the next entry when no node is pending, then test one 8-wide node
// and its leaf triangles.  Returns false once the ray is finished (stack empty, an any-hit
// found, or the iteration cap reached).  wr gives the world ray (WorldRegs, WorldMixed or
// WorldShared).
template <bool kAny, bool kCount, class World, class Stack>
__device__ __forceinline__ bool trace_step(TraceState& t, const Stack& stack, const DevScene& s, TraceCount* cnt,
                                           const World& wr) {
  V3 &ro = t.ro, &rd = t.rd, &rinv = t.rinv;
  float &h_t = t.t_hit, &next_d = t.next_d;
  int &sp = t.sp, &blas_base = t.blas_base;
  bool &in_blas = t.in_blas, &have_node = t.have_node;
  uint32_t &cur_inst = t.cur_inst, &node = t.node, &status = t.status, &leaf_mask = t.leaf_mask;
  if (!Stack::kScattered || leaf_mask == 0u) {  // else the last node's leaf slots come first
    if (t.iter > kIterationCap) {
      status |= kStatusIterationCap;
      return false;
    }
    ++t.iter;
    if (have_node && next_d >= h_t) have_node = false;  // a leaf was closer than the pending node
    if (!have_node) {
      // The next entry nearer than the hit.  The loop only finds it; what the entry needs is done once
      // after the loop by all lanes together, whichever pass they left it in: the world ray is brought
      // back only for a TLAS node, an instance's ray is made from it directly.
      bool left = false;  // a BLAS was finished on the way
      uint2 e = make_uint2(0u, 0u);
      bool found = false;
      while (!found) {
        if (in_blas && sp == blas_base) {
          in_blas = false;
          left = true;
        }
        if (sp == 0) break;
        --sp;
        e = stack.get(sp);
        found = __uint_as_float(e.y & ~7u) < h_t;  // raytracing_sw.wgsl:197,271
      }
      if (!found) return false;
      node = e.x;
      if (!in_blas && (e.x & kInstanceBit)) {
        // enter an instance: transform the world ray (raytracing_sw.wgsl:202-206)
        if (kCount) ++cnt->insts;
        const float4* it = s.inst_trace + 4 * (size_t)(e.x & ~kInstanceBit);
        const F8 i0 = ld8(it), i1 = ld8(it + 2);
        const float4 r0 = i0.a, r1 = i0.b, r2 = i1.a, r3 = i1.b;
        const V3 wo = wr.o(), wd = wr.d();
        ro = V3{r0.x * wo.x + r0.y * wo.y + r0.z * wo.z + r0.w * 1.0f,
                r1.x * wo.x + r1.y * wo.y + r1.z * wo.z + r1.w * 1.0f,
                r2.x * wo.x + r2.y * wo.y + r2.z * wo.z + r2.w * 1.0f};
        rd = V3{r0.x * wd.x + r0.y * wd.y + r0.z * wd.z, r1.x * wd.x + r1.y * wd.y + r1.z * wd.z,
                r2.x * wd.x + r2.y * wd.y + r2.z * wd.z};
        rinv = V3{safe_rcp(rd.x), safe_rcp(rd.y), safe_rcp(rd.z)};
        node = f2u(r3.x);
        cur_inst = f2u(r3.y);
        in_blas = true;
        blas_base = sp;
      } else if (left) {  // back to the world ray
        ro = wr.o();
        rd = wr.d();
        rinv = wr.inv();
      }
    }
    have_node = false;

    // ---- one 8-wide node: quantised slab tests of all children ----
    if (kCount) {
      ++(in_blas ? cnt->blas_nodes : cnt->tlas_nodes);
      const uint32_t together = __activemask();
      if (lowest_active(together)) {
        ++cnt->warp_steps;
        cnt->lane_steps += (uint32_t)__popc(together);
      }
    }
    const float4* np = (in_blas ? s.blas_wide : s.tlas_wide) + 6 * (size_t)node;
    const NodeHead nh = load_head(np);
    const F8 w1 = ld8(np + 2);
    const float4 q2 = w1.a, q3 = w1.b, q4 = ld4(np + 4);
    const float ax = nh.step_x * rinv.x, ay = nh.step_y * rinv.y, az = nh.step_z() * rinv.z;
    const float bx = (nh.p.x - ro.x) * rinv.x, by = (nh.p.y - ro.y) * rinv.y, bz = (nh.p.z - ro.z) * rinv.z;
    // A plane byte q is read as the float F = P + q, P = 2^15 or, for closest hits' far planes, 2^16
    // (Planes), and its distance taken as fma(F, a, b - P a).  With u = 2^-24, the folded constant, the margin
    // added to it and the FMA are off by at most u (|b| + P |a|), u (|b| + P |a|) and u (|b| + 255 |a|), and
    // where 2^16 a is folded in two halves by u (|b| + P |a|) more at most: each plane's distance lies within
    // 1.8e-7 |b| + (2^-9 + 1.6e-5) |a| of b + q a, with 2^16 within 2.4e-7 |b| + (2^-7 + 1.6e-5) |a|.
    // Near-plane constants are lowered by d = |a| / 128 + |b| / 2^19 per axis and far-plane constants raised
    // by d, with 2^16 by 2 d.  For every plane t = b + q a of the node (|t| <= |b| + 255 |a|) the margin
    // covers that, the approximate reciprocal (<= 2^-22 |t|) and the rounding of the plane evaluation
    // against the exact reference box (4e-7 |t|): together at most 8.8e-7 |b| + (2^-9 + 1.9e-4) |a| <= d, or
    // 8.8e-7 |b| + (2^-7 + 1.9e-4) |a| <= 2 d, so a box never rejects a ray the reference box accepts.
    using Q = Planes<kAny>;
    const float dx = fmaf(fabsf(ax), 0.0078125f, fabsf(bx) * 1.9073486328125e-6f);
    const float dy = fmaf(fabsf(ay), 0.0078125f, fabsf(by) * 1.9073486328125e-6f);
    const float dz = fmaf(fabsf(az), 0.0078125f, fabsf(bz) * 1.9073486328125e-6f);
    const float cx = fmaf(-Q::kOffset, ax, bx), cy = fmaf(-Q::kOffset, ay, by), cz = fmaf(-Q::kOffset, az, bz);
    const float cnx = cx - dx, cny = cy - dy, cnz = cz - dz;
    const float cfx = Q::far(ax, cx, dx), cfy = Q::far(ay, cy, dy), cfz = Q::far(az, cz, dz);
    // near/far planes per axis by the sign of the direction: the near plane of a child is its
    // low plane where rinv >= 0 (t grows with the quantised coordinate), else its high plane
    const bool pxs = rinv.x >= 0.0f, pys = rinv.y >= 0.0f, pzs = rinv.z >= 0.0f;
    const uint32_t nx0 = pxs ? f2u(q2.x) : f2u(q3.z), nx1 = pxs ? f2u(q2.y) : f2u(q3.w);
    const uint32_t fx0 = pxs ? f2u(q3.z) : f2u(q2.x), fx1 = pxs ? f2u(q3.w) : f2u(q2.y);
    const uint32_t ny0 = pys ? f2u(q2.z) : f2u(q4.x), ny1 = pys ? f2u(q2.w) : f2u(q4.y);
    const uint32_t fy0 = pys ? f2u(q4.x) : f2u(q2.z), fy1 = pys ? f2u(q4.y) : f2u(q2.w);
    const uint32_t nz0 = pzs ? f2u(q3.x) : f2u(q4.z), nz1 = pzs ? f2u(q3.y) : f2u(q4.w);
    const uint32_t fz0 = pzs ? f2u(q4.z) : f2u(q3.x), fz1 = pzs ? f2u(q4.w) : f2u(q3.y);
    // a child is hit when max(tn, 0) <= min(tf, the largest float below the closest hit)
    const float t_below = __uint_as_float(f2u(h_t) - 1u);  // h_t > 0
    // a child's near and far plane of an axis in one packed FMA
    const F2 ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
    const F2 cx2 = pack2(cnx, cfx), cy2 = pack2(cny, cfy), cz2 = pack2(cnz, cfz);
    uint32_t key[8];
    uint32_t misses = 0;
#pragma unroll
    for (int k = 7; k >= 0; --k) {
      const float2 tx = unpack2(fma2(Q::pair(k < 4 ? nx0 : nx1, k < 4 ? fx0 : fx1, k & 3), ax2, cx2));
      const float2 ty = unpack2(fma2(Q::pair(k < 4 ? ny0 : ny1, k < 4 ? fy0 : fy1, k & 3), ay2, cy2));
      const float2 tz = unpack2(fma2(Q::pair(k < 4 ? nz0 : nz1, k < 4 ? fz0 : fz1, k & 3), az2, cz2));
      const float lo = max3(fmaxf(tx.x, ty.x), tz.x, 0.0f);
      const float hi = min3(fminf(tx.y, ty.y), tz.y, t_below);
      // lo <= hi as the sign of hi - lo: neither is NaN, lo is >= +0 and hi never -0: the margin, >= +0, is in
      // its constant (and sums of these products are exact where they are denormal)
      misses = __funnelshift_l(f2u(hi - lo), misses, 1);
      key[k] = (f2u(lo) & ~7u) | (uint32_t)k;
    }
    const uint32_t hits = ~misses & nh.bits & 0xFFu;
    const uint32_t inner = in_blas ? nh.bits >> 8 : 0xFFu;  // children that are visited, not tested
    leaf_mask = hits & ~inner;
    t.leaf_base = nh.leaf_base;
    const uint32_t push_mask = hits & inner;
    const int n_push = __popc(push_mask);
#pragma unroll
    for (int k = 0; k < 8; ++k) key[k] = (push_mask & (1u << k)) ? key[k] : 0xFFFFFFFFu;

    // The hit children are ordered and pushed before the node's leaf triangles are tested:
    // the keys' registers are free again during the triangle loads (measured 1.6% faster than
    // testing leaves first).  A leaf hit closer than the child visited next drops that child.
    // ---- order hit children near to far (19-comparator network) ----
#define NB_CX(i, j)                                  \
{                                                  \
    const uint32_t lo_ = min(key[i], key[j]);        \
    key[j] = max(key[i], key[j]);                    \
    key[i] = lo_;                                    \
  }
    if (n_push > 0) {
      if (!Stack::kScattered && n_push == 1) {  // the single hit child: no sort
#pragma unroll
        for (int k = 1; k < 8; ++k) key[0] = min(key[0], key[k]);
      } else {
        NB_CX(0, 2) NB_CX(1, 3) NB_CX(4, 6) NB_CX(5, 7)
        NB_CX(0, 4) NB_CX(1, 5) NB_CX(2, 6) NB_CX(3, 7)
        NB_CX(0, 1) NB_CX(2, 3) NB_CX(4, 5) NB_CX(6, 7)
        NB_CX(2, 4) NB_CX(3, 5)
        NB_CX(1, 4) NB_CX(3, 6)
        NB_CX(1, 2) NB_CX(3, 4) NB_CX(5, 6)
      }
      // a child's stack entry: node or instance index and its key (its slot in the low 3 bits).  (Which of the
      // two by the mask, since a TLAS node's slots mix them.  With the inner children first and a comparison
      // 1920x1080 at 64 spp takes 0.4 ms less, camera rays on the soup 0.02, scattered any hit the same, but then an inner child came before an instance at the same distance, whatever their places in the tree.)
      const uint32_t inst_base = kInstanceBit + nh.leaf_base;
      auto entry = [&](uint32_t kk) {
        const uint32_t slot = kk & 7u;
        return make_uint2(((nh.bits & (0x100u << slot)) ? nh.child_base : inst_base) + slot, kk);
      };
      // far to near, the nearest at top; the nearest inner child is visited next without a push
      const int top = sp + n_push - 1;
      const uint2 first = entry(key[0]);
      have_node = !(first.x & kInstanceBit);
      if (top < Stack::kFast) {
        uint2* at = stack.fast(top);
        // (the branch over the last four: 1920x1080 at 64 spp 92.6 -> 91.0 ms, camera rays 2.29 -> 2.26;
        // over the last five and three 91.0 and 91.2, 2.23 and 2.25, scattered any hit 3.62, 3.58 against 3.59)
#pragma unroll
        for (int k = 1; k < 4; ++k)
          if (k < n_push) at[-k * Stack::kStride] = entry(key[k]);
        if (n_push > 4) {
#pragma unroll
          for (int k = 4; k < 8; ++k)
            if (k < n_push) at[-k * Stack::kStride] = entry(key[k]);
        }
        if (!have_node) at[0] = first;
        sp = have_node ? top : top + 1;
      } else {
        // one by one, the last ones only as far as they fit
#pragma unroll
        for (int k = 7; k >= 0; --k) {
          if (k >= n_push || (k == 0 && have_node)) continue;
          if (sp < kStackSize) stack.put(sp++, entry(key[k]));
          else status |= kStatusStackOverflow;
        }
      }
      if (kCount) cnt->pushes += (uint32_t)(n_push - (have_node ? 1 : 0));
      if (have_node) {
        node = first.x;
        next_d = __uint_as_float(first.y & ~7u);
      }
    }
#undef NB_CX
  }
  uint32_t together = 0, n_tris = 0;  // kCount: the lanes of this step, triangles tested by this one
  if (kCount) together = __activemask();
  // ---- BLAS leaf slots: Moller-Trumbore (raytracing_sw.wgsl:51-78, 274-286), all of the node's or as
  // many as enough lanes have (kLeafLanes) ----
  while (leaf_mask) {
    const uint32_t k = (uint32_t)(__ffs(leaf_mask) - 1);
    leaf_mask &= leaf_mask - 1;
    if (kCount) n_tris += f2u(ld4(s.tris + 6 * (size_t)(t.leaf_base + k) + 4).w) == 0xFFFFFFFFu ? 1u : 2u;
    bool found = false;
    triangle_pair_test(ro, rd, s.tris + 6 * (size_t)(t.leaf_base + k), h_t,
                       [&](float t, float u, float v, uint32_t tri) {
                         if (kAny && found) return;  // any hit: the first
                         h_t = t;
                         stack.local[kHitSlot] = make_uint2(f2u(u), f2u(v));
                         stack.local[kHitSlot + 1] = make_uint2(tri, cur_inst);
                         found = true;
                       });
    if (kAny && found) return false;
    if (Stack::kScattered && __popc(__ballot_sync(__activemask(), leaf_mask != 0u)) < kLeafLanes) break;
  }
  if (kCount) {  // closest hits only: every lane of the step comes here
    static_assert(!(kCount && kAny), "a lane whose any-hit query ends leaves the step");
    cnt->tris += n_tris;
    const uint32_t with_leaves = __ballot_sync(together, n_tris != 0u);
    const uint32_t most = __reduce_max_sync(together, n_tris);
    if (with_leaves && lowest_active(together)) {
      ++cnt->leaf_steps;
      cnt->leaf_lanes += (uint32_t)__popc(with_leaves);
      cnt->leaf_trips += most;
    }
  }
  return true;
}

// Closest (or any) hit of one world-space ray.  Returns the status bits it raised.
template <bool kAny, bool kCount = false>
__device__ __forceinline__ uint32_t trace_ray(const DevScene& s, const V3 wo, const V3 wd, Hit& h,
                                              TraceCount* cnt = nullptr) {
  TraceState t;
  uint2 stack[kStackSize + 2];
  trace_begin(t, stack, s, wo, wd);
  while (trace_step<kAny, kCount>(t, LocalStack{stack}, s, cnt, WorldRegs{t})) {
  }
  const uint2 uv = stack[kHitSlot], ti = stack[kHitSlot + 1];
  h.t = t.t_hit;
  h.u = __uint_as_float(uv.x);
  h.v = __uint_as_float(uv.y);
  h.tri = ti.x;
  h.inst = ti.y;
  return t.status;
}

// Traces rays 0 .. n-1 of a queue with one warp, refilling lanes: a lane whose ray finished
// takes a new one once kRefillIdle lanes of the warp are idle (a whole idle warp always takes
// 32), all of them with one atomic on *fetch.  load(r, o, d, sidx) reads ray r and its scene
// index; scene(sidx) gives that scene; finish(r, t_hit, uv, tri_inst) consumes ray r's hit
// record (t = kNoHit on a miss).  world is this warp's kWorldFloats floats of shared memory,
// where the lanes' world rays are kept (WorldShared).  Every lane of the warp must call it.
// Returns the status bits its rays raised.  Used where the rays of a warp are incoherent
// (secondary and shadow rays, caller rays): their traversal lengths differ widely, and without
// refill most lanes would idle while the longest ray of each 32 finishes.  Refill changes only
// which lane traces a ray, not its result.
constexpr uint32_t kRefillIdle = 6;
// kMixed: rays from any_from on are any-hit queries among closest-hit ones; such a ray ends with the node
// step that finds its hit.
template <bool kAny, bool kCount, bool kMixed = false, class Load, class SceneOf, class Finish>
__device__ __forceinline__ uint32_t trace_refill(uint32_t* fetch, uint32_t n, Load load, SceneOf scene, Finish finish,
                                                 TraceCount* cnt, float* world, uint2* entries,
                                                 uint32_t any_from = 0xFFFFFFFFu) {
  const WorldShared wr{world};
  const uint32_t lane = threadIdx.x & 31u;
  TraceState t;
  uint2 stack[kStackSize + 2];
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  uint32_t my = kNone, sidx = 0, st = 0;  // this lane's ray (queue index) and its scene
  bool exhausted = false;                 // warp-uniform: the queue has no rays left to take
  uint32_t idle = 0xFFFFFFFFu;            // lanes without a ray
  while (true) {
    if (!exhausted && (uint32_t)__popc(idle) >= (idle == 0xFFFFFFFFu ? 1u : kRefillIdle)) {
      const uint32_t want = (uint32_t)__popc(idle);
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, want);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base + want >= n) exhausted = true;
      if (my == kNone) {
        const uint32_t r = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
        if (r < n) {
          my = r;
          V3 o, d;
          load(r, o, d, sidx);
          trace_begin(t, stack, scene(sidx), o, d);
          wr.set(o, d);
          wr.set_inv(t.rinv);
        }
      }
    }
    if (my != kNone && (!trace_step<kAny, kCount>(t, SharedStack{stack, entries}, scene(sidx), cnt, wr) ||
                        (kMixed && my >= any_from && t.t_hit < kNoHit))) {
      finish(my, t.t_hit, stack[kHitSlot], stack[kHitSlot + 1]);
      st |= t.status;
      my = kNone;
    }
    idle = __ballot_sync(0xFFFFFFFFu, my == kNone);
    if (exhausted && idle == 0xFFFFFFFFu) break;
  }
  return st;
}

}  // namespace nbd

#include "nb_group.cuh"

namespace nbd {

// ------------------------------------------------------------------------------------------
// traversal-only query (nb_trace_rays)
// ------------------------------------------------------------------------------------------
// kRefill: lanes refill as they finish (trace_refill), for rays whose neighbours in the array
// are unrelated; else each warp traces 32 consecutive rays to the end.
template <bool kAny, bool kRefill>
__global__ void __launch_bounds__(kTraceThreads, kRefill ? kRefillBlocks : kAny ? kChunkBlocks : kQueryBlocks)
    k_trace_rays(DevScene s, const float4* __restrict__ rays, uint32_t n, float4* __restrict__ hits,
                 uint32_t* __restrict__ inst, uint32_t* __restrict__ fetch, uint32_t* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  uint32_t st = 0;
  if (kRefill) {
    __shared__ float world[kTraceWarps][kWorldFloats];
    __shared__ uint2 entries[kSharedEntries][kTraceThreads];
    st = trace_refill<kAny, false>(
        fetch, n,
        [&](uint32_t r, V3& o, V3& d, uint32_t& sidx) {
          o = xyz(__ldg(rays + 2 * (size_t)r));
          d = xyz(__ldg(rays + 2 * (size_t)r + 1));
          sidx = 0;
        },
        [&](uint32_t) -> const DevScene& { return s; },
        [&](uint32_t r, float t_hit, uint2 uv, uint2 ti) {
          hits[r] = make_float4(t_hit, __uint_as_float(uv.x), __uint_as_float(uv.y), __uint_as_float(ti.x));
          if (inst) inst[r] = ti.y;
        },
        nullptr, world[threadIdx.x >> 5], &entries[0][threadIdx.x]);
  } else {
    while (true) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, 32u);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base >= n) break;
      const uint32_t i = base + lane;
      if (i < n) {
        const float4 o = __ldg(rays + 2 * (size_t)i), d = __ldg(rays + 2 * (size_t)i + 1);
        Hit h;
        st |= trace_ray<kAny>(s, xyz(o), xyz(d), h);
        hits[i] = make_float4(h.t, h.u, h.v, __uint_as_float(h.tri));
        if (inst) inst[i] = h.inst;
      }
    }
  }
  if (st) atomicOr(status, st);
}


// First work item of this group, spread over the SMs first: with fewer items than groups, every
// warp has as few of them as possible.
__device__ __forceinline__ uint32_t first_group_item() {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  return (lane / kGroupLanes * (kGroupThreads / 32) + warp) * gridDim.x + blockIdx.x;
}
// The next one of a group that wants one: *fetch counts the items taken beyond the first of every
// group; with at most one item per group there is none, and the cursor is not touched.  All lanes of
// the warp call it.
__device__ __forceinline__ void next_group_item(const Group& g, uint32_t* fetch, uint32_t n, bool want, uint32_t& i) {
  const uint32_t groups = gridDim.x * kGroupsPerBlock;
  uint32_t r = n;
  if (n > groups) {
    if (want && g.sub == 0) r = groups + atomicAdd(fetch, 1u);
    r = g.shfl(r, 0);
  }
  if (want) i = r;
}

// nb_trace_rays with few rays: 8 lanes per ray (GroupTrace).
template <bool kAny>
__global__ void __launch_bounds__(kGroupThreads, 6)
    k_trace_rays_group(DevScene s, const float4* __restrict__ rays, uint32_t n, float4* __restrict__ hits,
                       uint32_t* __restrict__ inst, uint32_t* __restrict__ fetch, uint32_t* __restrict__ status) {
  __shared__ uint2 stacks[kGroupsPerBlock][kStackSize];
  const Group g;
  GroupTrace t;
  uint32_t i = first_group_item();
  bool fresh = true;
  while (__any_sync(kWarp, i < n)) {
    if (fresh && i < n) {
      const float4 o = __ldg(rays + 2 * (size_t)i), d = __ldg(rays + 2 * (size_t)i + 1);
      t.begin(s, xyz(o), xyz(d), kAny);
      fresh = false;
    }
    t.step(s, g, stacks[threadIdx.x / kGroupLanes]);
    const bool done = i < n && !t.active;
    if (__any_sync(kWarp, done)) {
      if (done && g.sub == 0) {
        hits[i] = make_float4(t.h.t, t.h.u, t.h.v, __uint_as_float(t.h.tri));
        if (inst) inst[i] = t.h.inst;
      }
      next_group_item(g, fetch, n, done, i);
      fresh = fresh || done;
    }
  }
  if (t.status && g.sub == 0) atomicOr(status, t.status);
}

// ------------------------------------------------------------------------------------------
// wavefront path tracer
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float4 sobol_read(const float4* table, uint32_t n_entries, uint32_t idx) {
  return idx < n_entries ? __ldg(table + idx) : make_float4(0.f, 0.f, 0.f, 0.f);  // robust buffer access
}

// generate_ray (pathtracing.wgsl:27-41); m is clip_to_world, column-major
__device__ __forceinline__ void generate_ray(uint32_t x, uint32_t y, uint32_t W, uint32_t H, float rx, float ry,
                                             const float* m, V3* o, V3* d) {
  float uvx = 2.0f * ((float)x + rx) / (float)W - 1.0f;
  float uvy = 2.0f * ((float)y + ry) / (float)H - 1.0f;
  V3 pos = V3{m[12], m[13], m[14]} / m[15];
  float cx = -uvx, cy = -uvy, cz = -1.0f, cw = 1.0f;
  float wd[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) wd[r] = m[r] * cx + m[4 + r] * cy + m[8 + r] * cz + m[12 + r] * cw;
  *o = pos;
  *d = pos - V3{wd[0], wd[1], wd[2]} / wd[3];
}

// index of the last segment whose begin (path or accumulate index) is <= p
template <bool kByPixel>
__device__ __forceinline__ uint32_t find_segment(const Segment* segs, uint32_t n, uint32_t p) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    const uint32_t b = kByPixel ? segs[mid].pix_begin : segs[mid].path_begin;
    if (b <= p) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void stage_segments(Segment* dst, const WaveTables& wt) {
  for (uint32_t i = threadIdx.x; i < wt.n_segs; i += blockDim.x) dst[i] = wt.segs[i];
  __syncthreads();
}

// Pixel of the i-th queue entry of one sample plane (a bijection of [0, W*H)): the image's
// 8x8 tiles in row order, Z-order inside a tile; the columns right of the last whole tile,
// then the rows below it, in row order.  Compact warps of primary rays measured 14% faster
// traversal than rows of 32 pixels.
__device__ __forceinline__ void tile_pixel(uint32_t i, uint32_t W, uint32_t H, uint32_t* x, uint32_t* y) {
  const uint32_t Wt = W & ~7u, Ht = H & ~7u;
  if (i < Wt * Ht) {
    const uint32_t tile = i >> 6, z = i & 63u, tiles_x = Wt >> 3;
    *x = ((tile % tiles_x) << 3) | (z & 1u) | ((z >> 1) & 2u) | ((z >> 2) & 4u);
    *y = ((tile / tiles_x) << 3) | ((z >> 1) & 1u) | ((z >> 2) & 2u) | ((z >> 3) & 4u);
    return;
  }
  i -= Wt * Ht;
  const uint32_t rw = W - Wt;
  if (i < rw * Ht) {
    *x = Wt + i % rw;
    *y = i / rw;
  } else {
    i -= rw * Ht;
    *x = i % W;
    *y = Ht + i / W;
  }
}

// Samples of one pixel queued together: a warp of camera rays is 32 samples of one pixel,
// nearly the same ray 32 times over, instead of one sample of an 8x4 pixel patch (the whole
// frame is one wave, so all samples are present): 12-14% faster traversal.
constexpr uint32_t kSampleGroup = 64;

// Camera ray of queue entry q (pathtracing.wgsl:245-255): origin with the path id in .w,
// direction with the scene index in .w.  Path ids stay row-major per sample (pixel = id %
// (W*H)); the queue lists them by sample group and tile order (tile_pixel), which every later
// kernel follows through the path id each ray carries.  segs: the wave's segments.
__device__ __forceinline__ void camera_ray(const Segment* segs, const WaveTables& wt, const PathBatch& pb, uint32_t q,
                                           float4& o4, float4& d4) {
  const Segment sg = segs[find_segment<false>(segs, wt.n_segs, q)];
  const JobParams& jp = wt.jobs[sg.job];
  const uint32_t local = q - sg.path_begin;
  // the segment's samples in groups of kSampleGroup: the queue runs over one group's samples
  // of a pixel, then the next pixel in tile order (a last, smaller group the same way)
  const uint32_t span = kSampleGroup * jp.npix, full = sg.n_samples / kSampleGroup;
  uint32_t plane, order;
  if (local < full * span) {
    const uint32_t grp = local / span, j = local - grp * span;
    plane = grp * kSampleGroup + j % kSampleGroup;
    order = j / kSampleGroup;
  } else {
    const uint32_t g = sg.n_samples - full * kSampleGroup, j = local - full * span;
    plane = full * kSampleGroup + j % g;
    order = j / g;
  }
  uint32_t x, y;
  tile_pixel(order, jp.width, jp.height, &x, &y);
  const uint32_t p = sg.path_begin + plane * jp.npix + y * jp.width + x;
  const uint32_t sample = sg.first_sample + plane;
  const float4 shift = hash4f(x, y);
  const float4 sb = sobol_read(pb.sobol, pb.sobol_entries, sample * kLdsStride);
  const float jx = fract(sb.x + shift.x), jy = fract(sb.y + shift.y);
  V3 o, d;
  generate_ray(x, y, jp.width, jp.height, jx, jy, jp.c2w, &o, &d);
  o4 = make_float4(o.x, o.y, o.z, __uint_as_float(p));
  d4 = make_float4(d.x, d.y, d.z, __uint_as_float(jp.scene));
}

// Start of a wave: the bounce counters and work cursors, and (kWaveZeroRadiance: waves whose
// shading adds to radiance) every path's radiance zeroed.  The camera rays themselves are made
// by the bounce-0 traversal, which writes them to the queue for shading (camera_ray).  A
// segment's queue positions and path ids cover the same range, so zeroing by queue position
// clears every path's radiance with coalesced stores.
__global__ void __launch_bounds__(256) k_raygen(PathBatch pb, const WaveTables wt) {
  const uint32_t n = wt.n_paths;
  if (blockIdx.x == 0 && threadIdx.x < kMaxBounceSlots) {
    pb.counts[threadIdx.x] = threadIdx.x == 0 ? n : 0u;
    pb.fetch[threadIdx.x] = 0u;
  }
  if (wt.flags & nb::kWaveZeroRadiance) {
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
      pb.radiance[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// Rays that the wave's per-bounce kernels trace and shade at a bounce: none if the queue is short
// enough for k_trace_paths, which has then run its paths to their ends.
__device__ __forceinline__ uint32_t queue_count(const PathBatch& pb, const WaveTables& wt, uint32_t bounce) {
  if (bounce == 0) return wt.n_paths;
  const uint32_t n = pb.counts[bounce];
  return n <= wt.group_limit ? 0u : n;
}

// An unoccluded shadow ray adds its contribution to the path.  A path has at most one shadow ray per
// bounce, so each radiance entry has one writer per launch.
__device__ __forceinline__ void add_shadow(const PathBatch& pb, const ShadowQueue& sq, uint32_t r) {
  const uint32_t id = __float_as_uint(sq.o[r].w);
  const float4 c = sq.c[r], rr = pb.radiance[id];
  pb.radiance[id] = make_float4(rr.x + c.x, rr.y + c.y, rr.z + c.z, 0.0f);
}

// kSingle: every ray of the wave uses wt.scenes[0]; else the scene index carried in q_d.w.
// Bounce 0 (camera rays): persistent warps take 32 consecutive queue entries per atomic - 32
// samples of one pixel - make each lane's camera ray (camera_ray), write it to the queue for
// shading and trace the 32 together, so the lanes walk largely the same nodes (shared cache
// lines, agreeing branches).  The world ray stays in registers, its box-test reciprocal in
// shared memory (WorldMixed).
// kCount: the instrumented variant, which also adds the TraceCount totals of the launch to
// counters[kTraceCounterSlots * bounce + ...] (run only when a caller asks for the counters).
//
// kRefill (bounces >= 1): a lane whose ray finished does not wait for the rest of its warp's
// 32 rays; once kRefillIdle lanes of the warp are idle, the warp takes that many new rays with
// one atomic and those lanes start on them (trace_refill, world rays in shared memory).
// Secondary rays of a warp come from different pixels and surfaces and their traversal lengths
// differ widely, so without refill most lanes idle while the longest ray finishes (11 of 32
// lanes active per instruction on bounce 1).  Camera rays keep whole-warp chunks: a warp's 32
// samples of one pixel finish together, and refilling them measured 9% slower traversal.
// Refill changes only which lane traces a ray, not its result.
// kShadow (lane refill only): the launch also traces the shadow rays that the bounce before queued
// (environment NEE), after the queue's rays.  They are independent of this bounce's rays, and in a
// launch of their own they added the tail of their longest ray to every bounce (~100 us of a
// 1-2 M path wave): 1013x571 at 3 spp with NEE 4.04 -> 3.66 ms.
template <bool kSingle, bool kCount, bool kRefill, bool kShadow = false>
__global__ void __launch_bounds__(kTraceThreads, kRefill ? kRefillBlocks : kChunkBlocks) k_trace_wave(PathBatch pb, const WaveTables wt,
                                                                     uint32_t bounce,
                                                       unsigned long long* __restrict__ ray_total,
                                                       unsigned long long* __restrict__ counters,
                                                       const ShadowQueue sq) {
  const uint32_t n = queue_count(pb, wt, bounce), n_shadow = kShadow ? sq.counts[bounce - 1u] : 0u;
  if (n + n_shadow == 0) return;
  __shared__ DevScene scenes[kSingle ? 1 : nb::kMaxWaveScenes];
  if (!kSingle) {
    for (uint32_t i = threadIdx.x; i < wt.n_scenes; i += blockDim.x) scenes[i] = wt.scenes[i];
    __syncthreads();
  }
  const float4* __restrict__ qo = (bounce & 1) ? pb.q_o[1] : pb.q_o[0];
  const float4* __restrict__ qd = (bounce & 1) ? pb.q_d[1] : pb.q_d[0];
  const int lane = threadIdx.x & 31;
  uint32_t st = 0;
  TraceCount cnt;
  if (!kRefill) {  // bounce 0: camera rays, made here and written to the queue for shading
    __shared__ Segment segs[nb::kMaxWaveSegments];
    __shared__ float inv_c[kTraceWarps][kInvFloats];
    stage_segments(segs, wt);
    while (true) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(pb.fetch + bounce, 32u);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      if (base >= n) break;
      const uint32_t i = base + lane;
      if (i < n) {
        float4 o, d;
        camera_ray(segs, wt, pb, i, o, d);
        pb.q_o[0][i] = o;
        pb.q_d[0][i] = d;
        const DevScene& sc0 = kSingle ? wt.scenes[0] : scenes[__float_as_uint(d.w)];
        TraceState t;
        uint2 stack[kStackSize + 2];
        trace_begin(t, stack, sc0, xyz(o), xyz(d));
        set_world_inv(inv_c[threadIdx.x >> 5], t.rinv);
        const WorldMixed wm{t, inv_c[threadIdx.x >> 5]};
        while (trace_step<false, kCount>(t, LocalStack{stack}, sc0, &cnt, wm)) {
        }
        st |= t.status;
        const uint2 uv = stack[kHitSlot], ti = stack[kHitSlot + 1];
        pb.hits[i] = make_float4(t.t_hit, __uint_as_float(uv.x), __uint_as_float(uv.y), __uint_as_float(ti.x));
        pb.hit_inst[i] = ti.y;
      }
    }
  } else {
    __shared__ float world[kTraceWarps][kWorldFloats];
    __shared__ uint2 entries[kSharedEntries][kTraceThreads];
    const DevScene* sc = kSingle ? wt.scenes : scenes;
    // (k_trace_paths takes the bounce's own cursor if the queue is short)
    st = trace_refill<false, kCount, kShadow>(
        kShadow ? sq.fetch + bounce - 1u : pb.fetch + bounce, n + n_shadow,
        [&](uint32_t r, V3& o, V3& d, uint32_t& sidx) {
          const bool shadow = kShadow && r >= n;
          const float4 o4 = shadow ? sq.o[r - n] : qo[r], d4 = shadow ? sq.d[r - n] : qd[r];
          o = xyz(o4);
          d = xyz(d4);
          sidx = kSingle ? 0u : __float_as_uint(d4.w);
        },
        [&](uint32_t sidx) -> const DevScene& { return sc[sidx]; },
        [&](uint32_t r, float t_hit, uint2 uv, uint2 ti) {
          if (kShadow && r >= n) {
            if (t_hit == kNoHit) add_shadow(pb, sq, r - n);
            return;
          }
          pb.hits[r] = make_float4(t_hit, __uint_as_float(uv.x), __uint_as_float(uv.y), __uint_as_float(ti.x));
          pb.hit_inst[r] = ti.y;
        },
        &cnt, world[threadIdx.x >> 5], &entries[0][threadIdx.x], n);
  }
  if (st) atomicOr(pb.status, st);
  if (kCount) {  // counters[kTraceCounterSlots * bounce + 0..10]: see nb_pathtracer_trace_counters
    const uint32_t c[10] = {cnt.tlas_nodes, cnt.blas_nodes, cnt.tris, cnt.insts, cnt.pushes,
                            cnt.warp_steps, cnt.lane_steps, cnt.leaf_steps, cnt.leaf_lanes, cnt.leaf_trips};
    unsigned long long* slot = counters + nb::kTraceCounterSlots * bounce;
#pragma unroll
    for (int k = 0; k < 10; ++k) {
      unsigned long long v = c[k];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
      if (lane == 0 && v) atomicAdd(slot + (k < 5 ? k : k + 1), v);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(slot + 5, (unsigned long long)n);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && n) atomicAdd(ray_total, (unsigned long long)n);
}

// Cube-map face of a direction and its coordinates s, t in [-1, 1] on that face: the standard
// cube-map table (Vulkan / D3D, which wgpu's cube textures follow) with faces 0..5 = +X, -X,
// +Y, -Y, +Z, -Z; the largest magnitude picks the face, ties going to X, then Y.
__device__ __forceinline__ uint32_t cube_face(V3 d, float* s, float* t) {
  const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  float sc, tc, ma;
  uint32_t f;
  if (ax >= ay && ax >= az) {
    f = d.x >= 0.0f ? 0u : 1u;
    ma = ax;
    sc = d.x >= 0.0f ? -d.z : d.z;
    tc = -d.y;
  } else if (ay >= az) {
    f = d.y >= 0.0f ? 2u : 3u;
    ma = ay;
    sc = d.x;
    tc = d.y >= 0.0f ? d.z : -d.z;
  } else {
    f = d.z >= 0.0f ? 4u : 5u;
    ma = az;
    sc = d.z >= 0.0f ? d.x : -d.x;
    tc = -d.y;
  }
  *s = sc / ma;
  *t = tc / ma;
  return f;
}

// Environment radiance seen along dir (pathtracing.wgsl:168).
//  equirect (the oracle's definition): u = atan2(d.x, -d.z)/(2 pi) + 0.5, v = acos(d.y)/pi of the
//    normalised direction, bilinear with wrap in u and clamp in v;
//  cube (the reference's texture_cube at mip 0 with a linear clamp-to-edge sampler,
//    texture.rs:89-144): face and (s, t) by cube_face, texel coordinates ((s + 1) / 2) N - 1/2,
//    bilinear inside the face with clamp at its edges (GPUs blend across face seams within half
//    a texel of an edge; this definition does not);
// NaN (and zero) directions see black.
__device__ V3 env_lookup(const DevEnv& env, V3 dir) {
  if (env.kind == kEnvConstant) return V3{env.r, env.g, env.b};
  if (env.kind == kEnvCube) {
    float s, t;
    const uint32_t f = cube_face(dir, &s, &t);
    const int N = (int)env.width;
    const float fx = (s + 1.0f) * 0.5f * (float)N - 0.5f, fy = (t + 1.0f) * 0.5f * (float)N - 0.5f;
    if (fx != fx || fy != fy) return V3{0.0f, 0.0f, 0.0f};
    const float x0 = floorf(fx), y0 = floorf(fy);
    const float tx = fx - x0, ty = fy - y0;
    const int xi = (int)x0, yi = (int)y0;
    const int xa = min(max(xi, 0), N - 1), xb = min(max(xi + 1, 0), N - 1);
    const int ya = (int)f * N + min(max(yi, 0), N - 1), yb = (int)f * N + min(max(yi + 1, 0), N - 1);
    const float4 t00 = __ldg(env.texels + (size_t)ya * N + xa), t10 = __ldg(env.texels + (size_t)ya * N + xb);
    const float4 t01 = __ldg(env.texels + (size_t)yb * N + xa), t11 = __ldg(env.texels + (size_t)yb * N + xb);
    return V3{(t00.x * (1.0f - tx) + t10.x * tx) * (1.0f - ty) + (t01.x * (1.0f - tx) + t11.x * tx) * ty,
              (t00.y * (1.0f - tx) + t10.y * tx) * (1.0f - ty) + (t01.y * (1.0f - tx) + t11.y * tx) * ty,
              (t00.z * (1.0f - tx) + t10.z * tx) * (1.0f - ty) + (t01.z * (1.0f - tx) + t11.z * tx) * ty};
  }
  V3 d = normalize(dir);
  float u = nb_atan2(d.x, -d.z) * 0.159154943f + 0.5f;
  float v = nb_acos(fminf(fmaxf(d.y, -1.0f), 1.0f)) * 0.318309886f;
  float fx = u * (float)env.width - 0.5f, fy = v * (float)env.height - 0.5f;
  if (fx != fx || fy != fy) return V3{0.0f, 0.0f, 0.0f};
  float x0 = floorf(fx), y0 = floorf(fy);
  float tx = fx - x0, ty = fy - y0;
  int W = (int)env.width, H = (int)env.height;
  int xi = (int)x0, yi = (int)y0;
  int xa = ((xi % W) + W) % W, xb = (((xi + 1) % W) + W) % W;
  int ya = yi < 0 ? 0 : (yi > H - 1 ? H - 1 : yi), yb = yi + 1 < 0 ? 0 : (yi + 1 > H - 1 ? H - 1 : yi + 1);
  float4 t00 = __ldg(env.texels + (size_t)ya * W + xa), t10 = __ldg(env.texels + (size_t)ya * W + xb);
  float4 t01 = __ldg(env.texels + (size_t)yb * W + xa), t11 = __ldg(env.texels + (size_t)yb * W + xb);
  return V3{(t00.x * (1.0f - tx) + t10.x * tx) * (1.0f - ty) + (t01.x * (1.0f - tx) + t11.x * tx) * ty,
            (t00.y * (1.0f - tx) + t10.y * tx) * (1.0f - ty) + (t01.y * (1.0f - tx) + t11.y * tx) * ty,
            (t00.z * (1.0f - tx) + t10.z * tx) * (1.0f - ty) + (t01.z * (1.0f - tx) + t11.z * tx) * ty};
}

// ---- environment importance sampling (NB_SAMPLE_ENV_NEE; no counterpart in the reference,
// whose README lists it as planned work) ----------------------------------------------------

// largest i in [0, n - 2] with c[i] <= u, for a CDF c[0] = 0 ... c[n - 1] = 1 and u in [0, 1)
__device__ __forceinline__ uint32_t cdf_index(const float* c, uint32_t n, float u) {
  uint32_t lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(c + mid) <= u) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Direction of an environment sample for uniform (u1, u2).  Constant environment: uniform on
// the sphere.  Equirect and cube: texel row by the marginal CDF, column by the row's CDF,
// uniform inside the texel cell, mapped like env_lookup.  Equirect: theta = pi v,
// phi = 2 pi (u - 1/2), d = (sin theta sin phi, cos theta, -sin theta cos phi).  Cube: row
// f N + r of face f, s = 2 (x + du) / N - 1, t = 2 (r + dv) / N - 1, d = the point (s, t) of
// face f (the inverse of cube_face), normalised.
__device__ V3 env_sample_dir(const DevEnv& env, float u1, float u2) {
  if (env.kind == kEnvConstant) {
    const float z = 1.0f - 2.0f * u1;
    const float r = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    float sp, cp;
    nb_sincos(kTwoPi * u2 - kPi, &sp, &cp);
    return V3{r * cp, r * sp, z};
  }
  const uint32_t W = env.width, H = env.height;
  const uint32_t y = cdf_index(env.cdf_rows, H + 1, u1);
  const float r0 = __ldg(env.cdf_rows + y), r1 = __ldg(env.cdf_rows + y + 1);
  const float dv = r1 > r0 ? fminf((u1 - r0) / (r1 - r0), 0.99999994f) : 0.5f;
  const float* row = env.cdf_cols + (size_t)y * (W + 1);
  const uint32_t x = cdf_index(row, W + 1, u2);
  const float c0 = __ldg(row + x), c1 = __ldg(row + x + 1);
  const float du = c1 > c0 ? fminf((u2 - c0) / (c1 - c0), 0.99999994f) : 0.5f;
  if (env.kind == kEnvCube) {
    const uint32_t f = y / W, r = y - f * W;
    const float s = 2.0f * (((float)x + du) / (float)W) - 1.0f, t = 2.0f * (((float)r + dv) / (float)W) - 1.0f;
    V3 d;
    switch (f) {
      case 0: d = V3{1.0f, -t, -s}; break;
      case 1: d = V3{-1.0f, -t, s}; break;
      case 2: d = V3{s, 1.0f, t}; break;
      case 3: d = V3{s, -1.0f, -t}; break;
      case 4: d = V3{s, -t, 1.0f}; break;
      default: d = V3{-s, -t, -1.0f}; break;
    }
    return normalize(d);
  }
  const float u = ((float)x + du) / (float)W, v = ((float)y + dv) / (float)H;
  float st, ct, sp, cp;
  nb_sincos(kPi * v, &st, &ct);
  nb_sincos(kTwoPi * (u - 0.5f), &sp, &cp);
  return V3{st * sp, ct, -st * cp};
}

// Solid-angle density with which env_sample_dir produces the unit direction d: 1/(4 pi) for a
// constant environment; pdf_uv of d's texel / (2 pi^2 sin theta) for an equirect map; for a
// cube map pdf_uv of d's texel x (1 + s^2 + t^2)^(3/2) / 24 (the table's v spans 6 faces,
// (s, t) spans [-1, 1]^2 per face, and d omega = ds dt / (1 + s^2 + t^2)^(3/2)).
__device__ float env_pdf(const DevEnv& env, V3 d) {
  if (env.kind == kEnvConstant) return 0.0795774715f;
  if (env.kind == kEnvCube) {
    float s, t;
    const uint32_t f = cube_face(d, &s, &t);
    if (s != s || t != t) return 0.0f;
    const int N = (int)env.width;
    const int x = min(max((int)((s + 1.0f) * 0.5f * (float)N), 0), N - 1);
    const int y = (int)f * N + min(max((int)((t + 1.0f) * 0.5f * (float)N), 0), N - 1);
    const float j = 1.0f + s * s + t * t;
    return __ldg(env.pdf_uv + (size_t)y * N + x) * (j * sqrtf(j)) * (1.0f / 24.0f);
  }
  const float u = nb_atan2(d.x, -d.z) * 0.159154943f + 0.5f;
  const float cy = fminf(fmaxf(d.y, -1.0f), 1.0f);
  const float v = nb_acos(cy) * 0.318309886f;
  if (u != u || v != v) return 0.0f;
  const int W = (int)env.width, H = (int)env.height;
  const int x = min(max((int)(u * (float)W), 0), W - 1), y = min(max((int)(v * (float)H), 0), H - 1);
  const float sin_t = sqrtf(fmaxf(0.0f, (1.0f - cy) * (1.0f + cy)));
  if (!(sin_t > 0.0f)) return 0.0f;
  return __ldg(env.pdf_uv + (size_t)y * W + x) / (19.7392088f * sin_t);  // 2 pi^2
}

// sample_vndf_iso (pathtracing.wgsl:68-98)
__device__ __forceinline__ V3 sample_vndf_iso(float r0, float r1, V3 wi, float alpha, V3 n) {
  if (alpha == 0.0f) return n;
  V3 wi_z = n * dot(wi, n);
  V3 wi_xy = wi - wi_z;
  V3 wiStd = normalize(wi_z - alpha * wi_xy);
  float wiStd_z = dot(wiStd, n);
  float phi = (2.0f * r0 - 1.0f) * kPi;
  float z = (1.0f - r1) * (1.0f + wiStd_z) - wiStd_z;
  float sinTheta = sqrtf(fminf(fmaxf(1.0f - z * z, 0.0f), 1.0f));
  float sp, cp;
  nb_sincos(phi, &sp, &cp);
  V3 cStd{sinTheta * cp, sinTheta * sp, z};
  V3 wr = n + V3{0.0f, 0.0f, 1.0f};
  float safe_wrz = fmaxf(wr.z, 1e-6f);
  V3 c = dot(wr, cStd) * wr / safe_wrz - cStd;
  V3 wmStd = c + wiStd;
  V3 wmStd_z = n * dot(n, wmStd);
  V3 wmStd_xy = wmStd_z - wmStd;
  return normalize(wmStd_z + alpha * wmStd_xy);
}

__device__ __forceinline__ V3 F_schlick(float hdotv, V3 r0) {  // pathtracing.wgsl:113-115
  float p = pow5(1.0f - hdotv);
  return r0 + (V3{1.0f, 1.0f, 1.0f} - r0) * p;
}
__device__ __forceinline__ float lambda_tr(float ndotv, float alpha2) {  // pathtracing.wgsl:119-125
  float cos2 = ndotv * ndotv;
  float sin2 = 1.0f - cos2;
  float tan2 = sin2 / cos2;
  return (-1.0f + sqrtf(1.0f + alpha2 * tan2)) / 2.0f;
}

// Appends the surviving rays of one block to the next bounce's queue grouped by direction (a
// counting sort over the block: one global atomic per block).  The block's input rays are
// neighbours in the image (tiled queue order), so each run of same-bin rays that a trace warp
// takes together starts from one small patch of the image and points nearly the same way.
// Bins: the cube face of the direction's major axis (6) x a 4 x 4 grid of the other two
// components over that face (96).  Against grouping by octant (itself 12% faster secondary
// traversal than the input order): 6.5% faster on uniform-hemisphere probe rays, +0.6% on the
// benchmark frame, whose cosine and GGX bounces the octant already groups well.
// The queue order changes no result: rays carry their path id.  Call from every thread of
// the block (block-uniform control flow); sh holds 2 kDirBins words, the first kDirBins
// zero before the first call (append_init) - each call leaves them zero again.
constexpr uint32_t kDirBins = 96;
__device__ __forceinline__ uint32_t dir_bin(float4 d) {
  const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  float a, u, v;
  uint32_t face;
  if (ax >= ay && ax >= az) {
    a = ax; face = d.x < 0.0f ? 1u : 0u; u = d.y; v = d.z;
  } else if (ay >= az) {
    a = ay; face = d.y < 0.0f ? 3u : 2u; u = d.z; v = d.x;
  } else {  // also NaN directions: face 4, cell 0
    a = az; face = d.z < 0.0f ? 5u : 4u; u = d.x; v = d.y;
  }
  const float h = 0.5f * a;
  const uint32_t qu = (uint32_t)(u > -h) + (uint32_t)(u > 0.0f) + (uint32_t)(u > h);
  const uint32_t qv = (uint32_t)(v > -h) + (uint32_t)(v > 0.0f) + (uint32_t)(v > h);
  return face * 16u + qu * 4u + qv;
}
__device__ __forceinline__ void append_init(uint32_t* sh) {
  for (uint32_t i = threadIdx.x; i < kDirBins; i += blockDim.x) sh[i] = 0u;
  __syncthreads();
}
// k_shade: blocks of 256 threads at 64 registers, 4 per SM.  Each block bins its survivors
// by direction, and the binning's two block-wide barriers stall only that block.  With one
// 1024-thread block per SM (twice the survivors per bin of 512 threads, which once paid) every
// barrier stalled the whole SM; since lanes refill during traversal, the larger bins save
// little: benchmark frame 101.1 ms with 1024 threads, 100.4 with 512, 100.1 with 256 (shading
// 9.6 -> 8.2 ms, traversal +0.3 ms); a warp-level append without binning: 100.4 (shading 7.4,
// traversal +1.4).  The NEE and cache shade kernels (78 registers) run 256 threads without the
// register cap, which would spill
constexpr int kShadeThreads = 256;
constexpr int kShadeBlocksPerSM = 4;
constexpr int kShadeExtThreads = 256;
__device__ __forceinline__ uint32_t block_append_binned(uint32_t* counter, bool active, float4 dir, uint32_t* sh) {
  uint32_t* cnt = sh;
  uint32_t* off = sh + kDirBins;
  const uint32_t key = active ? dir_bin(dir) : kDirBins;  // kDirBins: no bin
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t grp = __match_any_sync(0xFFFFFFFFu, key);
  const int leader = __ffs(grp) - 1;
  uint32_t woff = 0;
  if (active && lane == leader) woff = atomicAdd(&cnt[key], (uint32_t)__popc(grp));
  woff = __shfl_sync(0xFFFFFFFFu, woff, leader);
  const uint32_t rank = (uint32_t)__popc(grp & ((1u << lane) - 1u));
  __syncthreads();
  if (warp == 0) {  // exclusive bin offsets, one global atomic; counts cleared for the next call
    static_assert(kDirBins == 96, "three bins per lane of the scanning warp");
    const uint32_t c0 = cnt[3 * lane], c1 = cnt[3 * lane + 1], c2 = cnt[3 * lane + 2];
    const uint32_t own = c0 + c1 + c2;
    uint32_t incl = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d) incl += t;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    uint32_t base = 0;
    if (lane == 0 && total) base = atomicAdd(counter, total);
    base = __shfl_sync(0xFFFFFFFFu, base, 0) + incl - own;
    off[3 * lane] = base;
    off[3 * lane + 1] = base + c0;
    off[3 * lane + 2] = base + c0 + c1;
    cnt[3 * lane] = cnt[3 * lane + 1] = cnt[3 * lane + 2] = 0u;
  }
  __syncthreads();
  return active ? off[key] + woff + rank : 0u;
}

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool active) {
  const uint32_t mask = __ballot_sync(0xFFFFFFFFu, active);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(0xFFFFFFFFu, base, leader < 0 ? 0 : leader);
  return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}


// Material and geometry of a hit (raytracing_sw.wgsl:138-173).  pos / nrm / tng are only
// filled for non-emissive hits: an emissive hit ends the path (pathtracing.wgsl:172-174).
struct HitSurface {
  V3 color;
  float roughness, metallic;
  bool emissive;
  V3 pos, nrm, tng;
};

__device__ __forceinline__ void load_hit_surface(const DevScene& s, uint32_t inst, float4 O, float4 H, V3 rdir,
                                                 HitSurface& hs) {
  // the triangle's vertex indices are loaded before the instance record is looked at, so the
  // two loads overlap (they are valid for every hit, emissive or not)
  const uint32_t tri = __float_as_uint(H.w);
  const uint32_t i0 = __ldg(s.tri_idx + 3 * (size_t)tri), i1 = __ldg(s.tri_idx + 3 * (size_t)tri + 1),
                 i2 = __ldg(s.tri_idx + 3 * (size_t)tri + 2);
  const float4* sh = s.inst_shade + 6 * (size_t)inst;
  const float4 c0 = ld4(sh), c1 = ld4(sh + 1), c2 = ld4(sh + 2);
  const float4 l0 = ld4(sh + 3), l1 = ld4(sh + 4), l2 = ld4(sh + 5);
  hs.color = V3{c0.w, c1.w, c2.w};
  hs.roughness = l0.w;
  hs.metallic = l1.w;
  hs.emissive = l2.w > 0.0f;  // EMISSIVE (raytracing_sw.wgsl:168-170)
  if (hs.emissive) return;
  // hit attributes (raytracing_sw.wgsl:146-158)
  const float4 a0 = ld4(s.vattr + 2 * (size_t)i0), a1 = ld4(s.vattr + 2 * (size_t)i1),
               a2 = ld4(s.vattr + 2 * (size_t)i2);
  const float4 b0 = ld4(s.vattr + 2 * (size_t)i0 + 1), b1 = ld4(s.vattr + 2 * (size_t)i1 + 1),
               b2 = ld4(s.vattr + 2 * (size_t)i2 + 1);
  const float u = H.y, v = H.z;
  const float w0 = 1.0f - u - v;
  const V3 ln = xyz(a0) * w0 + xyz(a1) * u + xyz(a2) * v;
  const V3 lt = xyz(b0) * w0 + xyz(b1) * u + xyz(b2) * v;
  hs.nrm = V3{dot(xyz(c0), ln), dot(xyz(c1), ln), dot(xyz(c2), ln)};
  hs.tng = V3{dot(xyz(l0), lt), dot(xyz(l1), lt), dot(xyz(l2), lt)};
  hs.pos = xyz(O) + H.x * rdir;
}

// Rotated Sobol samples of a bounce (pathtracing.wgsl:151-159, 176-178)
__device__ __forceinline__ void bounce_samples(const PathBatch& pb, uint32_t sample, uint32_t bounce, float4 shift,
                                               float4& s0, float4& s1) {
  const uint32_t sb = sample * kLdsStride + 1u + bounce * kLdsPerBounce;
  s0 = sobol_read(pb.sobol, pb.sobol_entries, sb);
  s1 = sobol_read(pb.sobol, pb.sobol_entries, sb + 1u);
  s0 = make_float4(fract(s0.x + shift.x), fract(s0.y + shift.y), fract(s0.z + shift.z), 0.0f);
  s1 = make_float4(0.0f, fract(s1.y + shift.y), fract(s1.z + shift.z), 0.0f);
}

// Lobe choice and direction sampling at a non-emissive hit (pathtracing.wgsl:179-224).
// weight is the factor the throughput is multiplied by.  With kPdf, pdf is the solid-angle
// density of wi under the chosen lobe times its selection probability (used only by the
// radiance cache's path-spread heuristic; +inf for a perfect mirror).
struct BsdfSample {
  V3 wi, weight, wo, n;
  float cos_o, pdf;
};

template <bool kPdf>
__device__ __forceinline__ BsdfSample sample_bsdf(const HitSurface& hs, V3 rdir, float4 s0, float4 s1) {
  BsdfSample out;
  const V3 color = hs.color;
  const float roughness = hs.roughness, metallic = hs.metallic;
  const float alpha = roughness * roughness;
  const float alpha2 = alpha * alpha;
  const V3 nn = normalize(hs.nrm);
  const V3 wo = normalize(-rdir);
  const float cosThetaO = dot(wo, nn);
  V3 wi;
  const V3 F0 = V3{0.04f, 0.04f, 0.04f} * (1.0f - metallic) + color * metallic;
  const float specular_weight = luminance(F_schlick(dot(wo, nn), F0));
  const float diffuse_weight = (1.0f - metallic) * luminance(color);
  const float p_specular = specular_weight / (specular_weight + diffuse_weight);
  const float p_diffuse = 1.0f - p_specular;
  out.pdf = 0.0f;
  if (s0.x < p_specular) {
    const V3 wm = sample_vndf_iso(s0.y, s0.z, wo, alpha, nn);
    const V3 ni = -wo;
    wi = ni - (2.0f * dot(wm, ni)) * wm;  // reflect(-wo, wm)
    const float cosThetaD = dot(wo, wm);
    const float cosThetaI = dot(wi, nn);
    const V3 F = F_schlick(cosThetaD, F0);
    const float LambdaL = lambda_tr(cosThetaI, alpha2);
    const float LambdaV = lambda_tr(cosThetaO, alpha2);
    const V3 spec = F * (1.0f + LambdaV) / (1.0f + LambdaL + LambdaV);
    out.weight = spec / p_specular;
    if (kPdf) {
      // VNDF reflection density: G1(wo) D(wm) / (4 cos_o), D the Trowbridge-Reitz NDF
      const float nm = dot(nn, wm);
      const float den = nm * nm * (alpha2 - 1.0f) + 1.0f;
      const float D = alpha2 / (kPi * den * den);
      out.pdf = alpha2 > 0.0f ? p_specular * D / (4.0f * (1.0f + LambdaV) * fabsf(cosThetaO))
                              : __int_as_float(0x7f800000);
    }
  } else {
    const V3 nt = normalize(hs.tng - dot(hs.tng, nn) * nn);  // build_tbn (common.wgsl:55-59)
    const V3 bt = cross(nn, nt);
    const float phi = kTwoPi * s1.y;
    const float sinT = sqrtf(1.0f - s1.z);
    const float cosT = sqrtf(s1.z);
    float sp, cp;
    nb_sincos(phi, &sp, &cp);
    const V3 ls{cp * sinT, sp * sinT, cosT};
    wi = nt * ls.x + bt * ls.y + nn * ls.z;
    const V3 wm = normalize(wi + wo);
    const float cosThetaD = dot(wi, wm);
    const float cosThetaI = dot(wi, nn);
    const float FD90 = 0.5f + 2.0f * alpha * pow2(cosThetaD);
    const float response =
        (1.0f + (FD90 - 1.0f) * pow5(1.0f - cosThetaI)) * (1.0f + (FD90 - 1.0f) * pow5(1.0f - cosThetaO));
    const V3 diffuse = (1.0f - metallic) * color * response;
    out.weight = diffuse / p_diffuse;
    if (kPdf) out.pdf = p_diffuse * cosT * (1.0f / kPi);
  }
  out.wi = wi;
  out.wo = wo;
  out.n = nn;
  out.cos_o = cosThetaO;
  return out;
}

// Russian roulette probability (pathtracing.wgsl:225-236).  rr_start > 0 is the start-bounce
// variant (BASELINE's "RR from bounce 3"): survival 1 before that bounce, the reference's
// schedule from it on; 0 is the reference.
__device__ __forceinline__ float rr_continue(uint32_t bounce, const JobParams& jp, V3 T) {
  float p_continue = fminf(1.0f - pow8((float)bounce / (float)jp.bounces), 1.0f);
  p_continue = p_continue * fminf(luminance(T) * jp.cf, 1.0f);
  return bounce < jp.rr_start ? 1.0f : p_continue;
}

// The ray a path continues with: origin (.w path id), direction (.w scene index), throughput
// (.w, with environment NEE: density of the lobe sample that made the ray).
struct NextRay {
  float4 o, d, t;
};

// One vertex of the reference estimator (pathtracing.wgsl:161-241): radiance where the path ends
// (end(id, L), called at most once), else the next ray; returns whether the path goes on.
// inst() gives the hit's instance.
template <class InstOf, class End>
__device__ __forceinline__ bool shade_plain(const PathBatch& pb, const WaveTables& wt, const Segment* segs,
                                            uint32_t bounce, float4 O, float4 D, float4 H, float4 Tq, InstOf inst,
                                            End end, NextRay& next) {
  const uint32_t id = __float_as_uint(O.w);
  const Segment sg = segs[find_segment<false>(segs, wt.n_segs, id)];
  const JobParams& jp = wt.jobs[sg.job];
  const DevScene& s = wt.scenes[jp.scene];
  V3 T = xyz(Tq);
  const V3 rdir = xyz(D);
  if (H.x == kNoHit) {
    end(id, T * env_lookup(jp.env, rdir));
    return false;
  }
  HitSurface hs;
  load_hit_surface(s, inst(), O, H, rdir, hs);
  if (hs.emissive) {  // pathtracing.wgsl:172-174
    end(id, T * hs.color);
    return false;
  }
  const uint32_t local = id - sg.path_begin;
  const uint32_t pix = local % jp.npix;
  const uint32_t sample = sg.first_sample + local / jp.npix;
  float4 s0, s1;
  bounce_samples(pb, sample, bounce, hash4f(pix % jp.width, pix / jp.width), s0, s1);
  const BsdfSample bs = sample_bsdf<false>(hs, rdir, s0, s1);
  T = T * bs.weight;
  const float p_continue = rr_continue(bounce, jp, T);
  if (s0.z < p_continue && bounce < jp.bounces) {
    T = T / p_continue;
    next.o = make_float4(hs.pos.x, hs.pos.y, hs.pos.z, O.w);
    next.d = make_float4(bs.wi.x, bs.wi.y, bs.wi.z, D.w);
    next.t = make_float4(T.x, T.y, T.z, 0.0f);
    return true;
  }
  end(id, V3{0.0f, 0.0f, 0.0f});  // ends without radiance
  return false;
}

__global__ void __launch_bounds__(kShadeThreads, kShadeBlocksPerSM) k_shade(PathBatch pb, const WaveTables wt, uint32_t bounce) {
  __shared__ Segment segs[nb::kMaxWaveSegments];
  __shared__ uint32_t append_sh[2 * kDirBins];
  const uint32_t n = queue_count(pb, wt, bounce);
  if (n == 0) return;
  stage_segments(segs, wt);
  append_init(append_sh);
  const bool odd = (bounce & 1) != 0;
  const float4* __restrict__ in_o = odd ? pb.q_o[1] : pb.q_o[0];
  const float4* __restrict__ in_d = odd ? pb.q_d[1] : pb.q_d[0];
  const float4* __restrict__ in_t = odd ? pb.q_t[1] : pb.q_t[0];
  float4* __restrict__ out_o = odd ? pb.q_o[0] : pb.q_o[1];
  float4* __restrict__ out_d = odd ? pb.q_d[0] : pb.q_d[1];
  float4* __restrict__ out_t = odd ? pb.q_t[0] : pb.q_t[1];
  const uint32_t stride = gridDim.x * blockDim.x;
  // whole blocks iterate together: block_append_binned synchronises the block
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t i = base + threadIdx.x;
    bool cont = false;
    NextRay next;
    next.o = next.d = next.t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
      const float4 O = in_o[i], D = in_d[i], H = pb.hits[i];
      const float4 Tq = bounce == 0 ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : in_t[i];
      cont = shade_plain(
          pb, wt, segs, bounce, O, D, H, Tq, [&] { return pb.hit_inst[i]; },
          [&](uint32_t id, V3 L) { pb.radiance[id] = make_float4(L.x, L.y, L.z, 0.0f); }, next);
    }
    const uint32_t slot = block_append_binned(pb.counts + bounce + 1, cont, next.d, append_sh);
    if (cont) {
      out_o[slot] = next.o;
      out_d[slot] = next.d;
      out_t[slot] = next.t;
    }
  }
}

// 32-bit integer finaliser (Wellons' lowbias32)
__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

__device__ __forceinline__ nb::CacheFeatures cache_features(const HitSurface& hs, const BsdfSample& bs, uint32_t tag) {
  nb::CacheFeatures f;
  f.pos[0] = hs.pos.x; f.pos[1] = hs.pos.y; f.pos[2] = hs.pos.z;
  f.roughness = hs.roughness;
  f.wo[0] = bs.wo.x; f.wo[1] = bs.wo.y; f.wo[2] = bs.wo.z;
  f.metallic = hs.metallic;
  f.n[0] = bs.n.x; f.n[1] = bs.n.y; f.n[2] = bs.n.z;
  f.tag = tag;
  f.color[0] = hs.color.x; f.color[1] = hs.color.y; f.color[2] = hs.color.z;
  f.pad = 0.0f;
  return f;
}

// Shade for the radiance-cache mode.  The prefix of every path is the plain tracer's (same
// samples, lobes and Russian roulette); what changes is where it ends:
//  - path spread (Mueller et al. 2021, sec. 3.3): a0 = |x0 - x1|^2 / (4 pi cos1) at the
//    primary hit, and sqrt a(x1..xn) = sum_{i>=2} |x_{i-1} - x_i| / sqrt(p_{i-1} cos_i), with
//    p the density of the sampled direction.  At the first vertex where sqrt a > sqrt(c a0)
//    (or at the last bounce) the path becomes an image query: its sample is T * cache(x).
//  - one path per group of `stride` path ids (position in the group hashed from the group
//    and the frame) is a training path: it records each vertex (features and the factor its
//    throughput is multiplied by), continues past its query vertex for `extra` vertices and
//    ends in a tail query that closes its radiance chain with the cache (self-training),
//    unless a miss, an emitter or Russian roulette ends it first.
// What a vertex of the cache mode leaves behind besides radiance and the next ray: lookups and the
// path's cache state for the next vertex (q_x of CacheWave).
struct CacheVertex {
  nb::CacheFeatures f;
  V3 T;               // throughput of the image query
  float4 x;           // next state
  uint32_t slot;      // training slot, ~0u: none
  bool image_q, tail_q;
};

// One vertex of the cache mode.  X: the path's state (unused at bounce 0); end(id, L) takes the
// radiance of a path that ends without a lookup; lead: this thread writes the vertex' records
// (the threads of a group shade the same vertex).  Returns whether the path goes on.
template <class InstOf, class End>
__device__ __forceinline__ bool shade_cache(const PathBatch& pb, const WaveTables& wt, const Segment* segs,
                                            const nb::CacheWave& cw, uint32_t bounce, float4 O, float4 D, float4 H,
                                            float4 Tq, float4 X, InstOf inst, End end, bool lead, NextRay& next,
                                            CacheVertex& cv) {
  const uint32_t id = __float_as_uint(O.w);
  const Segment sg = segs[find_segment<false>(segs, wt.n_segs, id)];
  const JobParams& jp = wt.jobs[sg.job];
  const DevScene& s = wt.scenes[jp.scene];
  V3 T = xyz(Tq);
  const V3 rdir = xyz(D);
  float budget = 0.0f, pdf_prev = 0.0f;
  uint32_t flags = 0;
  uint32_t& slot = cv.slot;
  if (bounce == 0) {
    const uint32_t G = *cw.stride;
    const uint32_t frame_key = mix32(cw.frame ^ 0x5bd1e995u);
    const uint32_t group = id / G;
    const bool train = group < cw.max_slots && id % G == mix32(group ^ frame_key) % G;
    slot = train ? group : ~0u;
    flags = train ? nb::kPathTraining : 0u;
  } else {
    budget = X.x;
    pdf_prev = X.y;
    slot = __float_as_uint(X.z);
    flags = __float_as_uint(X.w);
  }
  const bool training = (flags & nb::kPathTraining) != 0;
  const bool image_done = (flags & nb::kPathImageDone) != 0;
  if (H.x == kNoHit) {
    const V3 E = env_lookup(jp.env, rdir);
    if (!image_done) end(id, T * E);
    if (training && lead) cw.tail[slot] = make_float4(E.x, E.y, E.z, 0.0f);
    return false;
  }
  HitSurface hs;
  load_hit_surface(s, inst(), O, H, rdir, hs);
  if (hs.emissive) {
    if (!image_done) end(id, T * hs.color);
    if (training && lead) cw.tail[slot] = make_float4(hs.color.x, hs.color.y, hs.color.z, 0.0f);
    return false;
  }
  const uint32_t local = id - sg.path_begin;
  const uint32_t pix = local % jp.npix;
  const uint32_t sample = sg.first_sample + local / jp.npix;
  float4 s0, s1;
  bounce_samples(pb, sample, bounce, hash4f(pix % jp.width, pix / jp.width), s0, s1);
  const BsdfSample bs = sample_bsdf<true>(hs, rdir, s0, s1);
  const float dist2 = H.x * H.x * dot(rdir, rdir);
  const float cos_v = fabsf(bs.cos_o);
  if (bounce == 0)
    budget = cw.spread_c < 0.0f ? -1.0f : sqrtf(cw.spread_c * dist2 / (4.0f * kPi * cos_v));
  else
    budget = budget - sqrtf(dist2 / (pdf_prev * cos_v));
  cv.f = cache_features(hs, bs, id);
  cv.T = T;
  const V3 Tn = T * bs.weight;
  const float p_continue = rr_continue(bounce, jp, Tn);
  const bool rr_ok = s0.z < p_continue && bounce < jp.bounces;
  // an infinite c turns the spread rule off; otherwise NaN budgets (degenerate
  // geometry) end the prefix as well
  const bool spread_end = !isinf(cw.spread_c) && !(budget >= 0.0f);
  cv.image_q = !image_done && (spread_end || bounce >= jp.bounces);
  bool go = false;
  if (!training) {
    go = !cv.image_q && rr_ok;
  } else {
    uint32_t since = (flags >> nb::kPathSinceShift) & 0xFFu;
    // a training path that reaches the vertex cap ends here, its pixel sample included
    if (bounce >= nb::kCacheMaxVertices) cv.image_q = !image_done;
    if (cv.image_q) {
      flags |= nb::kPathImageDone;
      since = 0;
    }
    if (((flags & nb::kPathImageDone) && since >= cw.extra) || bounce >= nb::kCacheMaxVertices) {
      cv.tail_q = true;
    } else {
      const V3 w = rr_ok ? bs.weight / p_continue : V3{0.0f, 0.0f, 0.0f};
      if (lead) {
        nb::TrainVertex tv;
        tv.f = cv.f;
        tv.w = make_float4(w.x, w.y, w.z, 0.0f);
        cw.verts[(size_t)slot * nb::kCacheMaxVertices + bounce] = tv;
        cw.vert_count[slot] = bounce + 1;
      }
      go = rr_ok;
      if (!go && lead) cw.tail[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (go && (flags & nb::kPathImageDone)) since += 1;
    }
    flags = (flags & 0xFFu) | (since << nb::kPathSinceShift);
  }
  if (go) {
    const V3 Tc = Tn / p_continue;
    next.o = make_float4(hs.pos.x, hs.pos.y, hs.pos.z, O.w);
    next.d = make_float4(bs.wi.x, bs.wi.y, bs.wi.z, D.w);
    next.t = make_float4(Tc.x, Tc.y, Tc.z, 0.0f);
    cv.x = make_float4(budget, bs.pdf, __uint_as_float(slot), __uint_as_float(flags));
  }
  return go;
}

// Writes lookup `at` of the wave (dropped beyond the capacity, which a wave's paths and training
// slots never exceed): the pixel's query, or the tail that closes a training path's chain.
__device__ __forceinline__ void put_image_query(const nb::CacheWave& cw, uint32_t at, const CacheVertex& cv) {
  if (at >= cw.max_queries) return;
  nb::CacheQuery q;
  q.f = cv.f;
  q.T = make_float4(cv.T.x, cv.T.y, cv.T.z, 0.0f);
  cw.queries[at] = q;
}
__device__ __forceinline__ void put_tail_query(const nb::CacheWave& cw, uint32_t at, const CacheVertex& cv) {
  if (at >= cw.max_queries) return;
  nb::CacheQuery q;
  q.f = cv.f;
  q.f.tag = nb::kCacheTailBit | cv.slot;
  q.T = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
  cw.queries[at] = q;
}

__global__ void __launch_bounds__(kShadeExtThreads, 3) k_shade_cache(PathBatch pb, const WaveTables wt, const nb::CacheWave cw,
                                                     uint32_t bounce) {
  __shared__ Segment segs[nb::kMaxWaveSegments];
  __shared__ uint32_t append_sh[2 * kDirBins];
  const uint32_t n = queue_count(pb, wt, bounce);
  if (n == 0) return;
  stage_segments(segs, wt);
  append_init(append_sh);
  const bool odd = (bounce & 1) != 0;
  const float4* __restrict__ in_o = odd ? pb.q_o[1] : pb.q_o[0];
  const float4* __restrict__ in_d = odd ? pb.q_d[1] : pb.q_d[0];
  const float4* __restrict__ in_t = odd ? pb.q_t[1] : pb.q_t[0];
  const float4* __restrict__ in_x = odd ? cw.q_x[1] : cw.q_x[0];
  float4* __restrict__ out_o = odd ? pb.q_o[0] : pb.q_o[1];
  float4* __restrict__ out_d = odd ? pb.q_d[0] : pb.q_d[1];
  float4* __restrict__ out_t = odd ? pb.q_t[0] : pb.q_t[1];
  float4* __restrict__ out_x = odd ? cw.q_x[0] : cw.q_x[1];
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t i = base + threadIdx.x;
    bool cont = false;
    NextRay next;
    next.o = next.d = next.t = make_float4(0.f, 0.f, 0.f, 0.f);
    CacheVertex cv;
    cv.image_q = cv.tail_q = false;
    if (i < n) {
      const float4 O = in_o[i], D = in_d[i], H = pb.hits[i];
      const float4 Tq = bounce == 0 ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : in_t[i];
      const float4 X = bounce == 0 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : in_x[i];
      cont = shade_cache(
          pb, wt, segs, cw, bounce, O, D, H, Tq, X, [&] { return pb.hit_inst[i]; },
          [&](uint32_t id, V3 L) { pb.radiance[id] = make_float4(L.x, L.y, L.z, 0.0f); }, true, next, cv);
    }
    const uint32_t at = block_append_binned(pb.counts + bounce + 1, cont, next.d, append_sh);
    if (cont) {
      out_o[at] = next.o;
      out_d[at] = next.d;
      out_t[at] = next.t;
      out_x[at] = cv.x;
    }
    const uint32_t qi = warp_append(cw.n_queries, cv.image_q);
    if (cv.image_q) put_image_query(cw, qi, cv);
    const uint32_t ti = warp_append(cw.n_queries, cv.tail_q);
    if (cv.tail_q) put_tail_query(cw, ti, cv);
  }
}

// f cos(theta_i) of each lobe of the reference BRDF for an arbitrary direction wi, and each
// lobe's sampling density for wi times its selection probability (the densities the lobe
// sampling of sample_bsdf realises).  Specular: F D G2 / (4 cos_o) with the Trowbridge-Reitz
// D and the reference's Lambda (so that f cos / pdf_vndf is the reference's F (1 + L_V) /
// (1 + L_L + L_V)); diffuse: (1 - metallic) color response cos_i / pi.  A perfect mirror
// (alpha = 0) has no specular part here: only lobe sampling can find it.
struct BsdfEval {
  V3 spec, diff;
  float q_spec, q_diff;
};

__device__ __forceinline__ BsdfEval eval_bsdf(const HitSurface& hs, const BsdfSample& bs, V3 wi) {
  BsdfEval ev;
  const V3 color = hs.color;
  const float metallic = hs.metallic;
  const float alpha = hs.roughness * hs.roughness;
  const float alpha2 = alpha * alpha;
  const V3 nn = bs.n, wo = bs.wo;
  const float cos_o = bs.cos_o, cos_i = dot(wi, nn);
  const V3 F0 = V3{0.04f, 0.04f, 0.04f} * (1.0f - metallic) + color * metallic;
  const float specular_weight = luminance(F_schlick(dot(wo, nn), F0));
  const float diffuse_weight = (1.0f - metallic) * luminance(color);
  const float p_specular = specular_weight / (specular_weight + diffuse_weight);
  const float p_diffuse = 1.0f - p_specular;
  const V3 wm = normalize(wi + wo);
  if (alpha2 > 0.0f) {
    const float nm = dot(nn, wm);
    const float den = nm * nm * (alpha2 - 1.0f) + 1.0f;
    const float D = alpha2 / (kPi * den * den);
    const float LambdaV = lambda_tr(cos_o, alpha2), LambdaL = lambda_tr(cos_i, alpha2);
    const V3 F = F_schlick(dot(wo, wm), F0);
    ev.spec = F * (D / ((1.0f + LambdaV + LambdaL) * 4.0f * cos_o));
    ev.q_spec = p_specular * D / (4.0f * (1.0f + LambdaV) * cos_o);
  } else {
    ev.spec = V3{0.0f, 0.0f, 0.0f};
    ev.q_spec = __int_as_float(0x7f800000);
  }
  const float cosThetaD = dot(wi, wm);
  const float FD90 = 0.5f + 2.0f * alpha * pow2(cosThetaD);
  const float response = (1.0f + (FD90 - 1.0f) * pow5(1.0f - cos_i)) * (1.0f + (FD90 - 1.0f) * pow5(1.0f - cos_o));
  ev.diff = (1.0f - metallic) * color * (response * cos_i * (1.0f / kPi));
  ev.q_diff = p_diffuse * cos_i * (1.0f / kPi);
  return ev;
}

__device__ __forceinline__ bool finite3(V3 v) { return isfinite(v.x) && isfinite(v.y) && isfinite(v.z); }

// Shade with environment next-event estimation (NB_SAMPLE_ENV_NEE).  The path is the
// reference's (same samples, lobe choice, VNDF / cosine sampling, Russian roulette); in
// addition every non-emissive vertex samples one environment direction (importance sampling
// of the environment's radiance, Sobol dimensions the reference leaves unused: sobol_0.w and
// sobol_1.x of the bounce) and queues a shadow ray carrying that sample's contribution.  The
// two techniques are combined per BRDF lobe with the power heuristic: an environment sample
// weighs lobe k by p_env^2 / (q_k^2 + p_env^2), a lobe-sampled ray that escapes to the
// environment by q^2 / (q^2 + p_env^2), q = the lobe's density (carried in q_t.w).  Where
// next-event estimation cannot reach a direction (below the shading normal, cos_o <= 0, a
// mirror lobe) the carried density is +inf and the lobe sample keeps full weight, so the
// estimator stays unbiased.  Radiance accumulates per path (+=) instead of being written once.
//
// One vertex: add(id, L) takes the radiance a path gains, shadow(o, d, c) the shadow ray and the
// radiance it carries.  Returns whether the path goes on.
template <class InstOf, class Add, class Shadow>
__device__ __forceinline__ bool shade_nee(const PathBatch& pb, const WaveTables& wt, const Segment* segs,
                                          uint32_t bounce, float4 O, float4 D, float4 H, float4 Tq, InstOf inst,
                                          Add add, Shadow shadow, NextRay& next) {
  const float kInf = __int_as_float(0x7f800000);
  const uint32_t id = __float_as_uint(O.w);
  const Segment sg = segs[find_segment<false>(segs, wt.n_segs, id)];
  const JobParams& jp = wt.jobs[sg.job];
  const DevScene& s = wt.scenes[jp.scene];
  V3 T = xyz(Tq);
  const V3 rdir = xyz(D);
  if (H.x == kNoHit) {
    V3 L = T * env_lookup(jp.env, rdir);
    const float q = Tq.w;  // density of the lobe sample that made this ray (bounce > 0)
    if (bounce > 0 && q < kInf) {
      const float pe = env_pdf(jp.env, normalize(rdir));
      L = L * (q * q / (q * q + pe * pe));
    }
    add(id, L);
    return false;
  }
  HitSurface hs;
  load_hit_surface(s, inst(), O, H, rdir, hs);
  if (hs.emissive) {
    add(id, T * hs.color);
    return false;
  }
  const uint32_t local = id - sg.path_begin;
  const uint32_t pix = local % jp.npix;
  const uint32_t sample = sg.first_sample + local / jp.npix;
  const float4 shift = hash4f(pix % jp.width, pix / jp.width);
  float4 s0, s1;
  bounce_samples(pb, sample, bounce, shift, s0, s1);
  const BsdfSample bs = sample_bsdf<true>(hs, rdir, s0, s1);
  // jobs without the flag take the plain estimator's exact path (one contribution
  // added onto zero, lobe samples at full weight)
  const bool nee_ok = (jp.flags & nb::kJobEnvNee) && bs.cos_o > 0.0f;
  if (nee_ok) {
    const uint32_t sb = sample * kLdsStride + 1u + bounce * kLdsPerBounce;
    const float u1 = fract(sobol_read(pb.sobol, pb.sobol_entries, sb).w + shift.w);
    const float u2 = fract(sobol_read(pb.sobol, pb.sobol_entries, sb + 1u).x + shift.x);
    const V3 we = env_sample_dir(jp.env, u1, u2);
    const float pe = env_pdf(jp.env, we);
    if (pe > 0.0f && dot(we, bs.n) > 0.0f) {
      const BsdfEval ev = eval_bsdf(hs, bs, we);
      const float pe2 = pe * pe;
      const float ws = pe2 / (ev.q_spec * ev.q_spec + pe2), wd = pe2 / (ev.q_diff * ev.q_diff + pe2);
      const V3 C = T * env_lookup(jp.env, we) * (ev.spec * ws + ev.diff * wd) / pe;
      if (finite3(C) && (C.x > 0.0f || C.y > 0.0f || C.z > 0.0f))
        shadow(make_float4(hs.pos.x, hs.pos.y, hs.pos.z, O.w), make_float4(we.x, we.y, we.z, D.w),
               make_float4(C.x, C.y, C.z, 0.0f));
    }
  }
  T = T * bs.weight;
  const float p_continue = rr_continue(bounce, jp, T);
  if (!(s0.z < p_continue && bounce < jp.bounces)) return false;
  T = T / p_continue;
  const float q = (nee_ok && dot(bs.wi, bs.n) > 0.0f) ? bs.pdf : kInf;
  next.o = make_float4(hs.pos.x, hs.pos.y, hs.pos.z, O.w);
  next.d = make_float4(bs.wi.x, bs.wi.y, bs.wi.z, D.w);
  next.t = make_float4(T.x, T.y, T.z, q);
  return true;
}

__global__ void __launch_bounds__(kShadeExtThreads) k_shade_nee(PathBatch pb, const WaveTables wt, const ShadowQueue sq,
                                                   uint32_t bounce) {
  __shared__ Segment segs[nb::kMaxWaveSegments];
  __shared__ uint32_t append_sh[2 * kDirBins];
  const uint32_t n = queue_count(pb, wt, bounce);
  if (n == 0) return;
  stage_segments(segs, wt);
  append_init(append_sh);
  const bool odd = (bounce & 1) != 0;
  const float4* __restrict__ in_o = odd ? pb.q_o[1] : pb.q_o[0];
  const float4* __restrict__ in_d = odd ? pb.q_d[1] : pb.q_d[0];
  const float4* __restrict__ in_t = odd ? pb.q_t[1] : pb.q_t[0];
  float4* __restrict__ out_o = odd ? pb.q_o[0] : pb.q_o[1];
  float4* __restrict__ out_d = odd ? pb.q_d[0] : pb.q_d[1];
  float4* __restrict__ out_t = odd ? pb.q_t[0] : pb.q_t[1];
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t i = base + threadIdx.x;
    bool cont = false, shadow = false;
    NextRay next;
    next.o = next.d = next.t = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 sh_o = next.o, sh_d = next.o, sh_c = next.o;
    if (i < n) {
      const float4 O = in_o[i], D = in_d[i], H = pb.hits[i];
      const float4 Tq = bounce == 0 ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : in_t[i];
      cont = shade_nee(
          pb, wt, segs, bounce, O, D, H, Tq, [&] { return pb.hit_inst[i]; },
          [&](uint32_t id, V3 L) {
            const float4 c = pb.radiance[id];
            pb.radiance[id] = make_float4(c.x + L.x, c.y + L.y, c.z + L.z, 0.0f);
          },
          [&](float4 o, float4 d, float4 c) {
            shadow = true;
            sh_o = o;
            sh_d = d;
            sh_c = c;
          },
          next);
    }
    const uint32_t slot = block_append_binned(pb.counts + bounce + 1, cont, next.d, append_sh);
    if (cont) {
      out_o[slot] = next.o;
      out_d[slot] = next.d;
      out_t[slot] = next.t;
    }
    const uint32_t ss = warp_append(sq.counts + bounce, shadow);
    if (shadow) {
      sq.o[ss] = sh_o;
      sq.d[ss] = sh_d;
      sq.c[ss] = sh_c;
    }
  }
}

// Shadow rays of the last bounce (and, beside the instrumented traversal, of every bounce): an any-hit
// query each (raytracing_sw.wgsl's triangle test and BIAS, so the ray leaves its own surface like the
// reference's extension rays), with lane refill (trace_refill).  .w of a shadow ray's direction is the
// index of its scene in the wave.
__global__ void __launch_bounds__(kTraceThreads, kRefillBlocks) k_trace_shadow(PathBatch pb, const WaveTables wt, const ShadowQueue sq,
                                                      uint32_t bounce) {
  const uint32_t n = sq.counts[bounce];
  if (n == 0) return;
  __shared__ DevScene scenes[nb::kMaxWaveScenes];
  for (uint32_t i = threadIdx.x; i < wt.n_scenes; i += blockDim.x) scenes[i] = wt.scenes[i];
  __syncthreads();
  __shared__ float world[kTraceWarps][kWorldFloats];
  __shared__ uint2 entries[kSharedEntries][kTraceThreads];
  const uint32_t st = trace_refill<true, false>(
      sq.fetch + bounce, n,
      [&](uint32_t r, V3& o, V3& d, uint32_t& sidx) {
        const float4 d4 = sq.d[r];
        o = xyz(sq.o[r]);
        d = xyz(d4);
        sidx = __float_as_uint(d4.w);
      },
      [&](uint32_t sidx) -> const DevScene& { return scenes[sidx]; },
      [&](uint32_t r, float t_hit, uint2, uint2) {
        if (t_hit == kNoHit) add_shadow(pb, sq, r);
      },
      nullptr, world[threadIdx.x >> 5], &entries[0][threadIdx.x]);
  if (st) atomicOr(pb.status, st);
}

__device__ __forceinline__ void accumulate_sample(float4& c, V3 L, uint32_t sample) {
  const float w = 1.0f / (float)sample;
  c.x = c.x * (1.0f - w) + L.x * w;
  c.y = c.y * (1.0f - w) + L.y * w;
  c.z = c.z * (1.0f - w) + L.z * w;
}
// A path's final radiance: kept for k_accumulate, or (kWaveDirect) added to its pixel.
__device__ __forceinline__ void put_radiance(const PathBatch& pb, const WaveTables& wt, const Segment* segs,
                                             uint32_t id, V3 L, bool lead) {
  if (!lead) return;
  if (!(wt.flags & nb::kWaveDirect)) {
    pb.radiance[id] = make_float4(L.x, L.y, L.z, 0.0f);
    return;
  }
  const Segment sg = segs[find_segment<false>(segs, wt.n_segs, id)];
  float4* out = wt.jobs[sg.job].out + (id - sg.path_begin);
  float4 c = *out;
  accumulate_sample(c, L, sg.first_sample);
  *out = make_float4(c.x, c.y, c.z, 1.0f);
}

// Paths run to their ends, 8 lanes per path (GroupTrace): the camera paths of a small wave
// (bounce0 = 0), or the queue of a bounce that no longer fills the GPU (queue_count).  Traversal and
// shading of a path follow one another here without a launch between them, so the time is that of
// the longest path and not the sum over the bounces of each bounce's longest ray.  All lanes of a
// group shade the same vertex; lane 0 writes.  Samples, arithmetic and the order of a path's
// radiance additions are those of the per-bounce kernels.  Bound by the latency of a path's steps
// (0.8 us each): the schedulers issue in 37% of the cycles in which they have warps at 3,072 paths, in 42% at
// 19,200.
// With kWaveDirect (one sample per pixel, reference or NEE estimator) a path adds its radiance to its
// pixel itself (accumulate_sample) and the wave needs no other launch.
enum EstimatorKind : int { kEstPlain, kEstNee, kEstCache };
template <int kEst>
__global__ void __launch_bounds__(kGroupThreads, 4)
    k_trace_paths(PathBatch pb, const WaveTables wt, const nb::CacheWave cw, uint32_t bounce0,
                  unsigned long long* __restrict__ ray_total) {
  const uint32_t n = bounce0 == 0 ? wt.n_paths : pb.counts[bounce0];
  if (n == 0 || (bounce0 != 0 && n > wt.group_limit)) return;
  __shared__ Segment segs[nb::kMaxWaveSegments];
  __shared__ uint2 stacks[kGroupsPerBlock][kStackSize];
  stage_segments(segs, wt);
  const Group g;
  uint2* stack = stacks[threadIdx.x / kGroupLanes];
  const bool lead = g.sub == 0;
  const bool odd = (bounce0 & 1) != 0;
  uint32_t rays = 0, b = bounce0, scene = 0;
  GroupTrace t;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  NextRay ray;              // the ray traced (kEstNee, during a shadow ray: the one traced after it)
  float4 X = zero;          // kEstCache: the path's state
  float4 acc = zero;        // kEstNee: the path's radiance so far
  V3 shadow_c{0.0f, 0.0f, 0.0f};
  bool more = false;        // kEstNee, during a shadow ray: the path goes on after it
  bool fresh = true;
  uint32_t i = first_group_item();
  while (__any_sync(kWarp, i < n)) {
    if (fresh && i < n) {
      if (bounce0 == 0) {
        camera_ray(segs, wt, pb, i, ray.o, ray.d);
        ray.t = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        acc = zero;
        if (kEst == kEstCache && lead) pb.radiance[__float_as_uint(ray.o.w)] = zero;  // lookups add to it
      } else {
        ray.o = (odd ? pb.q_o[1] : pb.q_o[0])[i];
        ray.d = (odd ? pb.q_d[1] : pb.q_d[0])[i];
        ray.t = (odd ? pb.q_t[1] : pb.q_t[0])[i];
        if (kEst == kEstCache) X = (odd ? cw.q_x[1] : cw.q_x[0])[i];
        if (kEst == kEstNee) acc = pb.radiance[__float_as_uint(ray.o.w)];
      }
      scene = __float_as_uint(ray.d.w);
      b = bounce0;
      ++rays;
      t.begin(wt.scenes[scene], xyz(ray.o), xyz(ray.d), false);
      fresh = false;
    }
    t.step(wt.scenes[scene], g, stack);
    const bool done = i < n && !t.active;
    if (!__any_sync(kWarp, done)) continue;
    bool ended = false;
    if (done) {
      bool cont;
      if (kEst == kEstNee && t.any) {  // a shadow ray
        if (t.h.t == kNoHit) acc = make_float4(acc.x + shadow_c.x, acc.y + shadow_c.y, acc.z + shadow_c.z, 0.0f);
        cont = more;
      } else {
        const float4 H = make_float4(t.h.t, t.h.u, t.h.v, __uint_as_float(t.h.tri));
        const float4 O = ray.o, D = ray.d, T = ray.t;
        const auto inst = [&] { return t.h.inst; };
        const auto end = [&](uint32_t id, V3 L) { put_radiance(pb, wt, segs, id, L, lead); };
        if (kEst == kEstPlain) {
          cont = shade_plain(pb, wt, segs, b, O, D, H, T, inst, end, ray);
        } else if (kEst == kEstNee) {
          bool shadow = false;
          V3 so{0.0f, 0.0f, 0.0f}, sd = so;
          cont = shade_nee(
              pb, wt, segs, b, O, D, H, T, inst,
              [&](uint32_t, V3 L) { acc = make_float4(acc.x + L.x, acc.y + L.y, acc.z + L.z, 0.0f); },
              [&](float4 o, float4 d, float4 c) {
                shadow = true;
                so = xyz(o);
                sd = xyz(d);
                shadow_c = xyz(c);
              },
              ray);
          if (shadow) {
            more = cont;
            t.begin(wt.scenes[scene], so, sd, true);
            // a ray that traces nothing (no TLAS, non-finite) is finished at once, unoccluded
            if (t.active) {
              b += 1;
              goto traced;
            }
            acc = make_float4(acc.x + shadow_c.x, acc.y + shadow_c.y, acc.z + shadow_c.z, 0.0f);
          }
        } else {
          CacheVertex cv;
          cv.image_q = cv.tail_q = false;
          cont = shade_cache(pb, wt, segs, cw, b, O, D, H, T, X, inst, end, lead, ray, cv);
          X = cv.x;
          if (lead && cv.image_q) put_image_query(cw, atomicAdd(cw.n_queries, 1u), cv);
          if (lead && cv.tail_q) put_tail_query(cw, atomicAdd(cw.n_queries, 1u), cv);
        }
        b += 1;
      }
      if (cont) {
        ++rays;
        t.begin(wt.scenes[scene], xyz(ray.o), xyz(ray.d), false);
      } else {
        if (kEst == kEstNee) put_radiance(pb, wt, segs, __float_as_uint(ray.o.w), xyz(acc), lead);
        ended = true;
      }
    traced:;
    }
    next_group_item(g, pb.fetch + bounce0, n, ended, i);
    fresh = ended;
  }
  if (lead) {
    if (t.status) atomicOr(pb.status, t.status);
    if (rays) atomicAdd(ray_total, (unsigned long long)rays);
  }
}

__global__ void k_env_sample(const DevEnv env, const float* __restrict__ u, uint32_t n, float4* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const V3 d = env_sample_dir(env, u[2 * i], u[2 * i + 1]);
    out[i] = make_float4(d.x, d.y, d.z, env_pdf(env, d));
  }
}

// running mean in sample order: out = mix(out, L_k, 1/k) (pathtracing.wgsl:246-260).  Each job
// has at most one segment per wave, so every pixel has one writer.
__global__ void __launch_bounds__(256) k_accumulate(PathBatch pb, const WaveTables wt) {
  __shared__ Segment segs[nb::kMaxWaveSegments];
  stage_segments(segs, wt);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < wt.n_pix; t += gridDim.x * blockDim.x) {
    const Segment sg = segs[find_segment<true>(segs, wt.n_segs, t)];
    const JobParams& jp = wt.jobs[sg.job];
    const uint32_t pix = t - sg.pix_begin;
    float4 c = jp.out[pix];
    for (uint32_t k = 0; k < sg.n_samples; ++k)
      accumulate_sample(c, xyz(pb.radiance[(size_t)sg.path_begin + (size_t)k * jp.npix + pix]), sg.first_sample + k);
    jp.out[pix] = make_float4(c.x, c.y, c.z, 1.0f);
  }
}

}  // namespace nbd

// ------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------
namespace nb {

static int blocks_for(const void* kernel, int threads, int sms) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return per_sm * sms;
}

cudaError_t launch_trace_rays(const nbd::DevScene& s, const float* rays, uint32_t n, bool any, bool refill,
                              float* hits, uint32_t* inst, uint32_t* fetch, uint32_t* status, int sms,
                              cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (n <= (refill ? kGroupScattered : kGroupRays)) {
    const void* kernel = any ? (const void*)nbd::k_trace_rays_group<true> : (const void*)nbd::k_trace_rays_group<false>;
    static const int full[2] = {blocks_for((const void*)nbd::k_trace_rays_group<false>, nbd::kGroupThreads, sms),
                                blocks_for((const void*)nbd::k_trace_rays_group<true>, nbd::kGroupThreads, sms)};
    const unsigned blocks = (unsigned)std::min(full[any], (int)n);
    if (n > blocks * nbd::kGroupsPerBlock) {
      const cudaError_t e = cudaMemsetAsync(fetch, 0, sizeof(uint32_t), st);
      if (e != cudaSuccess) return e;
    }
    const float4* r4 = (const float4*)rays;
    float4* h4 = (float4*)hits;
    void* args[] = {(void*)&s, (void*)&r4, (void*)&n, (void*)&h4, (void*)&inst, (void*)&fetch, (void*)&status};
    return cudaLaunchKernel(kernel, dim3(blocks), dim3(nbd::kGroupThreads), args, 0, st);
  }
  const cudaError_t e = cudaMemsetAsync(fetch, 0, sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
#define NB_TRACE_RAYS(A, R)                                                                            \
  {                                                                                                    \
    static const int g = blocks_for((const void*)nbd::k_trace_rays<A, R>, nbd::kTraceThreads, sms);                  \
    nbd::k_trace_rays<A, R><<<g, nbd::kTraceThreads, 0, st>>>(s, (const float4*)rays, n, (float4*)hits, inst, fetch, status); \
  }
  if (any) {
    if (refill) NB_TRACE_RAYS(true, true) else NB_TRACE_RAYS(true, false)
  } else {
    if (refill) NB_TRACE_RAYS(false, true) else NB_TRACE_RAYS(false, false)
  }
#undef NB_TRACE_RAYS
  return cudaGetLastError();
}

cudaError_t launch_raygen(const PathBatch& pb, const WaveTables& wt, int sms, cudaStream_t st) {
  int g = (wt.flags & kWaveZeroRadiance) ? (int)std::min<uint64_t>((wt.n_paths + 255) / 256, (uint64_t)sms * 16) : 1;
  nbd::k_raygen<<<g < 1 ? 1 : g, 256, 0, st>>>(pb, wt);
  return cudaGetLastError();
}

cudaError_t launch_trace_wave(const PathBatch& pb, const WaveTables& wt, bool single_scene, uint32_t bounce,
                              const ShadowQueue* shadow, unsigned long long* ray_total, int sms, cudaStream_t st,
                              unsigned long long* counters) {
  const bool refill = bounce >= 1;
  const ShadowQueue sq = shadow ? *shadow : ShadowQueue{};
#define NB_TRACE_WAVE(S, C, ...)                                                                              \
  {                                                                                                           \
    static const int g = blocks_for((const void*)nbd::k_trace_wave<S, C, __VA_ARGS__>, nbd::kTraceThreads, sms); \
    nbd::k_trace_wave<S, C, __VA_ARGS__><<<g, nbd::kTraceThreads, 0, st>>>(pb, wt, bounce, ray_total, counters, sq); \
  }
  if (counters) {
    if (single_scene) {
      if (refill) NB_TRACE_WAVE(true, true, true) else NB_TRACE_WAVE(true, true, false)
    } else {
      if (refill) NB_TRACE_WAVE(false, true, true) else NB_TRACE_WAVE(false, true, false)
    }
  } else if (shadow && refill) {
    if (single_scene) NB_TRACE_WAVE(true, false, true, true) else NB_TRACE_WAVE(false, false, true, true)
  } else if (single_scene) {
    if (refill) NB_TRACE_WAVE(true, false, true) else NB_TRACE_WAVE(true, false, false)
  } else {
    if (refill) NB_TRACE_WAVE(false, false, true) else NB_TRACE_WAVE(false, false, false)
  }
#undef NB_TRACE_WAVE
  return cudaGetLastError();
}

cudaError_t launch_shade(const PathBatch& pb, const WaveTables& wt, uint32_t bounce, int sms, cudaStream_t st) {
  static const int g = blocks_for((const void*)nbd::k_shade, nbd::kShadeThreads, sms);
  nbd::k_shade<<<g, nbd::kShadeThreads, 0, st>>>(pb, wt, bounce);
  return cudaGetLastError();
}

cudaError_t launch_shade_cache(const PathBatch& pb, const WaveTables& wt, const CacheWave& cw, uint32_t bounce,
                               int sms, cudaStream_t st) {
  static const int g = blocks_for((const void*)nbd::k_shade_cache, nbd::kShadeExtThreads, sms);
  nbd::k_shade_cache<<<g, nbd::kShadeExtThreads, 0, st>>>(pb, wt, cw, bounce);
  return cudaGetLastError();
}

cudaError_t launch_shade_nee(const PathBatch& pb, const WaveTables& wt, const ShadowQueue& sq, uint32_t bounce,
                             int sms, cudaStream_t st) {
  static const int g = blocks_for((const void*)nbd::k_shade_nee, nbd::kShadeExtThreads, sms);
  nbd::k_shade_nee<<<g, nbd::kShadeExtThreads, 0, st>>>(pb, wt, sq, bounce);
  return cudaGetLastError();
}

cudaError_t launch_trace_shadow(const PathBatch& pb, const WaveTables& wt, const ShadowQueue& sq, uint32_t bounce,
                                int sms, cudaStream_t st) {
  static const int g = blocks_for((const void*)nbd::k_trace_shadow, nbd::kTraceThreads, sms);
  nbd::k_trace_shadow<<<g, nbd::kTraceThreads, 0, st>>>(pb, wt, sq, bounce);
  return cudaGetLastError();
}

cudaError_t launch_trace_paths(const PathBatch& pb, const WaveTables& wt, Estimator est, const CacheWave& cw,
                               uint32_t bounce, unsigned long long* ray_total, int sms, cudaStream_t st) {
#define NB_TRACE_PATHS(E)                                                                                   \
  {                                                                                                         \
    static const int g = blocks_for((const void*)nbd::k_trace_paths<E>, nbd::kGroupThreads, sms);           \
    const unsigned blocks = (unsigned)std::min<uint64_t>((uint64_t)g, wt.n_paths);                          \
    if (bounce == 0 && wt.n_paths > blocks * nbd::kGroupsPerBlock) { /* a whole wave: no k_raygen before */ \
      const cudaError_t e = cudaMemsetAsync(pb.fetch, 0, sizeof(uint32_t), st);                             \
      if (e != cudaSuccess) return e;                                                                       \
    }                                                                                                       \
    nbd::k_trace_paths<E><<<blocks, nbd::kGroupThreads, 0, st>>>(pb, wt, cw, bounce, ray_total);            \
  }
  if (est == Estimator::kPlain) NB_TRACE_PATHS(nbd::kEstPlain)
  else if (est == Estimator::kNee) NB_TRACE_PATHS(nbd::kEstNee)
  else NB_TRACE_PATHS(nbd::kEstCache)
#undef NB_TRACE_PATHS
  return cudaGetLastError();
}

cudaError_t launch_env_sample(const nbd::DevEnv& env, const float* u, uint32_t n, float4* out, int sms,
                              cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int g = (int)std::min<uint64_t>((n + 255) / 256, (uint64_t)sms * 8);
  nbd::k_env_sample<<<g, 256, 0, st>>>(env, u, n, out);
  return cudaGetLastError();
}

cudaError_t launch_accumulate(const PathBatch& pb, const WaveTables& wt, int sms, cudaStream_t st) {
  if (wt.flags & kWaveDirect) return cudaSuccess;
  int g = (int)std::min<uint64_t>((wt.n_pix + 255) / 256, (uint64_t)sms * 16);
  nbd::k_accumulate<<<g < 1 ? 1 : g, 256, 0, st>>>(pb, wt);
  return cudaGetLastError();
}

}  // namespace nb
