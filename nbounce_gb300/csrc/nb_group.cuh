// Traversal of one ray by a group of 8 lanes, for queries with too few rays to fill the GPU.
//
// With a ray per lane (trace_step) a node step is 500-650 dependent warp instructions whatever the
// number of rays, and the lanes of a warp take turns wherever their rays disagree: a launch of a few
// thousand rays lasts as long as its longest ray (150-190 us per bounce of a 300K-triangle scene,
// ~2 us per step).  Here lane k of the group tests child k of the node, the hit children are ranked
// by comparing their keys, the leaf slots' triangles are tested by the lanes that hold them, and the
// stack is popped 8 entries at a time from shared memory: 0.8 us per step, of which about half is the
// latency of the node, triangle and instance loads.  A ray costs ~2.5 times the instructions, so the
// callers use this only below the ray counts at which a ray per lane fills the GPU (kGroupPaths).
//
// The triangles' arithmetic, the sort keys, the order in which nodes are visited and the order in which
// equal distances win are those of trace_step, so a ray's hit is the same bits.  (Only the rounding of
// closest hits' far planes differs, Planes: another box may be opened in vain.)
#pragma once

namespace nbd {

constexpr uint32_t kGroupLanes = 8;
constexpr uint32_t kGroupsPerWarp = 32 / kGroupLanes;
constexpr int kGroupThreads = 128;
constexpr uint32_t kGroupsPerBlock = kGroupThreads / kGroupLanes;

// A warp traces one ray per group in lockstep: every function below is called by all 32 lanes
// together, and what a group does not take part in is predicated off.  (Groups that branch on their
// own run one after the other: 12 of 32 lanes active, 3 times the instructions.)
constexpr uint32_t kWarp = 0xFFFFFFFFu;

// This lane's group: its first lane in the warp and the lane's place in it.
struct Group {
  uint32_t shift, sub;
  __device__ __forceinline__ Group() {
    const uint32_t lane = threadIdx.x & 31u;
    shift = lane & ~(kGroupLanes - 1u);
    sub = lane & (kGroupLanes - 1u);
  }
  __device__ __forceinline__ uint32_t ballot(bool p) const { return (__ballot_sync(kWarp, p) >> shift) & 0xFFu; }
  template <class T>
  __device__ __forceinline__ T shfl(T v, uint32_t from) const {
    return __shfl_sync(kWarp, v, (int)from, (int)kGroupLanes);
  }
};

__device__ __forceinline__ float plane_float(uint32_t q) { return __uint_as_float(0x47000000u | (q << 8)); }

// Traversal state of a group's ray, the same in its 8 lanes.
struct GroupTrace {
  V3 wo, wd, winv;      // world ray
  V3 ro, rd, rinv;      // current ray (world, or local to an instance)
  Hit h;
  int sp, blas_base;
  uint32_t cur_inst, node, status, iter;
  bool in_blas, have_node, any;
  bool active;          // the ray is not finished

  // A group without a ray.
  __device__ __forceinline__ GroupTrace() {
    wo = wd = winv = ro = rd = rinv = V3{0.0f, 0.0f, 0.0f};
    h = Hit{kNoHit, 0.0f, 0.0f, 0xFFFFFFFFu, 0xFFFFFFFFu};
    sp = blas_base = 0;
    cur_inst = node = status = iter = 0;
    in_blas = have_node = any = active = false;
  }

  // any_hit: stop at the first accepted triangle
  __device__ __forceinline__ void begin(const DevScene& s, V3 o, V3 d, bool any_hit) {
    wo = ro = o;
    wd = rd = d;
    winv = rinv = V3{safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z)};
    h = Hit{kNoHit, 0.0f, 0.0f, 0xFFFFFFFFu, 0xFFFFFFFFu};
    sp = blas_base = 0;
    cur_inst = node = iter = 0;
    in_blas = false;
    any = any_hit;
    const float fin = fabsf(o.x) + fabsf(o.y) + fabsf(o.z) + fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    active = have_node = s.has_tlas != 0u && fin <= 3.4028235e38f;  // trace_begin's rule
  }

  // One step of every active group: pop if no node is pending, test a node, its leaf triangles.
  // stack: kStackSize entries of shared memory of this group.
  __device__ __forceinline__ void step(const DevScene& s, const Group& g, uint2* stack) {
    if (active && iter++ > kIterationCap) {
      status |= kStatusIterationCap;
      active = false;
    }
    bool need = active && !have_node;
    if (__any_sync(kWarp, need)) {
      __syncwarp();  // the pushes of earlier steps
      // 8 entries at a time: those above the first one still nearer than the hit are dropped
      bool got = false;
      do {
        if (need && in_blas && sp == blas_base) {  // BLAS finished: back to the world ray
          in_blas = false;
          ro = wo;
          rd = wd;
          rinv = winv;
        }
        if (need && sp == 0) active = need = false;
        const int avail = need ? sp - (in_blas ? blas_base : 0) : 0;
        const bool have = (int)g.sub < avail;
        const uint2 en = have ? stack[sp - 1 - (int)g.sub] : make_uint2(0u, 0u);
        const uint32_t live = g.ballot(have && __uint_as_float(en.y) < h.t);
        const uint32_t f = live ? (uint32_t)__ffs(live) - 1u : 0u;
        const uint32_t e = g.shfl(en.x, f);
        if (live) {
          sp -= (int)f + 1;
          node = e;
          got = true;
          need = false;
        } else {
          sp -= min(avail, (int)kGroupLanes);
        }
      } while (__any_sync(kWarp, need));
      const bool enter = got && (node & kInstanceBit) != 0u;
      if (__any_sync(kWarp, enter)) {
        if (enter) {  // transform the world ray (raytracing_sw.wgsl:202-206)
          const float4* it = s.inst_trace + 4 * (size_t)(node & ~kInstanceBit);
          const F8 i0 = ld8(it), i1 = ld8(it + 2);
          const float4 r0 = i0.a, r1 = i0.b, r2 = i1.a, r3 = i1.b;
          ro = V3{r0.x * wo.x + r0.y * wo.y + r0.z * wo.z + r0.w * 1.0f,
                  r1.x * wo.x + r1.y * wo.y + r1.z * wo.z + r1.w * 1.0f,
                  r2.x * wo.x + r2.y * wo.y + r2.z * wo.z + r2.w * 1.0f};
          rd = V3{r0.x * wd.x + r0.y * wd.y + r0.z * wd.z, r1.x * wd.x + r1.y * wd.y + r1.z * wd.z,
                  r2.x * wd.x + r2.y * wd.y + r2.z * wd.z};
          rinv = V3{safe_rcp(rd.x), safe_rcp(rd.y), safe_rcp(rd.z)};
          cur_inst = f2u(r3.y);
          in_blas = true;
          blas_base = sp;
          node = f2u(r3.x);
        }
      }
      __syncwarp();  // the entries are read before the pushes below
    }

    // ---- this lane's child: the slab test of trace_step, near and far planes with offset 2^15 ----
    // plane bytes (WideNode): lo x, y, z at 32, 40, 48 and hi x, y, z at 56, 64, 72, one per child;
    // the near plane is the low one where the direction is positive
    NodeHead nh{};
    uint32_t nx = 0, ny = 0, nz = 0, fx = 0, fy = 0, fz = 0;
    if (active) {
      const unsigned char* p = (const unsigned char*)((in_blas ? s.blas_wide : s.tlas_wide) + 6 * (size_t)node);
      const uint32_t x = rinv.x >= 0.0f ? 0u : 24u, y = rinv.y >= 0.0f ? 0u : 24u, z = rinv.z >= 0.0f ? 0u : 24u;
      nh = load_head((const float4*)p);
      p += g.sub;
      nx = __ldg(p + 32 + x);
      ny = __ldg(p + 40 + y);
      nz = __ldg(p + 48 + z);
      fx = __ldg(p + 56 - x);
      fy = __ldg(p + 64 - y);
      fz = __ldg(p + 72 - z);
    }
    const float ax = nh.step_x * rinv.x, ay = nh.step_y * rinv.y, az = nh.step_z() * rinv.z;
    const float bx = (nh.p.x - ro.x) * rinv.x, by = (nh.p.y - ro.y) * rinv.y, bz = (nh.p.z - ro.z) * rinv.z;
    const float dx = fmaf(fabsf(ax), 0.0078125f, fabsf(bx) * 1.9073486328125e-6f);
    const float dy = fmaf(fabsf(ay), 0.0078125f, fabsf(by) * 1.9073486328125e-6f);
    const float dz = fmaf(fabsf(az), 0.0078125f, fabsf(bz) * 1.9073486328125e-6f);
    const float cx = fmaf(-32768.0f, ax, bx), cy = fmaf(-32768.0f, ay, by), cz = fmaf(-32768.0f, az, bz);
    const float tn = fmaxf(fmaxf(fmaf(plane_float(nx), ax, cx - dx), fmaf(plane_float(ny), ay, cy - dy)),
                           fmaf(plane_float(nz), az, cz - dz));
    const float tf = fminf(fminf(fmaf(plane_float(fx), ax, cx + dx), fmaf(plane_float(fy), ay, cy + dy)),
                           fmaf(plane_float(fz), az, cz + dz));
    const float lo = fmaxf(tn, 0.0f);
    const float t_below = __uint_as_float(f2u(h.t) - 1u);
    const bool hit = (nh.bits >> g.sub & 1u) != 0u && lo <= fminf(tf, t_below);
    const bool inner = (nh.bits >> g.sub & 0x100u) != 0u;
    const bool leaf = hit && in_blas && !inner, push = hit && !leaf;
    const uint32_t key = push ? (f2u(lo) & ~7u) | g.sub : 0xFFFFFFFFu;
    const uint32_t slot = nh.leaf_base + g.sub;  // of a leaf child
    const uint32_t ref = inner ? nh.child_base + g.sub : kInstanceBit | slot;

    // ---- rank the hit children; the nearest inner child is visited next, the others pushed ----
    const uint32_t pm = g.ballot(push);
    uint32_t rank = 0, first = pm ? (uint32_t)__ffs(pm) - 1u : 0u;
    if (__any_sync(kWarp, (pm & (pm - 1u)) != 0u)) {
#pragma unroll
      for (int k = 1; k < (int)kGroupLanes; ++k) rank += __shfl_xor_sync(kWarp, key, k) < key ? 1u : 0u;
      const uint32_t nearest = g.ballot(push && rank == 0u);
      if (pm) first = (uint32_t)__ffs(nearest) - 1u;
    }
    const uint32_t first_ref = g.shfl(ref, first);
    const float next_d = __uint_as_float(g.shfl(key, first) & ~7u);
    const int n = __popc(pm);
    have_node = n != 0 && (first_ref & kInstanceBit) == 0u;
    const int at = sp + n - 1 - (int)rank;
    if (push && !(have_node && rank == 0u) && at < kStackSize) stack[at] = make_uint2(ref, key & ~7u);
    sp += n - (have_node ? 1 : 0);
    if (sp > kStackSize) {
      sp = kStackSize;
      status |= kStatusStackOverflow;
    }
    if (have_node) node = first_ref;

    // ---- leaf triangles, one slot per lane ----
    if (__any_sync(kWarp, leaf)) {
      float bt = h.t, bu = 0.0f, bv = 0.0f;
      uint32_t btri = 0;
      bool better = false;
      if (leaf) {
        triangle_pair_test(ro, rd, s.tris + 6 * (size_t)slot, bt, [&](float t, float u, float v, uint32_t tri) {
          if (any && better) return;  // any hit: the first
          bt = t;
          bu = u;
          bv = v;
          btri = tri;
          better = true;
        });
      }
      const uint32_t bm = g.ballot(better);
      if (__any_sync(kWarp, bm != 0u)) {
        // any hit: the first slot's; closest: the smallest distance, of equal ones the first slot's
        float m = bt;
        m = fminf(m, __shfl_xor_sync(kWarp, m, 4));
        m = fminf(m, __shfl_xor_sync(kWarp, m, 2));
        m = fminf(m, __shfl_xor_sync(kWarp, m, 1));
        const uint32_t closest = g.ballot(better && bt == m);
        const uint32_t em = any ? bm : closest;
        const uint32_t who = em ? (uint32_t)__ffs(em) - 1u : 0u;
        const float wt = g.shfl(bt, who), wu = g.shfl(bu, who), wv = g.shfl(bv, who);
        const uint32_t wtri = g.shfl(btri, who);
        if (bm) {
          h.t = wt;
          h.u = wu;
          h.v = wv;
          h.tri = wtri;
          h.inst = cur_inst;
          if (any) active = false;
        }
      }
    }
    if (have_node && next_d >= h.t) have_node = false;  // a leaf above is closer than the next node
  }
};

}  // namespace nbd
