// Compressed 8-wide BVH and the closest-hit traversal with the reference's hit semantics.
//
// Node record: 80 bytes = five float4, 16-byte aligned (every node touches exactly three 32-byte
// sectors). Child boxes are quantised to 8 bits per plane on a per-node power-of-two grid
// (after Ylitie, Karras, Laine, "Efficient Incoherent Ray Traversal on GPUs Through Compressed
// Wide BVHs", HPG 2017); the encoding details below are this project's own.
//
//   f4[0] = p.x p.y p.z | ex | ey<<8 | ez<<16 | imask<<24     grid origin, exponents, inner mask
//           (a plane byte q lies at p + level(q) * 2^e, plane_grid.h)
//   f4[1] = child_base | tri_base | meta[0..3] | meta[4..7]    meta = (count<<5)|offset for leaf
//                                                               slots, 0 for inner/empty slots
//   f4[2] = qlo_x[0..7] | qlo_y[0..7]
//   f4[3] = qlo_z[0..7] | qhi_x[0..7]
//   f4[4] = qhi_y[0..7] | qhi_z[0..7]
//
// Inner children of a node are stored contiguously from child_base in increasing slot order;
// triangles of its leaf children contiguously from tri_base (at most 24 per node, at most 3 per
// leaf). The builder places children so that slot s holds the child lying towards octant corner s;
// a ray whose direction has sign bits `oct` visits slots in increasing (s ^ oct), near to far.
//
// Triangle record: 48 bytes = three float4:
//   v0.x v0.y v0.z e0.x | e0.y e0.z e1.x e1.y | e1.z id rank obj
// where e0 = v1 - v0, e1 = v2 - v0 exactly as the reference's Triangle computes them, id is the
// global triangle id, rank its position in the reference's visit order (ties), obj its object.
//
// Hit rule (what makes the result bit-identical to Scene::traceRay, scene.cpp:22-56): the
// reference tests every triangle whose own box and whose object's box pass its slab test, with
// its Moller-Trumbore arithmetic, and keeps the smallest squared distance, the first in its
// visit order on ties. Here candidates come from the wide BVH (boxes conservatively enlarged,
// nodes farther than the current best times (1 + 2^-10) pruned), and the best by (distance^2, rank)
// is kept without the slab tests. Only the finished ray's hit is put to both reference slab tests
// (Traversal::settled): when it passes, it is the best of all candidates and a valid one, so it is
// the best valid one; when it fails (a hit on the very rim of its triangle's box), the ray is
// traced once more with the tests made on every candidate (in scenes where whole walls fail, they are
// made on every candidate from the start: DevScene::ray_flags). The kernels settle the finished rays of
// a warp together, at the next refill: the tests are a third of a step's instructions, and made at
// each acceptance they ran for one or two lanes in nearly every step of a warp.
#pragma once

#include "plane_grid.h"
#include "swr_exact.cuh"

namespace swrx {

constexpr int kNodeF4 = 5;
constexpr int kTriF4 = 3;
// Lanes of a warp with a triangle left that keep a step testing (kTriLoop). RayTrace frame and path
// traced image of the Cornell box, ms: 1.07 and 0.94 without the loop; 0.86 and 0.85 with 2 lanes,
// 0.88 and 0.84 with 4, 0.91 and 0.85 with 6, 0.96 and 0.85 with 10.
constexpr int kTriLoopLanes = 4;
// Scenes of at most this many triangles take the kernels with kTriLoop: their trees are a few levels
// deep and their rays test more triangles than nodes (Cornell: 3.5 and 1.4). Image, RayTrace frame,
// bidirectional image, adjoint: Cornell -10, -17, -7, -15 %; 1,000 triangles -2 to -8 %; 2,700 to
// 47,000 triangles within 2 % either way; 200,000 triangles and terrains +3 % and more.
constexpr uint32_t kFewTriangles = 2048;
// The same for closest-hit queries, whose rays are less alike: Cornell -16, 1,000 triangles -10,
// 5,000 -5, 30,000 and 47,000 -2 %, a 2.4 M-triangle terrain +1.5 %. Batches always take it (64
// uneven scenes of 1,000 to 50,000 triangles: 1.82 -> 1.78 ms).
constexpr uint32_t kFewTrianglesQuery = 1u << 16;
constexpr int kTraceThreads = 128;  // block size of every traversal kernel
constexpr int kStackShared = 8;   // stack entries per thread kept in shared memory
// Shared memory of a traversal kernel: rows of one 8-byte entry per thread. Rows 0..7 are the top
// of the stack; then (hit slot, hit t), (hit squared distance, flags) and one row for the kernel's
// own use (the index of the lane's ray). What a ray writes only when it finds a closer hit, and
// reads only when a triangle passes the intersection test, would cost registers for its whole walk:
// with these rows the bounce traversal runs in 48 registers without spills, 10 blocks per SM instead
// of 9 (terrain image 18.1 -> 17.5 ms of bounce traversal, 16.4 -> 16.0 after the child loop below).
// 40 registers (12 blocks) spill and lose 8 %.
constexpr int kRowHit = kStackShared, kRowDist = kStackShared + 1, kRowUser = kStackShared + 2;
constexpr int kTraceRows = kStackShared + 3;
constexpr int kTraceMem = kTraceRows + 2;  // two more rows: the visit-order table (Traversal::prepare)
constexpr int kStackTotal = 64;   // maximum traversal stack depth (checked at build time)
constexpr float kPruneSlack = 1.0f + 1.0f / 1024.0f;

// Hit rules of Traversal::step.
//   kRuleReference  the software renderer's: smallest (squared distance, visit rank) among the
//                   triangles whose reference slab tests pass (see above).
//   kRuleRayQuery   the closest hit that the Vulkan renderers ask the ray tracing pipeline for
//                   (traceRay, v1.glsl:148-161: opaque geometry, tmin 0.001, tmax 10000): the
//                   smallest t in [kRqTmin, kRqTmax], ties to the lower triangle id, with the same
//                   Moller-Trumbore arithmetic; hit.d2 is left unset.
enum HitRule : int { kRuleReference = 0, kRuleRayQuery = 1 };
constexpr float kRqTmin = 0.001f;
constexpr float kRqTmax = 10000.0f;

struct Hit {
  uint32_t slot;   // index into the triangle records, 0xFFFFFFFF on a miss
  uint32_t id;     // global triangle id
  uint32_t rank;
  uint32_t obj;
  float t;
  float d2;
};

struct TraceStats {
  uint32_t nodes;
  uint32_t tris;
};

// Node groups and postponed triangle groups share the stack; triangle groups carry kTriGroup in .x.
constexpr uint32_t kTriGroup = 0x80000000u;

// The rows of one thread. On the device `at` is the shared-memory address of the next free stack
// entry: the block's rows are 1024-byte aligned and 1024 bytes apart, so it holds the stack depth
// and the thread's column at once, and the array's own address is a constant of the kernel. Entries
// beyond the shared rows go to thread-local memory.
struct TraceRows {
#if defined(__CUDA_ARCH__)
  static constexpr uint32_t kRow = kTraceThreads * (uint32_t)sizeof(uint2);
  uint32_t at;
#else
  uint2* rows;
  uint2 own[3];
  int sp;
#endif
  uint2 local[kStackTotal - kStackShared];

#if defined(__CUDA_ARCH__)
  static __device__ __forceinline__ uint32_t base(const uint2* mem) { return (uint32_t)__cvta_generic_to_shared(mem); }
  static __device__ __forceinline__ uint2 lds(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
  }
  static __device__ __forceinline__ uint32_t lds_u8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
  }
  static __device__ __forceinline__ void sts(uint32_t a, uint2 v) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(v.x), "r"(v.y) : "memory");
  }
  __device__ __forceinline__ uint32_t row(const uint2* mem, int r) const {
    return base(mem) + (uint32_t)r * kRow + (at & (kRow - 1u));
  }
  __device__ __forceinline__ void bind(uint2* mem) { at = base(mem) + threadIdx.x * (uint32_t)sizeof(uint2); }
  __device__ __forceinline__ bool empty(const uint2* mem) const { return at < base(mem) + kRow; }
  __device__ __forceinline__ void clear(const uint2* mem) { at = row(mem, 0); }
  __device__ __forceinline__ void push(const uint2* mem, uint2 v) {
    if (at < base(mem) + kStackShared * kRow) sts(at, v);
    else local[(at - base(mem)) / kRow - kStackShared] = v;
    at += kRow;
  }
  __device__ __forceinline__ uint2 pop(const uint2* mem) {
    at -= kRow;
    return at < base(mem) + kStackShared * kRow ? lds(at) : local[(at - base(mem)) / kRow - kStackShared];
  }
  __device__ __forceinline__ uint2 get(const uint2* mem, int r) const { return lds(row(mem, r)); }
  __device__ __forceinline__ void set(uint2* mem, int r, uint2 v) { sts(row(mem, r), v); }
#else
  void bind(uint2* mem) {
    rows = mem;
    sp = 0;
  }
  bool empty(const uint2*) const { return sp == 0; }
  void clear(const uint2*) { sp = 0; }
  void push(const uint2*, uint2 v) {
    if (sp < kStackShared) rows[sp] = v;
    else local[sp - kStackShared] = v;
    ++sp;
  }
  uint2 pop(const uint2*) {
    --sp;
    return sp < kStackShared ? rows[sp] : local[sp - kStackShared];
  }
  uint2 get(const uint2*, int r) const { return own[r - kStackShared]; }
  void set(uint2*, int r, uint2 v) { own[r - kStackShared] = v; }
#endif
};

SWR_HD float4 ldg4(const float4* p) {
#if defined(__CUDA_ARCH__)
  return __ldg(p);
#else
  return *p;
#endif
}

// min of three floats, NaN operands ignored as by fminf
SWR_HD float fmin3(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fminf(fminf(a, b), c);
#endif
}

// max(a, b, c, 0): as integers, floats above zero compare as floats do and those below are negative.
// (A NaN, which only overflowing coordinates give, makes the box test pass.)
SWR_HD float fmax3_relu(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __int_as_float(__vimax3_s32_relu(__float_as_int(a), __float_as_int(b), __float_as_int(c)));
#else
  return fmaxf(fmaxf(a, b), fmaxf(c, 0.0f));
#endif
}
// (x0, y0) = (a0 * b0 + c0, a1 * b1 + c1), each rounded once: one instruction for both on the device
SWR_HD void fma2(float a0, float a1, float b0, float b1, float c0, float c1, float& x0, float& x1) {
#if defined(__CUDA_ARCH__)
  asm("{.reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
      " fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;}"
      : "=f"(x0), "=f"(x1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
#else
  x0 = fmaf(a0, b0, c0);
  x1 = fmaf(a1, b1, c1);
#endif
}
// m shifted left by one with x's sign let in
SWR_HD uint32_t push_sign(uint32_t m, float x) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(__float_as_uint(x), m, 1);
#else
  return (m << 1) | (x < 0.0f ? 1u : 0u);
#endif
}
// byte k (0..7) of the pair (lo, hi)
SWR_HD uint32_t byte_of(uint32_t lo, uint32_t hi, uint32_t k) {
#if defined(__CUDA_ARCH__)
  return __byte_perm(lo, hi, 0x4440u + k) & 0xFFu;
#else
  return ((k < 4 ? lo : hi) >> (8 * (k & 3))) & 0xFFu;
#endif
}

// `width` one bits starting at bit `pos` (pos < 32, width <= 8 here); zero when width is 0.
SWR_HD uint32_t bit_run(uint32_t pos, uint32_t width) {
#if defined(__CUDA_ARCH__)
  uint32_t r;
  asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(r) : "r"(pos), "r"(width));
  return r;
#else
  return ((1u << width) - 1u) << pos;
#endif
}

// An 8-bit slot mask moved into visit order: bit s goes to bit s ^ oct.
SWR_HD uint32_t slots_to_visit_order(uint32_t m, uint32_t oct) {
  if (oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
  if (oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
  if (oct & 4u) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
  return m;
}

// Resumable closest-hit traversal of one ray: init() sets the ray up, each step() expands at
// most one wide node and tests the triangles of its hit leaves, and returns true once the ray is
// finished (hit holds the result). The persistent kernels keep one Traversal per lane and refill
// lanes whose ray finished; trace_closest() runs a single ray to completion.
struct Traversal {
  static constexpr uint32_t kAny = 1u;     // occlusion query: stop at the first accepted candidate
  static constexpr uint32_t kStrict = 2u;  // slab tests on every candidate (after a failed settled())
  f3 o, d;
  float idx, idy, idz;  // traversal reciprocal (zero components replaced by a tiny value)
  uint32_t oct;
  float tprune;
  uint2 ng;  // node group: x = child_base, y = hits (bits 24..31, visit order) | imask (bits 0..7)
  uint2 tg;  // triangle group: x = base, y = hit bits 0..23
  TraceRows st;
  uint32_t host_turn;  // host build only: drives the alternating postponing decision

  // Before the first ray: the block's visit-order table, [oct][slot mask] -> mask in visit order (one
  // shared-memory byte instead of 13 instructions per node), by all threads of the block.
  static SWR_HD void prepare(uint2* mem) {
#if defined(__CUDA_ARCH__)
    uint32_t* t = (uint32_t*)(mem + kTraceRows * kTraceThreads);
    for (uint32_t k = threadIdx.x; k < 512u; k += kTraceThreads) {
      uint32_t w = 0;
      for (uint32_t b = 0; b < 4; ++b) w |= slots_to_visit_order((4 * k + b) & 0xFFu, k >> 6) << (8 * b);
      t[k] = w;
    }
    __syncthreads();
#endif
  }
  SWR_HD void setup(uint2* mem) {
    st.bind(mem);
    prepare(mem);
  }
  // mem: the block's kTraceMem rows (a kernel's own 1024-byte aligned array, so that its address is a
  // constant), of which prepare() has filled the last two
  // flags: 0, or kStrict for the slab tests on every candidate from the start (DevScene::ray_flags)
  SWR_HD void init(f3 o_, f3 d_, uint2* mem, uint32_t flags = 0u) {
    o = o_;
    d = d_;
    host_turn = f2bits(o_.x) ^ f2bits(d_.y);
    const float tiny = 1e-20f;
    const float dx = (fabsf(d.x) < tiny) ? copysignf(tiny, d.x) : d.x;
    const float dy = (fabsf(d.y) < tiny) ? copysignf(tiny, d.y) : d.y;
    const float dz = (fabsf(d.z) < tiny) ? copysignf(tiny, d.z) : d.z;
    idx = 1.0f / dx;
    idy = 1.0f / dy;
    idz = 1.0f / dz;
    oct = (idx < 0.0f ? 1u : 0u) | (idy < 0.0f ? 2u : 0u) | (idz < 0.0f ? 4u : 0u);
    st.bind(mem);
    start(mem, flags, INFINITY);
  }

  // the ray at the root, with no hit yet
  SWR_HD void start(uint2* mem, uint32_t flags, float d2) {
    tprune = INFINITY;
    st.clear(mem);
    st.set(mem, kRowHit, make_uint2(0xFFFFFFFFu, f2bits(INFINITY)));
    st.set(mem, kRowDist, make_uint2(f2bits(d2), flags));
    ng = make_uint2(0u, (1u << (24 + oct)) | 1u);  // the root, as inner slot 0
    tg = make_uint2(0u, 0u);
  }

  // Occlusion query (Scene::isOccluded, scene.cpp:58-83): finished at the first candidate whose
  // squared distance is <= dist2; the hit slot stays 0xFFFFFFFF when there is none. The candidate
  // rule is the closest-hit one started from a best of (dist2, no rank), whose first acceptance is
  // exactly "d2 <= dist2"; nodes beyond sqrt(dist2) (with the pruning slack) are skipped, which
  // keeps every such candidate because d is of unit length.
  SWR_HD void init_occlusion(f3 o_, f3 d_, float dist2, uint2* mem, uint32_t flags = 0u) {
    init(o_, d_, mem);
    start(mem, kAny | flags, dist2);
    tprune = sqrtf(dist2) * kPruneSlack;
  }

  SWR_HD uint32_t hit_slot(const uint2* mem) const { return st.get(mem, kRowHit).x; }
  SWR_HD float hit_t(const uint2* mem) const { return bits2f(st.get(mem, kRowHit).y); }
  // A finished, settled ray made from a stored hit (a sample that starts at its camera record): the
  // kernels whose lanes wait for one another between rays keep nothing of a ray but this object.
  SWR_HD void resume(f3 o_, f3 d_, uint32_t slot, float t, uint2* mem) {
    o = o_;
    d = d_;
    st.set(mem, kRowHit, make_uint2(slot, f2bits(t)));
    st.set(mem, kRowDist, make_uint2(0u, kStrict));
  }

  // Whether a finished ray's hit stands: always for a miss (no candidate at all) and after a strict
  // pass; otherwise when the hit triangle's and its object's reference boxes pass the slab test.
  SWR_HD bool settled(const float4* __restrict__ tris, const float* __restrict__ tri_boxes,
                      const float* __restrict__ obj_boxes, const uint2* mem) const {
    const uint32_t s = hit_slot(mem);
    return s == 0xFFFFFFFFu || (st.get(mem, kRowDist).y & kStrict) || boxes_hit(s, tris, tri_boxes, obj_boxes);
  }
  // Starts the ray again with the slab tests made on every candidate.
  SWR_HD void start_strict(uint2* mem) { start(mem, kStrict, INFINITY); }
  SWR_HD void start_occlusion_strict(float dist2, uint2* mem) {
    start(mem, kAny | kStrict, dist2);
    tprune = sqrtf(dist2) * kPruneSlack;
  }
  SWR_HD bool boxes_hit(uint32_t s, const float4* __restrict__ tris, const float* __restrict__ tri_boxes,
                        const float* __restrict__ obj_boxes) const {
    const uint32_t obj = f2bits(ldg4(tris + (size_t)s * kTriF4 + 2).w);
    const f3 inv = vinv(d);  // exact reciprocal of the reference's slab tests
    return ref_slab(tri_boxes + (size_t)s * 6, tri_boxes + (size_t)s * 6 + 3, o, inv) &&
           ref_slab(obj_boxes + (size_t)obj * 6, obj_boxes + (size_t)obj * 6 + 3, o, inv);
  }
  // A record's tie-break key: the visit rank, or the triangle id for ray queries; above every key
  // when there is no hit.
  template <int kRule>
  SWR_HD uint32_t key_of(uint32_t s, const float4* __restrict__ tris) const {
    if (s == 0xFFFFFFFFu) return 0xFFFFFFFFu;
    const float4 c = ldg4(tris + (size_t)s * kTriF4 + 2);
    return f2bits(kRule == kRuleRayQuery ? c.y : c.z);
  }

  // The finished ray's hit with its triangle id and object read from the triangle record.
  SWR_HD Hit result(const float4* __restrict__ tris, const uint2* mem) const {
    Hit h;
    const uint2 w = st.get(mem, kRowHit);
    h.slot = w.x;
    h.t = bits2f(w.y);
    h.d2 = bits2f(st.get(mem, kRowDist).x);
    h.id = h.rank = h.obj = 0xFFFFFFFFu;
    if (h.slot != 0xFFFFFFFFu) {
      const float4 c = ldg4(tris + (size_t)h.slot * kTriF4 + 2);
      h.id = f2bits(c.y);
      h.rank = f2bits(c.z);
      h.obj = f2bits(c.w);
    }
    return h;
  }

  template <bool kStats, int kRule, bool kFlat>
  SWR_HD void test_triangle(const float4* __restrict__ tris, const float* __restrict__ tri_boxes,
                            const float* __restrict__ obj_boxes, uint2* mem, TraceStats* stats) {
    do {
      const uint32_t j = (uint32_t)ffs(tg.y) - 1u;
      tg.y &= tg.y - 1u;
      const uint32_t s = tg.x + j;
      if (kStats) stats->tris++;
      const float4* tp = tris + (size_t)s * kTriF4;
      const float4 a = ldg4(tp + 0), b = ldg4(tp + 1), c = ldg4(tp + 2);
      float t, d2;
      if (!ref_intersect<kFlat>(o, d, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, c.x), t, d2)) break;
      const uint2 w = st.get(mem, kRowHit);  // (slot, t) of the best hit so far
      if (kRule == kRuleRayQuery) {
        if (!(t >= kRqTmin && t <= kRqTmax)) break;
        const float bt = bits2f(w.y);
        if (!(t < bt || (t == bt && f2bits(c.y) < key_of<kRule>(w.x, tris)))) break;
        st.set(mem, kRowHit, make_uint2(s, f2bits(t)));
        tprune = t * kPruneSlack;
        break;
      }
      const uint2 v = st.get(mem, kRowDist);
      const float bd2 = bits2f(v.x);
      if (!(d2 < bd2 || (d2 == bd2 && f2bits(c.z) < key_of<kRule>(w.x, tris)))) break;
      if ((v.y & kStrict) && !boxes_hit(s, tris, tri_boxes, obj_boxes)) break;
      st.set(mem, kRowHit, make_uint2(s, f2bits(t)));
      st.set(mem, kRowDist, make_uint2(f2bits(d2), v.y));
      tprune = t * kPruneSlack;
      if (v.y & kAny) {  // occluded: drop the remaining work so the pop below ends the query
        ng.y = 0u;
        tg.y = 0u;
        st.clear(mem);
      }
    } while (false);
  }

  // kPostpone: triangle postponing. While fewer than a fifth of the warp's active lanes have
  // triangles to test, a lane that could still expand nodes parks its triangle group on its
  // stack, so the warp runs one phase at a time. Without it a lane with pending triangles tests
  // one of them per step and a lane without expands a node. (The visit order never changes the
  // result: the closest hit is an arg-min over the same candidates.)
  // kTriLoop: the lanes with more triangles go on testing them while enough of the warp's lanes
  // have some (below).
  template <bool kStats, bool kPostpone = false, int kRule = kRuleReference, bool kTriLoop = false,
            bool kFlat = false>
  SWR_HD bool step(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                   const float* __restrict__ tri_boxes, const float* __restrict__ obj_boxes,
                   uint2* mem, TraceStats* stats) {
    const bool has_nodes = (ng.y & 0xFF000000u) != 0;
    bool tri_now = tg.y != 0;
    if (kPostpone) {
#if defined(__CUDA_ARCH__)
      const unsigned act = __activemask();
      const unsigned with_tris = __ballot_sync(act, tg.y != 0);
      tri_now = tri_now && (!has_nodes || __popc(with_tris) * 5 >= __popc(act));
#else
      // host build: alternate the decision deterministically so both paths are exercised
      tri_now = tri_now && (!has_nodes || ((host_turn++ * 2654435761u) >> 31) != 0);
#endif
    }
    if (!tri_now && has_nodes) {
      if (tg.y) {
        st.push(mem, make_uint2(tg.x | kTriGroup, tg.y));
        tg.y = 0;
      }
      const uint32_t k = (uint32_t)ffs(ng.y >> 24) - 1u;
      ng.y &= ~(1u << (24 + k));
      const uint32_t slot = k ^ oct;
      const uint32_t child = ng.x + (uint32_t)popc(ng.y & ((1u << slot) - 1u) & 0xFFu);
      if (ng.y & 0xFF000000u) st.push(mem, ng);
      if (kStats) stats->nodes++;

      const float4* np = nodes + (size_t)child * kNodeF4;
      const float4 n0 = ldg4(np + 0), n1 = ldg4(np + 1), n2 = ldg4(np + 2);
      const float4 n3 = ldg4(np + 3), n4 = ldg4(np + 4);
      const uint32_t hdr = f2bits(n0.w);
      const float ex = bits2f((hdr & 0xFFu) << 23);
      const float ey = bits2f(((hdr >> 8) & 0xFFu) << 23);
      const float ez = bits2f(((hdr >> 16) & 0xFFu) << 23);
      const uint32_t imask = hdr >> 24;
      const float ax = ex * idx, ay = ey * idy, az = ez * idz;
      const float bx = (n0.x - o.x) * idx, by = (n0.y - o.y) * idy, bz = (n0.z - o.z) * idz;
      // near/far plane bytes by direction sign
      const uint32_t lox0 = f2bits(n2.x), lox1 = f2bits(n2.y), loy0 = f2bits(n2.z), loy1 = f2bits(n2.w);
      const uint32_t loz0 = f2bits(n3.x), loz1 = f2bits(n3.y), hix0 = f2bits(n3.z), hix1 = f2bits(n3.w);
      const uint32_t hiy0 = f2bits(n4.x), hiy1 = f2bits(n4.y), hiz0 = f2bits(n4.z), hiz1 = f2bits(n4.w);
      const uint32_t nx0 = (oct & 1u) ? hix0 : lox0, nx1 = (oct & 1u) ? hix1 : lox1;
      const uint32_t fx0 = (oct & 1u) ? lox0 : hix0, fx1 = (oct & 1u) ? lox1 : hix1;
      const uint32_t ny0 = (oct & 2u) ? hiy0 : loy0, ny1 = (oct & 2u) ? hiy1 : loy1;
      const uint32_t fy0 = (oct & 2u) ? loy0 : hiy0, fy1 = (oct & 2u) ? loy1 : hiy1;
      const uint32_t nz0 = (oct & 4u) ? hiz0 : loz0, nz1 = (oct & 4u) ? hiz1 : loz1;
      const uint32_t fz0 = (oct & 4u) ? loz0 : hiz0, fz1 = (oct & 4u) ? loz1 : hiz1;
      const uint32_t meta0 = f2bits(n1.z), meta1 = f2bits(n1.w);
      // Branch-free child loop, last slot first: what bounds it is the integer pipe (two cycles per
      // instruction and warp; it also runs min, max, permutes and selects), so the work is put where
      // that pipe is not: the comparison is a subtraction whose sign bit the funnel shift collects,
      // the maximum with zero rides on a three-way integer maximum, and the triangle runs are looked
      // up for the hit leaves only. Bounce traversal of the terrain image: 17.5 ms with a set and a
      // select per slot and every slot's run, 17.1 with the leaf loop, 16.7 with the sign bits, 16.4
      // with the integer maximum, at 9 blocks per SM.
      uint32_t miss = 0;
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        const float qnx = plane_level(i < 4 ? nx0 : nx1, i & 3);
        const float qny = plane_level(i < 4 ? ny0 : ny1, i & 3);
        const float qnz = plane_level(i < 4 ? nz0 : nz1, i & 3);
        const float qfx = plane_level(i < 4 ? fx0 : fx1, i & 3);
        const float qfy = plane_level(i < 4 ? fy0 : fy1, i & 3);
        const float qfz = plane_level(i < 4 ? fz0 : fz1, i & 3);
        float tnx, tny, tnz, tfx, tfy, tfz;
        fma2(qnx, qny, ax, ay, bx, by, tnx, tny);
        fma2(qfx, qfy, ax, ay, bx, by, tfx, tfy);
        tnz = fmaf(qnz, az, bz);
        tfz = fmaf(qfz, az, bz);
        const float tn = fmax3_relu(tnx, tny, tnz);
        const float tf = fmin3(tfx, tfy, fminf(tfz, tprune));
        miss = push_sign(miss, fsub(tf, tn));
      }
      const uint32_t hm = ~miss & 0xFFu;
      uint32_t trih = 0;  // an empty slot never passes the box test, and its run would be empty
      for (uint32_t leaves = hm & ~imask; leaves; leaves &= leaves - 1u) {
        const uint32_t m = byte_of(meta0, meta1, (uint32_t)ffs(leaves) - 1u);
        trih |= bit_run(m & 31u, m >> 5);
      }
#if defined(__CUDA_ARCH__)
      const uint32_t inner =
          TraceRows::lds_u8(TraceRows::base(mem) + kTraceRows * TraceRows::kRow + oct * 256u + (hm & imask));
#else
      const uint32_t inner = slots_to_visit_order(hm & imask, oct);
#endif
      ng = make_uint2(f2bits(n1.x), (inner << 24) | imask);
      tg = make_uint2(f2bits(n1.y), trih);
      if (kPostpone) return false;
      tri_now = true;
    }

    // One triangle per step: a lane with many candidate triangles then holds the warp for one test
    // per step while the other lanes go on expanding nodes (terrain image: testing all of them in the
    // step cost 16 %). With kTriLoop the step goes on as long as kTriLoopLanes lanes have a triangle
    // left: where nodes are few and most steps test triangles, the loop around the step (refill and
    // stage ballots) is what a test costs. See kFewTriangles.
    if (tri_now && tg.y) {
      for (;;) {
        test_triangle<kStats, kRule, kFlat>(tris, tri_boxes, obj_boxes, mem, stats);
        if (!kTriLoop) break;
        const bool more = tg.y != 0;
#if defined(__CUDA_ARCH__)
        if (__popc(__ballot_sync(__activemask(), more)) < kTriLoopLanes) break;
#endif
        if (!more) break;
      }
    }

    if (!(ng.y & 0xFF000000u) && tg.y == 0) {
      if (st.empty(mem)) return true;
      const uint2 g = st.pop(mem);
      if (g.x & kTriGroup) tg = make_uint2(g.x & ~kTriGroup, g.y);
      else ng = g;
    }
    return false;
  }
};

// Closest hit of ray (o, d), run to completion. obj_boxes/tri_boxes hold the reference's own
// boxes (lo.xyz, hi.xyz) per object and per triangle record; mem: the block's kTraceMem rows, after
// Traversal::prepare (host build: kStackShared entries); the int is not used. Returns false on a miss.
template <bool kStats, bool kPostpone = false, int kRule = kRuleReference>
SWR_HD bool trace_closest(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                          const float* __restrict__ tri_boxes, const float* __restrict__ obj_boxes,
                          f3 o, f3 d, uint2* mem, int, Hit& hit, TraceStats* stats, uint32_t flags = 0u) {
  Traversal tr;
  tr.init(o, d, mem, flags);
  for (;;) {
    while (!tr.template step<kStats, kPostpone, kRule>(nodes, tris, tri_boxes, obj_boxes, mem, stats)) {
    }
    if (kRule == kRuleRayQuery || tr.settled(tris, tri_boxes, obj_boxes, mem)) break;
    tr.start_strict(mem);
  }
  hit = tr.result(tris, mem);
  return hit.slot != 0xFFFFFFFFu;
}

}  // namespace swrx
