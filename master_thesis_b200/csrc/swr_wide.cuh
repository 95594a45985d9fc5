// Closest hit of one ray by eight lanes of a warp: each lane tests one child of the ray's node, then
// one of its hit triangles. Device only; the hits are Traversal's (the arg-min over the same
// candidates, swr_bvh.cuh).
//
// A launch of few rays takes as long as its longest ray, and a lane that walks alone pays the whole
// step for each node: about 400 instructions, one after the other. Eight lanes need about a quarter
// of them per node, and all of a node's hit triangles cost one or two tests. Kernel time of a launch
// of 4,000 closest-hit queries, one lane and eight lanes per ray: 5,000 triangles 25.0 and 14.5 us,
// 50,000 triangles 33.8 and 16.5 us, a 0.5 M-triangle terrain 49.9 and 28.0 us, the Cornell box 12.2
// and 7.9 us.
//
// These are kernels of their own: as a branch of the one-lane kernels, or a call from them, they cost
// these spills (terrain image 4 to 6 % slower). The host picks them by what it knows: the number of
// queries or pixels, or for the wavefront's rounds the paths in flight, which bound every round.
#pragma once

#include "swr_bvh.cuh"

namespace swrx {

// Launches of at most this many rays give each ray eight lanes: about as many as the GPU holds groups
// of eight at once (10 blocks of 16 on each of 148 SMs). With 24,000 rays the time is 18.2 against
// 27.6 us (5,000 triangles), 24.0 against 41.9 (50,000), 36.1 against 61.0 (terrain) and 11.0 against
// 12.8 (Cornell); with 40,000 it is 28.6 / 30.4, 30.8 / 43.2, 62.2 / 67.1 and 16.9 / 13.3.
constexpr unsigned kWideRays = 24000;
constexpr int kWideLanes = 8;
constexpr int kWideGroups = kTraceThreads / kWideLanes;  // per block
static_assert(kWideGroups * kStackTotal <= kTraceRows * kTraceThreads, "the groups' stacks fit the rows");

struct WideHit {
  uint32_t slot;
  float t, d2;
};

// The calling lane's group works on one ray (o, d), the same in its eight lanes; mem: the block's
// rows, of which the group uses its own kStackTotal entries. kStrict: the slab tests are made on every
// candidate from the start (DevScene::ray_flags; a template parameter, since a flag read at run time took
// one more register, which these kernels spill: 12,000 queries of the tessellated Cornell box 37.8 against
// 37.0 us).
template <bool kStats, int kRule, bool kStrict>
__device__ __forceinline__ WideHit wide_closest(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                             const float* __restrict__ tri_boxes, const float* __restrict__ obj_boxes,
                                             f3 o, f3 d, uint2* mem, TraceStats* stats) {
  const uint32_t c = threadIdx.x & 7u, shift = threadIdx.x & 24u;
  const uint32_t gmask = 0xFFu << shift;
  uint2* stack = mem + (threadIdx.x / kWideLanes) * kStackTotal;
  const float tiny = 1e-20f;
  const float idx = 1.0f / ((fabsf(d.x) < tiny) ? copysignf(tiny, d.x) : d.x);
  const float idy = 1.0f / ((fabsf(d.y) < tiny) ? copysignf(tiny, d.y) : d.y);
  const float idz = 1.0f / ((fabsf(d.z) < tiny) ? copysignf(tiny, d.z) : d.z);
  const uint32_t oct = (idx < 0.0f ? 1u : 0u) | (idy < 0.0f ? 2u : 0u) | (idz < 0.0f ? 4u : 0u);
  // plane bytes of this lane's child, near and far by direction sign: byte offsets in the node
  const uint32_t nx = 32u + c + ((oct & 1u) ? 24u : 0u), fx = 32u + c + ((oct & 1u) ? 0u : 24u);
  const uint32_t ny = 40u + c + ((oct & 2u) ? 24u : 0u), fy = 40u + c + ((oct & 2u) ? 0u : 24u);
  const uint32_t nz = 48u + c + ((oct & 4u) ? 24u : 0u), fz = 48u + c + ((oct & 4u) ? 0u : 24u);
  for (bool strict = kStrict;; strict = true) {
    uint32_t bslot = 0xFFFFFFFFu, bkey = 0xFFFFFFFFu;
    float bt = INFINITY, bd2 = INFINITY, tprune = INFINITY;
    uint2 ng = make_uint2(0u, (1u << (24 + oct)) | 1u);
    int sp = 0;
    for (;;) {
      while (ng.y & 0xFF000000u) {
        const uint32_t k = (uint32_t)__ffs(ng.y >> 24) - 1u;
        ng.y &= ~(1u << (24 + k));
        const uint32_t child = ng.x + (uint32_t)__popc(ng.y & ((1u << (k ^ oct)) - 1u) & 0xFFu);
        if (ng.y & 0xFF000000u) {
          if (c == 0u) stack[sp] = ng;
          ++sp;
        }
        if (kStats && c == 0u) stats->nodes++;
        const float4* np = nodes + (size_t)child * kNodeF4;
        const unsigned char* nb = (const unsigned char*)np;
        const float4 n0 = __ldg(np), n1 = __ldg(np + 1);
        const uint32_t qnx = __ldg(nb + nx), qny = __ldg(nb + ny), qnz = __ldg(nb + nz);
        const uint32_t qfx = __ldg(nb + fx), qfy = __ldg(nb + fy), qfz = __ldg(nb + fz);
        const uint32_t hdr = f2bits(n0.w);
        const float ax = bits2f((hdr & 0xFFu) << 23) * idx, ay = bits2f(((hdr >> 8) & 0xFFu) << 23) * idy,
                    az = bits2f(((hdr >> 16) & 0xFFu) << 23) * idz;
        const uint32_t imask = hdr >> 24;
        const float bx = (n0.x - o.x) * idx, by = (n0.y - o.y) * idy, bz = (n0.z - o.z) * idz;
        const float tn = fmax3_relu(fmaf(plane_level(qnx, 0), ax, bx), fmaf(plane_level(qny, 0), ay, by),
                                    fmaf(plane_level(qnz, 0), az, bz));
        const float tf = fmin3(fmaf(plane_level(qfx, 0), ax, bx), fmaf(plane_level(qfy, 0), ay, by),
                               fminf(fmaf(plane_level(qfz, 0), az, bz), tprune));
        const bool hit = (f2bits(fsub(tf, tn)) >> 31) == 0u;
        const uint32_t hm = (__ballot_sync(gmask, hit) >> shift) & 0xFFu;
        const uint32_t m = byte_of(f2bits(n1.z), f2bits(n1.w), c);
        uint32_t trih = 0;
        if (hm & ~imask) trih = __reduce_or_sync(gmask, hit ? bit_run(m & 31u, m >> 5) : 0u);
        ng = make_uint2(f2bits(n1.x), (slots_to_visit_order(hm & imask, oct) << 24) | imask);
        // the node's hit triangles, eight at a time
        for (uint32_t j = c; trih; j += 8u, trih >>= 8) {
          if (!(trih & 0xFFu)) continue;
          uint32_t key = 0xFFFFFFFFu, order = 0xFFFFFFFFu;  // distance bits, tie-break
          const uint32_t s = f2bits(n1.y) + j;
          float t = 0.0f, d2 = 0.0f;
          if ((trih >> c) & 1u) {
            if (kStats) stats->tris++;
            const float4* tp = tris + (size_t)s * kTriF4;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), e = __ldg(tp + 2);
            if (ref_intersect(o, d, mk(a.x, a.y, a.z), mk(a.w, b.x, b.y), mk(b.z, b.w, e.x), t, d2)) {
              const float dist = kRule == kRuleRayQuery ? t : d2, best = kRule == kRuleRayQuery ? bt : bd2;
              const uint32_t tie = f2bits(kRule == kRuleRayQuery ? e.y : e.z);
              bool ok = dist < best || (dist == best && tie < bkey);
              if (kRule == kRuleRayQuery) ok = ok && t >= kRqTmin && t <= kRqTmax;
              if (ok && strict) {
                const uint32_t obj = f2bits(e.w);
                const f3 inv = vinv(d);
                ok = ref_slab(tri_boxes + (size_t)s * 6, tri_boxes + (size_t)s * 6 + 3, o, inv) &&
                     ref_slab(obj_boxes + (size_t)obj * 6, obj_boxes + (size_t)obj * 6 + 3, o, inv);
              }
              if (ok) {
                key = f2bits(dist);  // not negative: ordered as its bits
                order = tie;
              }
            }
          }
          const uint32_t kmin = __reduce_min_sync(gmask, key);
          if (kmin != 0xFFFFFFFFu) {
            const uint32_t omin = __reduce_min_sync(gmask, key == kmin ? order : 0xFFFFFFFFu);
            const uint32_t who = __ballot_sync(gmask, key == kmin && order == omin);
            const int src = __ffs(who) - 1;
            bslot = __shfl_sync(gmask, s, src);
            bt = __shfl_sync(gmask, t, src);
            bd2 = __shfl_sync(gmask, d2, src);
            bkey = omin;
            tprune = bt * kPruneSlack;
          }
        }
      }
      if (sp == 0) break;
      --sp;
      __syncwarp(gmask);
      ng = stack[sp];
      __syncwarp(gmask);
    }
    bool settled = true;
    if (kRule == kRuleReference && bslot != 0xFFFFFFFFu && !strict) {
      const uint32_t obj = f2bits(__ldg(tris + (size_t)bslot * kTriF4 + 2).w);
      const f3 inv = vinv(d);
      settled = ref_slab(tri_boxes + (size_t)bslot * 6, tri_boxes + (size_t)bslot * 6 + 3, o, inv) &&
                ref_slab(obj_boxes + (size_t)obj * 6, obj_boxes + (size_t)obj * 6 + 3, o, inv);
    }
    if (settled) return WideHit{bslot, bt, bd2};
  }
}

// First ray of the calling lane's group in a launch of a full grid, and the stride to its next: rays
// go to one group of every warp before any warp gets a second one.
__device__ __forceinline__ uint32_t wide_first() {
  const uint32_t warps = gridDim.x * (kTraceThreads / 32);
  return blockIdx.x * (kTraceThreads / 32) + (threadIdx.x >> 5) + warps * ((threadIdx.x & 31u) >> 3);
}
__device__ __forceinline__ uint32_t wide_stride() { return gridDim.x * kWideGroups; }

}  // namespace swrx
