// A warp a ray: the watertight traversal of short queues.
//
// A queue of fewer rays than the GPU has warps lasts as long as its longest ray, and a ray on
// one lane is a chain of dependent fetches as long as the nodes it visits: 197 rays of a
// 100k-triangle view take 82 us on the BVH2, some 200 visits of about 350 ns. Here the 32
// lanes share one ray's traversal of the 8-wide tree. A step takes up to four entries off a
// stack in shared memory, eight lanes each: a node's lanes test its eight child boxes, a
// leaf's its triangles, all loads of a step in flight together; the children that are hit go
// back on the stack with one ballot. The chain is then the tree's levels plus a quarter of the
// entries, at the price of entries that a one-lane walk would have culled by a hit it finds
// first, which idle lanes pay.
//
// Entries come off nearest first: a node's children by direction octant (wide.cpp's slots), the
// groups' children in their parents' order. The triangles, their test and the tie rule (equal t:
// the smaller source id) are the BVH2's, so closest hits equal the other walks' bit for bit;
// any-hit answers agree on existence only (no caller that reports the hit takes this walk).
//
// The stack: an entry's children go on top of it, so entries of one level are all there are
// of it until they are gone (a step that takes one of a level takes every entry above), and
// a step leaves at most 31 of the level it takes from: 31 a level, and the last step's 32.
#pragma once

#include "traverse.cuh"

namespace lr {

// Rays a warp of the launch up to which a queue is walked a warp a ray, by the scene's
// triangles: the shallower the tree, the shorter the chain a lane would walk. Measured against
// the BVH2 walk on 4,736 warps: on a 34-triangle box 3,234 rays 26 -> 13 us, 14,009 27 -> 23,
// 19,807 25 -> 27; on a 15k-triangle box 16,851 76 -> 33, 56,286 78 -> 73; on 100k triangles 3,326
// 91 -> 20, 53,621 109 -> 100; on 1M 26,548 136 -> 67, 60,000 105 -> 95, 100,000 112 -> 146. In
// whole passes, where a round's shadow rays share the machine, 8 beats 12 on the 15k-triangle
// box (3,008 against 3,130 us) and 4 beats 8 on the 34-triangle one (637 against 662).
__host__ __device__ constexpr uint32_t warp_rays_for(uint64_t triangles) {
    return triangles < 1024u ? 4u : 8u;
}

constexpr uint32_t warp_stack_ints(uint32_t levels) { return 31u * levels + 32u; }

// Whether a scene's 8-wide tree can be walked by warps with `ints` words of stack each.
__host__ __device__ inline bool warp_walkable(const DeviceScene &s, uint32_t ints) {
    return s.wide8.boxes != nullptr && warp_stack_ints(s.wide8.max_stack) <= ints;
}

// From child slots to nearest-first ranks for a direction octant (bit s to bit s ^ oct).
__device__ __forceinline__ uint32_t octant_ranks(uint32_t mask, uint32_t oct) {
    if (oct & 1u) mask = ((mask & 0x55u) << 1) | ((mask >> 1) & 0x55u);
    if (oct & 2u) mask = ((mask & 0x33u) << 2) | ((mask >> 2) & 0x33u);
    if (oct & 4u) mask = ((mask & 0x0fu) << 4) | ((mask >> 4) & 0x0fu);
    return mask;
}

// The hit of ray `r`, the same on every lane of the warp, which calls it together with the
// same arguments; `stack` is the warp's, of `ints` words. Ends: a step takes entries of a
// finite tree off the stack for good.
template <bool kAny>
__device__ __forceinline__ Hit walk_warp(const DeviceScene &s, const Ray &r, int *stack, uint32_t ints, bool &overflow) {
    constexpr uint32_t kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, c = lane & 7u, group = lane >> 3;
    Hit h{r.tmax, -1, -1, 0.0f, 0.0f};  // the nearest of the triangles this lane tested
    if (s.bvh.empty) return h;
    const float3 inv = safe_inverse(r.d), oinv = neg_origin_times(r.o, inv);
    const Shear sh = make_shear(r.o, r.d);
    const uint32_t oct = (inv.x < 0.0f ? 1u : 0u) | (inv.y < 0.0f ? 2u : 0u) | (inv.z < 0.0f ? 4u : 0u);
    float bound = r.tmax;  // the nearest hit so far
    float limit = r.tmax;  // triangles hit before it, as ExactTracer's
    bool found = false;
    uint32_t sp = 0, taken = 1;
    int link = 0;  // this group's entry when group < taken: the root first
    for (;;) {
        const bool node = group < taken && link >= 0, leaf = group < taken && link < 0;
        uint32_t first = 0, n = 0;
        if (leaf) leaf_range(link, first, n);
        // A child's box and link, or a triangle: the loads of nodes and leaves go out together.
        const float4 *at = node ? s.wide8.boxes + ((size_t)(uint32_t)link * 16u + 2u * c) : s.tris + (size_t)(first + c) * 3u;
        float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f), q = p, v2 = p;
        if (node || c < n) {
            p = __ldg(at);
            q = __ldg(at + 1);
            if (leaf) v2 = __ldg(at + 2);
        }
        // Nodes first, against the hits so far.
        float entry = 0.0f;
        bool in = node && box_exact(p.x, q.x, p.y, q.y, p.z, q.z, inv, oinv, r.tmin, bound, entry) && q.w != 0.0f;
        if (__any_sync(kAll, leaf)) {
            bool better = false;
            for (uint32_t i = c; i < n; i += 8u) {
                float4 a = p, b = q, d = v2;
                if (i >= 8u) {
                    const float4 *tri = s.tris + (size_t)(first + i) * 3u;
                    a = __ldg(tri);
                    b = __ldg(tri + 1);
                    d = __ldg(tri + 2);
                }
                float t, u, v;
                if (!watertight(sh, r.tmin, limit, false, a, b, d, t, u, v)) continue;
                const int id = __float_as_int(a.w);
                if (h.id >= 0 && (t > h.t || (t == h.t && id > h.id))) continue;
                h = Hit{t, id, (int)(first + i), u, v};
                better = true;
            }
            if (__any_sync(kAll, better)) {
                found = true;
                if (kAny) break;
                float t = h.id >= 0 ? h.t : bound;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) t = fminf(t, __shfl_xor_sync(kAll, t, step));
                bound = t;
                limit = next_above(t);
                // Against this step's hits too, with the box test's slack: far from the scene an
                // entry's rounding exceeds the boxes' widening.
                in = in && entry <= exit_slack(bound);
            }
        }
        // The children that are hit, the first group's nearest on top.
        const uint32_t mask = __ballot_sync(kAll, in);
        const uint32_t ranks = octant_ranks((mask >> (8u * group)) & 0xffu, oct);
        const uint32_t above = (group == 3u ? 0u : (uint32_t)__popc(mask >> (8u * group + 8u))) +
                               (uint32_t)__popc(ranks >> ((c ^ oct) + 1u));
        const uint32_t total = (uint32_t)__popc(mask);
        if (in) {
            if (sp + above < ints) stack[sp + above] = __float_as_int(p.w);
            else overflow = true;
        }
        sp = min(sp + total, ints);
        __syncwarp();
        if (sp == 0u) break;
        taken = min(sp, 4u);
        if (group < taken) link = stack[sp - 1u - group];
        sp -= taken;
        __syncwarp();
    }
    if (!found) return h;
    // The nearest of the lanes' hits, the smaller id on equal t; any-hit: any of them.
    const bool mine = h.id >= 0 && (kAny || h.t == bound);
    const uint32_t id = __reduce_min_sync(kAll, mine ? (uint32_t)h.id : kAll);
    const int from = __ffs(__ballot_sync(kAll, mine && (uint32_t)h.id == id)) - 1;
    return Hit{__shfl_sync(kAll, h.t, from), (int)id, __shfl_sync(kAll, h.slot, from), __shfl_sync(kAll, h.u, from),
               __shfl_sync(kAll, h.v, from)};
}

// A launch's warps over a queue of `count` rays, one ray a warp: the first as numbered, the
// rest from `next` (zero at launch). `body(j)` takes entry j, the whole warp together.
template <class Body>
__device__ __forceinline__ void warp_rays(uint32_t count, uint32_t *next, Body body) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    uint32_t j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    while (j < count) {
        body(j);
        if (count <= warps) break;
        uint32_t more = 0;
        if ((threadIdx.x & 31u) == 0u) more = atomicAdd(next, 1u);
        j = warps + __shfl_sync(0xffffffffu, more, 0);
    }
}

}  // namespace lr
