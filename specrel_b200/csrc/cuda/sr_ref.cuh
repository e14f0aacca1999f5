// The reference's traversal on its own nodes: the plain path's, and the caller rays' that the fast
// path's layouts do not take.
#pragma once
#include "sr_kernels.h"
#include "sr_device.cuh"

namespace srk {

using namespace srd;

// Iteration bound per ray: a tree checked at upload never gets near it; a corrupted one sets
// ERR_TRAVERSAL_LIMIT and the ray ends instead of spinning.
constexpr uint32_t MAX_VISITS = 1u << 22;

struct NodeRef {
    float4 bmin, bmax;
    uint4 meta;  // right_or_first, count, left, pad
};
__device__ __forceinline__ NodeRef load_node(const SrGpuNode* nodes, uint32_t i) {
    const float4* p = reinterpret_cast<const float4*>(nodes + i);
    NodeRef n;
    n.bmin = __ldg(p);
    n.bmax = __ldg(p + 1);
    n.meta = __ldg(reinterpret_cast<const uint4*>(p + 2));
    return n;
}
__device__ __forceinline__ float child_enter(const SrGpuNode* nodes, uint32_t i, float4 o, float4 inv, float t_min,
                                             float t_max) {
    const float4* p = reinterpret_cast<const float4*>(nodes + i);
    return slab_enter(__ldg(p), __ldg(p + 1), o, inv, t_min, t_max);
}

// Bvh4D::trace (bvh4d.rs:445-520). Returns the leaf slot of the closest hit or -1.
static __device__ int trace_ref(const SceneDev& s, float4 o, float4 d, float t_min, float t_max, GeomHit* best,
                         uint32_t* err) {
    if (s.num_nodes == 0u) return -1;
    float4 inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
    float re = child_enter(s.nodes, 0, o, inv, t_min, t_max);
    if (re < 0.0f) return -1;
    uint32_t sn[SR_STACK_SIZE];
    float stt[SR_STACK_SIZE];
    uint32_t sp = 1;
    sn[0] = 0;
    stt[0] = re;
    int slot = -1;
    uint32_t visits = 0;
    while (sp > 0) {
        if (++visits > MAX_VISITS) { atomicOr(err, ERR_TRAVERSAL_LIMIT); break; }
        --sp;
        uint32_t ni = sn[sp];
        if (stt[sp] >= t_max) continue;
        uint4 meta = __ldg(reinterpret_cast<const uint4*>(s.nodes + ni) + 2);
        if (meta.y > 0u) {
            uint32_t first = meta.x, end = meta.x + meta.y;
            for (uint32_t k = first; k < end; ++k) {
                GeomHit gh;
                if (intersect_geom(s.geoms + 5u * k, o, d, t_min, t_max, &gh)) {
                    t_max = gh.lambda;
                    *best = gh;
                    slot = (int)k;
                }
            }
        } else {
            uint32_t li = meta.z, ri = meta.x;
            float tl = child_enter(s.nodes, li, o, inv, t_min, t_max);
            float tr = child_enter(s.nodes, ri, o, inv, t_min, t_max);
            bool hl = tl >= 0.0f, hr = tr >= 0.0f;
            if (hl && hr) {
                if (sp + 2u <= SR_STACK_SIZE) {
                    if (tl <= tr) { sn[sp] = ri; stt[sp] = tr; sn[sp + 1] = li; stt[sp + 1] = tl; }
                    else { sn[sp] = li; stt[sp] = tl; sn[sp + 1] = ri; stt[sp + 1] = tr; }
                    sp += 2u;
                }
            } else if (hl) {
                if (sp < SR_STACK_SIZE) { sn[sp] = li; stt[sp] = tl; ++sp; }
            } else if (hr) {
                if (sp < SR_STACK_SIZE) { sn[sp] = ri; stt[sp] = tr; ++sp; }
            }
        }
    }
    return slot;
}

}  // namespace srk
