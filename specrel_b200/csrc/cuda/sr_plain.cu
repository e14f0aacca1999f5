// The plain path: one thread per pixel in 8x8 tiles (the reference's dispatch, gpu.rs:28, 834-844),
// the reference's BVH2 traversal with a 64-entry per-thread stack (bvh4d.rs:445-578), then
// shading, shadow rays and the star term. It is the baseline the fast path is measured against,
// and it reproduces the reference traversal order exactly (ties at equal lambda included).
#include "sr_kernels.h"
#include "sr_ref.cuh"
#include "sr_shade.cuh"

namespace srk {

using namespace srd;

// Bvh4D::is_occluded (bvh4d.rs:523-578).
__device__ bool occluded_ref(const SceneDev& s, float4 o, float4 d, float t_min, float t_max, uint32_t* err) {
    if (s.num_nodes == 0u) return false;
    float4 inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
    if (child_enter(s.nodes, 0, o, inv, t_min, t_max) < 0.0f) return false;
    uint32_t st[SR_STACK_SIZE];
    uint32_t sp = 1;
    st[0] = 0;
    uint32_t visits = 0;
    while (sp > 0) {
        if (++visits > MAX_VISITS) { atomicOr(err, ERR_TRAVERSAL_LIMIT); return false; }
        uint32_t ni = st[--sp];
        uint4 meta = __ldg(reinterpret_cast<const uint4*>(s.nodes + ni) + 2);
        if (meta.y > 0u) {
            for (uint32_t k = meta.x; k < meta.x + meta.y; ++k) {
                GeomHit gh;
                if (intersect_geom(s.geoms + 5u * k, o, d, t_min, t_max, &gh)) return true;
            }
        } else {
            uint32_t li = meta.z, ri = meta.x;
            bool hl = child_enter(s.nodes, li, o, inv, t_min, t_max) >= 0.0f;
            bool hr = child_enter(s.nodes, ri, o, inv, t_min, t_max) >= 0.0f;
            if (hr && sp < SR_STACK_SIZE) st[sp++] = ri;
            if (hl && sp < SR_STACK_SIZE) st[sp++] = li;
        }
    }
    return false;
}

struct RefOccluder {
    const SceneDev* s;
    uint32_t* err;
    __device__ bool operator()(float4 o, float4 d, float t0, float t1) { return occluded_ref(*s, o, d, t0, t1, err); }
};

__global__ void __launch_bounds__(64, 16) k_render_plain(SceneDev s, SrGpuUniforms U, const float4* cam_dev, FrameDev f,
                                                     BBConst bb) {
    uint32_t px = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= U.size[0] || py >= U.size[1]) return;
    const Cam cam = load_cam(U, cam_dev);
    float4 o, d;
    float sx, sy;
    camera_ray(U, cam, px, py, &o, &d, &sx, &sy);
    GeomHit gh;
    int slot = trace_ref(s, o, d, 1e-3f, 180.0f, &gh, f.counters + 1);
    uint32_t shadow_rays = 0;
    F3 color;
    Hit h;
    if (slot >= 0) {
        interpolate(s.attrs + 12u * (uint32_t)slot, o, d, gh, &h);
        RefOccluder occ{&s, f.counters + 1};
        color = shade_hit(s, U, cam, d, h, occ, &shadow_rays);
        if (U.num_haze > 0u) color = apply_haze(color, h.event, U);
    } else {
        color = shade_sky(d);
    }
    if (U.mode == 0u && s.num_stars > 0u)
        color = add(color, stars_brute(s, U, cam, o, d, sx, sy, slot >= 0 ? h.lambda : INFINITY, bb));
    size_t idx = (size_t)py * U.size[0] + px;
    f.hdr[idx] = make_float4(color.x, color.y, color.z, 0.0f);
    if (f.hit_id) f.hit_id[idx] = slot < 0 ? 0xFFFFFFFFu : (s.leaf_to_orig ? __ldg(s.leaf_to_orig + slot) : (uint32_t)slot);
    if (f.lambda) f.lambda[idx] = slot < 0 ? 0.0f : h.lambda;
    if (f.tau) f.tau[idx] = slot < 0 ? 0.0f : h.tau;
    if (shadow_rays) atomicAdd(f.counters, shadow_rays);
}

cudaError_t launch_render_plain(const SceneDev& s, const SrGpuUniforms& u, const float4* cam_dev, const FrameDev& f,
                                const BBConst& bb, cudaStream_t st) {
    dim3 block(8, 8);
    dim3 grid((u.size[0] + 7) / 8, (u.size[1] + 7) / 8);
    k_render_plain<<<grid, block, 0, st>>>(s, u, cam_dev, f, bb);
    return cudaGetLastError();
}

}  // namespace srk
