// The fast path: the B200 node layout, and a batch of observers rendered as one sequence of
// launches (captured once into a CUDA graph and replayed):
//
//   k_camera_batch   FP64 observers (tetrad from rapidity in double, event rebased to the anchor)
//   k_fan_trace, k_fan_shadow   persistent traversal (the default): each warp walks the 64 rays of an
//                    8x8-pixel tile as one packet (closest hits), then the main light's shadow rays.
//   k_trace_lean     the same work ray by ray (SrTuning.packet = 0, and small launches): warps take 32-ray tiles from a
//                    global counter; each lane traces its pixel's primary ray, then its shadow ray.
//   k_trace_batch    the same work under the other schedules of SrTuning (per-warp chunks of
//                    tiles, partial refills, postponed or cooperative leaf tests).
//   k_shade_batch    one thread per pixel: interpolation and shading, with the main light's
//                    shadow result from the trace kernel (renderer.rs:414-489, 609-653)
//   bloom            the pyramid of every observer, one launch per level
//
// The trace kernel decides "shadow ray needed" with the same code the shading evaluates
// (checkerboard material, light in front in the surface's rest frame), and the shading checks the
// two agree.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstddef>
#include <cstring>

#include "sr_camera.cuh"
#include "sr_fast.h"
#include "sr_ref.cuh"
#include "sr_shade.cuh"
#include "sr_traverse.cuh"
#include "sr_fan.cuh"

namespace srk {

using namespace srd;

// ---------------------------------------------------------------------------------------------
// Layout build.
// ---------------------------------------------------------------------------------------------
// The internal nodes of the top TOP_LEVELS levels, breadth first, from an internal root (node 0):
// topid[node] = its position + 1 (topid zeroed before), level_end[k] = nodes in levels 0..k. One block, a
// node of the level per thread (one thread for all of them took 94 us, 2% of a small rebuild).
__global__ void __launch_bounds__(TOP_NODES / 2 + 1) k_top_levels(const SrGpuNode* nodes, uint32_t* topid, uint32_t* level_end) {
    __shared__ uint32_t q[TOP_NODES], per_warp[(TOP_NODES / 2 + 1) / 32];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    uint32_t start = 0, end = 1;
    if (t == 0) {
        q[0] = 0;
        topid[0] = 1;
        level_end[0] = 1;
    }
    __syncthreads();
    for (uint32_t lv = 1; lv < TOP_LEVELS; ++lv) {
        uint32_t c[2] = {0, 0};
        bool in[2] = {false, false};
        if (start + t < end) {
            const SrGpuNode& nd = nodes[q[start + t]];
            c[0] = nd.left;
            c[1] = nd.right_or_first;
            for (int k = 0; k < 2; ++k) in[k] = nodes[c[k]].count == 0;
        }
        const uint32_t ml = __ballot_sync(0xFFFFFFFFu, in[0]), mr = __ballot_sync(0xFFFFFFFFu, in[1]);
        if (lane == 0) per_warp[warp] = (uint32_t)(__popc(ml) + __popc(mr));
        __syncthreads();
        const uint32_t below = (1u << lane) - 1u;
        uint32_t at = end + (uint32_t)(__popc(ml & below) + __popc(mr & below)), total = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
            if (w < warp) at += per_warp[w];
            total += per_warp[w];
        }
        for (int k = 0; k < 2; ++k)
            if (in[k]) {
                q[at] = c[k];
                topid[c[k]] = ++at;
            }
        start = end;
        end += total;
        if (t == 0) level_end[lv] = end;
        __syncthreads();
    }
}

// Internal nodes below the top levels: they take the positions after the top levels' in the
// reference's depth-first order.
__global__ void k_wide_flags(const SrGpuNode* nodes, uint32_t n, const uint32_t* topid, uint32_t* flags) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flags[i] = nodes[i].count == 0 && topid[i] == 0 ? 1u : 0u;
}

__device__ __forceinline__ uint32_t wide_index(const uint32_t* topid, const uint32_t* wid, uint32_t n_top, uint32_t i) {
    const uint32_t t = topid[i];
    return t ? t - 1u : n_top + wid[i];
}

// One wide node: both children's boxes in each of the `copies` sign-octant copies (near corner,
// far corner; see WideScene; copy 0 is the plain (min, max) layout), the packed child references,
// and the up links of its children (an internal child's in `up`, a leaf child's records' in
// `leafpar`: this node's index, bit 31 set for the right child).
__global__ void k_wide_fill(const SrGpuNode* nodes, uint32_t n, const uint32_t* topid, const uint32_t* wid,
                            uint32_t n_top, float4* boxes, size_t oct_stride, uint32_t copies, uint2* refs, uint32_t* up,
                            uint32_t* leafpar) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || nodes[i].count != 0) return;
    const uint32_t wi = wide_index(topid, wid, n_top, i);
    const SrGpuNode& nd = nodes[i];
    uint32_t c[2] = {nd.left, nd.right_or_first}, ref[2];
    for (int k = 0; k < 2; ++k) {
        const SrGpuNode& ch = nodes[c[k]];
        for (uint32_t oct = 0; oct < copies; ++oct) {
            float nr[4], fr[4];
            for (int a = 0; a < 4; ++a) {
                const bool neg = (oct >> a) & 1u;
                nr[a] = neg ? ch.max[a] : ch.min[a];
                fr[a] = neg ? ch.min[a] : ch.max[a];
            }
            float4* b = boxes + oct * oct_stride + 4ull * wi;
            b[2 * k] = make_float4(nr[0], nr[1], nr[2], nr[3]);
            b[2 * k + 1] = make_float4(fr[0], fr[1], fr[2], fr[3]);
        }
        ref[k] = ch.count > 0 ? pack_leaf(ch.right_or_first, ch.count) : wide_index(topid, wid, n_top, c[k]);
        const uint32_t link = wi | ((uint32_t)k << 31);
        if (ch.count > 0)
            for (uint32_t p = ch.right_or_first; p < ch.right_or_first + ch.count; ++p) leafpar[p] = link;
        else
            up[ref[k]] = link;
    }
    refs[wi] = make_uint2(ref[0], ref[1]);
}

// The packet walk's counters, a line each for those that many warps change.
// FAN_DIRTY: the word of FastCtx::sched that outlives a launch (the list holds entries), the others are cleared.
enum { FAN_NEXT = 0, FAN_HEAD = 32, FAN_TAIL = 64, FAN_FINISHED = 96, FAN_FIRST_DONE = 97, FAN_COUNTERS = 128, FAN_DIRTY = 2 * FAN_COUNTERS + 1 };

static cudaError_t lean_kernel_attrs(int max_smem);
static cudaError_t fan_resident(int threads, int* blocks);
bool lean_stack_supported(uint32_t s);

// Dynamic shared memory of the lean kernel: S + 1 stack words per thread (S of them used).
static size_t lean_stack_bytes(const SrTuning& t) {
    return t.stack_smem ? (size_t)t.block_threads * (t.stack_smem + 1) * sizeof(uint2) : 0;
}

cudaError_t fast_init(FastCtx& c, const cudaDeviceProp& prop) {
    c.num_sms = prop.multiProcessorCount;
    c.max_smem = (int)prop.sharedMemPerBlockOptin;
    const int sizes[4] = {64, 128, 256, 512};
    for (int threads : sizes) {
        int n = 0;
        cudaError_t e = fan_resident(threads, &n);
        if (e != cudaSuccess) return e;
        c.fan_blocks[threads / 128] = (uint32_t)std::max(n, 1);
    }
    return lean_kernel_attrs(c.max_smem);
}

cudaError_t fast_queued(const FastCtx& c, uint32_t queued[2], cudaStream_t st) {
    queued[0] = queued[1] = 0;
    if (!c.sched.p) return cudaSuccess;
    for (int k = 0; k < 2; ++k) {
        cudaError_t e = cudaMemcpyAsync(queued + k, c.sched.as<uint32_t>() + (uint32_t)k * FAN_COUNTERS + FAN_TAIL, 4, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(st);
}

void fast_release(FastCtx& c) {
    for (auto& kv : c.graphs) {
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
        if (kv.second.graph) cudaGraphDestroy(kv.second.graph);
    }
    c.graphs.clear();
}

// Launches whose rays walk alone (k_trace_lean) all the same: few of them through a small scene, where no
// walk is long and the packet's two launches, bounds and queue cost more than they save. Trace time, lone
// against packet: 37k tetrahedra, 320x200: 13 against 30 us, 16 frames of about that size 110 against 231, 8 of
// 640x400 142 against 242, but 1920x1200 88 against 65; 111k, 320x200: 18 against 34, 8 of 640x400 194 against
// 305; 147k, 640x400: 69 against 61, four of them 267 against 211.
constexpr uint64_t LONE_PRIMS = 1u << 17;
static bool lone_rays(uint64_t prims, uint64_t pixels) { return prims <= LONE_PRIMS && prims * pixels < 1ull << 36; }

// The fan layout of a scene that has been waiting for it.
static cudaError_t fan_ready(FastScene& s, const SceneDev& sd, cudaStream_t st) {
    if (!s.fan_pending) return cudaSuccess;
    s.fan_pending = false;
    return fan_build(s, sd.nodes, sd.num_nodes, st);
}

cudaError_t fast_build(FastCtx& c, FastScene& s, const SrGpuNode* nodes, uint32_t n, uint32_t depth, uint32_t num_prims,
                       uint32_t max_leaf, cudaStream_t st) {
    // Captured batch graphs hold the scene's parameters (root box, octant stride, counts) and are
    // keyed by buffer addresses that a rebuilt or re-uploaded scene can reuse: drop them all, once
    // the launches already queued on the stream have finished.
    cudaError_t e0 = cudaStreamSynchronize(st);
    if (e0 != cudaSuccess) return e0;
    fast_release(c);
    s.num_wide = 0;
    s.fan_levels = 0;
    s.fan_pending = false;
    s.depth = depth;
    s.empty = n == 0;
    s.max_leaf = max_leaf;
    s.usable = depth <= FAST_MAX_DEPTH && num_prims < MAX_PACKED_PRIMS && max_leaf <= MAX_LEAF_PRIMS;
    if (n == 0 || !s.usable) return cudaSuccess;
    SrGpuNode root;
    cudaError_t e = cudaMemcpyAsync(&root, nodes, sizeof(root), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    for (int k = 0; k < 4; ++k) { s.root_min[k] = root.min[k]; s.root_max[k] = root.max[k]; }
    if (SR_NODE_IS_NOTHING(&root)) {  // an empty tree (an arena with nothing written)
        s.empty = true;
        return cudaSuccess;
    }
    if (root.count > 0) {
        s.root_ref = pack_leaf(root.right_or_first, root.count);
        return cudaSuccess;
    }
    s.root_ref = 0;  // internal root: wide node 0 (the top levels come first)
    size_t temp = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, temp, (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, st);
    const size_t own = 3 * (size_t)n * 4 + 64 + temp + 512;
    if ((e = s.scratch.ensure(num_prims > LONE_PRIMS ? std::max(own, fan_scratch(n)) : own)) != cudaSuccess) {
        cudaGetLastError();  // without room for the fan layout's, no fan layout
        if ((e = s.scratch.ensure(own)) != cudaSuccess) return e;
    }
    uint32_t* flags = s.scratch.as<uint32_t>();
    uint32_t* wid = flags + n;
    uint32_t* topid = wid + n;
    uint32_t* level_end = topid + n;  // 16 words after topid
    uintptr_t tp = reinterpret_cast<uintptr_t>(level_end + 16);
    void* tmp = reinterpret_cast<void*>((tp + 255) & ~uintptr_t(255));
    if ((e = cudaMemsetAsync(topid, 0, (size_t)n * 4 + 64, st)) != cudaSuccess) return e;
    k_top_levels<<<1, TOP_NODES / 2 + 1, 0, st>>>(nodes, topid, level_end);
    k_wide_flags<<<(n + 255) / 256, 256, 0, st>>>(nodes, n, topid, flags);
    if ((e = cub::DeviceScan::ExclusiveSum(tmp, temp, flags, wid, (int)n, st)) != cudaSuccess) return e;
    uint32_t last[2] = {0, 0};
    cudaMemcpyAsync(&last[0], wid + n - 1, 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&last[1], flags + n - 1, 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(s.top_end, level_end, sizeof(s.top_end), cudaMemcpyDeviceToHost, st);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    const uint32_t n_top = s.top_end[TOP_LEVELS - 1];
    s.num_wide = n_top + last[0] + last[1];
    // Box copies: 16 sign-octant copies, or one (the compact layout) when asked for, or when the
    // 15 extra copies would take more than an eighth of the device or not fit in free memory.
    const uint32_t before = s.copies;
    s.copies = 16;
    if (s.layout == SR_LAYOUT_COMPACT) {
        s.copies = 1;
    } else if (s.layout == SR_LAYOUT_AUTO) {
        size_t free_b = 0, total_b = 0;
        if ((e = cudaMemGetInfo(&free_b, &total_b)) != cudaSuccess) return e;
        const size_t one = (size_t)s.num_wide * 64;
        if (15 * one > total_b / 8 || 16 * one > free_b + s.boxes.bytes) s.copies = 1;
    }
    if (before && before != s.copies) s.boxes.release();  // a layout change does not keep the old size
    if ((e = s.boxes.ensure_grow((size_t)s.num_wide * 64 * s.copies)) != cudaSuccess) return e;
    if ((e = s.refs.ensure_grow((size_t)s.num_wide * 8)) != cudaSuccess) return e;
    if ((e = s.up.ensure_grow((size_t)s.num_wide * 4)) != cudaSuccess) return e;
    if ((e = s.leafpar.ensure_grow((size_t)num_prims * 4 + 4)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(s.up.p, 0xFF, (size_t)s.num_wide * 4, st)) != cudaSuccess) return e;  // the root: ~0
    k_wide_fill<<<(n + 255) / 256, 256, 0, st>>>(nodes, n, topid, wid, n_top, s.boxes.as<float4>(), 4ull * s.num_wide,
                                                 s.copies, s.refs.as<uint2>(), s.up.as<uint32_t>(),
                                                 s.leafpar.as<uint32_t>());
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // Most frames of a small scene walk alone, and it may be changed for every one of them (a dirty-range update of
    // 12,672 tetrahedra took 397 us with this layout and 324 without): it is made when something wants it.
    if (num_prims <= LONE_PRIMS) {
        s.fan_pending = true;
        return cudaStreamSynchronize(st);
    }
    return fan_build(s, nodes, n, st);
}

SrTuning fast_default_tuning(const FastCtx& c) {
    (void)c;
    SrTuning t{};
    t.block_threads = 128;
    t.blocks_per_sm = 8;  // the packet kernels take as many of these as are resident (fan_blocks)
    t.tile_w = 4;
    t.tile_h = 8;
    t.chunk_tiles = 1;
    t.refill_lanes = 32;
    t.leaf_coop = 0;
    t.leaf_batch = 1;
    t.home_pct = 0;
    t.packet = 1;
    return t;
}

bool fast_tuning_valid(const FastCtx& c, const SrTuning& t) {
    bool bt = t.block_threads == 64 || t.block_threads == 128 || t.block_threads == 256 || t.block_threads == 512;
    const size_t stack_bytes = lean_stack_bytes(t);
    return bt && t.blocks_per_sm >= 1 && t.blocks_per_sm <= 16 && t.tile_w >= 1 && t.tile_w * t.tile_h == 32 &&
           t.chunk_tiles >= 1 && t.chunk_tiles <= 64 && t.refill_lanes >= 1 && t.refill_lanes <= 32 &&
           t.leaf_coop <= 1 && t.leaf_batch >= 1 && t.leaf_batch <= 32 && t.home_pct <= 100 &&
           lean_stack_supported(t.stack_smem) && t.top_levels <= TOP_LEVELS &&
           (t.top_levels == 0 || t.stack_smem == 0 || t.stack_smem == 12) &&
           stack_bytes + (t.top_levels ? ((size_t)1 << t.top_levels) * 72u : 0u) <= (size_t)c.max_smem && t.packet <= 1 &&
           (t.packet == 0 || (t.stack_smem == 0 && t.top_levels == 0 && !t.leaf_coop && t.leaf_batch == 1 &&
                              t.refill_lanes == 32 && t.chunk_tiles == 1));
}

// ---------------------------------------------------------------------------------------------
// Batch kernels.
// ---------------------------------------------------------------------------------------------

// The observer holding global index x: the largest o with pre[o] <= x (pre[0] = 0, pre[n] = total).
__device__ __forceinline__ uint32_t find_obs(const uint32_t* pre, uint32_t n, uint32_t x) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(pre + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ Cam cam_of(const float4* cam, uint32_t o) {
    const float4* c = cam + 6ull * o;
    Cam r;
    r.pos = __ldg(c);
    r.e0 = __ldg(c + 1);
    r.e1 = __ldg(c + 2);
    r.e2 = __ldg(c + 3);
    r.e3 = __ldg(c + 4);
    r.frontier = __ldg(c + 5);
    return r;
}

// The observers of a batch; also clears the batch's counters (no launch of their own), and the packet walk's
// queue where a wait that ran out in an earlier batch left entries in it.
__global__ void k_camera_batch(uint32_t n, const SrGpuUniforms* U, const SrCameraF64* cam64, const ObsDev* obs,
                               double a0, double a1, double a2, double a3, float4* cam, uint32_t* counters,
                               uint32_t num_counters, uint32_t* sched, uint32_t num_sched, uint32_t* fan_list,
                               size_t num_fan_list) {
    uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && sched[FAN_DIRTY]) {
        for (size_t k = threadIdx.x; k < num_fan_list; k += blockDim.x) fan_list[k] = 0u;
        __syncthreads();
        if (threadIdx.x == 0) sched[FAN_DIRTY] = 0u;
    }
    for (uint32_t k = o; k < num_counters; k += gridDim.x * blockDim.x) counters[k] = 0u;
    for (uint32_t k = o; k < num_sched; k += gridDim.x * blockDim.x)
        if (k != FAN_DIRTY) sched[k] = 0u;
    if (o >= n) return;
    float4* out = cam + 6ull * o;
    if (obs[o].has_cam64) {
        double anchor[4] = {a0, a1, a2, a3};
        camera_f64(cam64[o], anchor, U[o], out);
    } else {
        const SrGpuUniforms& u = U[o];
        out[0] = v4(u.cam_pos[0], u.cam_pos[1], u.cam_pos[2], u.cam_pos[3]);
        for (int a = 0; a < 4; ++a) out[1 + a] = v4(u.e[a][0], u.e[a][1], u.e[a][2], u.e[a][3]);
        out[5] = v4(u.frontier_origin[0], u.frontier_origin[1], u.frontier_origin[2], u.frontier_origin[3]);
    }
}

__device__ __forceinline__ void add_work(unsigned long long* c, const Work& w) {
    atomicAdd(c + 0, (unsigned long long)w.nodes);
    atomicAdd(c + 1, (unsigned long long)w.leaves);
    atomicAdd(c + 2, (unsigned long long)w.tets);
}

struct TraceBatchArgs {
    WideScene ws;
    const float4* attrs;
    const float4* mats;
    const SrGpuUniforms* U;
    const float4* cam;
    const ObsDev* obs;
    const uint32_t* tile_pre;
    uint32_t n, total_rays, tile_w, tile_h;
    uint32_t chunk_rays;    // rays a warp takes from the global counter at a time (a multiple of 32)
    uint32_t refill_lanes;  // idle lanes that make the warp fetch new rays
    uint32_t leaf_batch;    // lanes on a leaf before the warp tests leaves
    uint32_t top_n;         // lean kernel: wide nodes staged in shared memory (the top levels)
    // Lean kernel tile order: SM band b holds tiles [b * band_tiles, (b + 1) * band_tiles) and is
    // taken through sched[b]; the shared pool, tiles [num_bands * band_tiles, total), through
    // sched[num_bands].
    uint32_t num_bands, band_tiles;
    uint32_t* sched;
    float4* hits;
    uint32_t* slots;
    uint8_t* shadow;  // 0: no main-light shadow ray, 1: cast and clear, 2: cast and occluded
    uint32_t* counter;
    uint32_t* err;
    unsigned long long* work;
};

// Ray index r -> pixel: rays run tile by tile (32 consecutive rays = one tile_w x tile_h tile).
__device__ __forceinline__ bool ray_pixel(const TraceBatchArgs& a, uint32_t r, uint32_t* obs, uint32_t* px, uint32_t* py,
                                          uint32_t* p) {
    uint32_t t = r >> 5, l = r & 31u;
    uint32_t o = find_obs(a.tile_pre, a.n, t);
    const ObsDev& od = a.obs[o];
    uint32_t lt = t - __ldg(a.tile_pre + o);
    uint32_t x = (lt % od.tiles_x) * a.tile_w + l % a.tile_w;
    uint32_t y = (lt / od.tiles_x) * a.tile_h + l / a.tile_w;
    *obs = o;
    *px = x;
    *py = y;
    *p = od.pix_base + y * od.width + x;
    return x < od.width && y < od.height;
}

// Shared memory of one warp for the cooperative leaf tests: the rays of the lanes at a leaf, and
// per lane the best (lambda bits << 32 | tetrahedron index in the leaf) key with its barycentrics.
constexpr uint32_t COOP_SMEM_PER_WARP = 32u * 4u * sizeof(float4) + 32u * sizeof(unsigned long long);

// Persistent traversal (see the top of the file). Each pass of the loop, with the warp converged:
//   refill     when at least `refill_lanes` lanes are idle, they take the next rays of the warp's
//              chunk (chunk_rays consecutive rays, a block of neighbouring tiles);
//   internal   every lane standing on an internal node takes one step (descend, push, or pop);
//   leaves     lanes standing on a leaf wait until `leaf_batch` lanes do (or no lane is on an
//              internal node); then the leaves are tested. With COOP the warp tests all its lanes'
//              tetrahedra together, 32 at a time, and each lane keeps the smallest lambda, ties going
//              to the first tetrahedron of the leaf, as in the sequential loop (whose test
//              `lambda >= t_max` rejects an equal lambda).
// Each ray visits exactly the nodes of the reference's traversal, in its order.
template <bool COUNT, bool COOP>
__global__ void __launch_bounds__(512) k_trace_batch(TraceBatchArgs a) {
    extern __shared__ float4 coop_smem[];
    const uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lanes_below = (1u << lane) - 1u;
    float4* s_o = coop_smem + warp * 128u;
    float4* s_d = s_o + 32;
    float4* s_t = s_d + 32;
    float4* s_h = s_t + 32;
    unsigned long long* s_key = reinterpret_cast<unsigned long long*>(coop_smem + (blockDim.x >> 5) * 128u) + warp * 32u;

    Work wp{0, 0, 0}, wsh{0, 0, 0};
    bool has = false, occluded = false;
    uint32_t obs = 0, pix = 0, phase = 0, cur = 0, visits = 0;
    int sp = 0, slot = -1;
    float4 o = v4(0, 0, 0, 0), d = o, inv = o;
    float t_min = 0.0f, t_max = 0.0f;
    GeomHit best{0.0f, 0.0f, 0.0f, 0.0f};
    uint32_t st_ref[FAST_STACK];
    float st_t[FAST_STACK];
    uint32_t c_next = 0, c_end = 0;  // the warp's chunk (uniform across the warp)
    bool exhausted = false;          // uniform

    // Next node from the stack; primary rays skip entries entered at or beyond the closest hit.
    auto pop = [&]() -> bool {
        while (sp > 0) {
            --sp;
            if (phase != 0 || st_t[sp] < t_max) {
                cur = st_ref[sp];
                return true;
            }
        }
        return false;
    };
    // The current query is over: store its result, and start the shadow query when the main light
    // needs one.
    auto end_phase = [&]() {
        if (phase != 0) {
            a.shadow[pix] = occluded ? 2 : 1;
            has = false;
            return;
        }
        a.hits[pix] = make_float4(best.lambda, best.u, best.v, best.w);
        a.slots[pix] = slot < 0 ? 0xFFFFFFFFu : (uint32_t)slot;
        uint8_t sh_state = 0;
        has = false;
        const SrGpuUniforms& U = a.U[obs];
        if (slot >= 0 && U.mode == 0u && U.shadow_mode != 0u && U.num_flashes == 0u) {
            // compute_illumination's shadow-ray condition (renderer.rs:617-633).
            const float4* at = a.attrs + 12u * (uint32_t)slot;
            uint32_t mat = __float_as_uint(__ldg(at + 10).z);
            if (__float_as_uint(__ldg(a.mats + 3u * mat + 2u).y) == 0u) {
                float4 ev = add4(o, mul4(d, best.lambda));
                const Cam cam = cam_of(a.cam, obs);
                float4 tl;
                float dist;
                light_ray(U, cam, ev, &tl, &dist);
                if (fmaxf(rest_frame_cos(tl, __ldg(at + 8), __ldg(at + 9)), 0.0f) > 0.0f) {
                    // Bvh4D::is_occluded(hit.event, to_light, 2e-3, dist - 2e-3) (renderer.rs:636-641).
                    sh_state = 1;
                    o = ev;
                    d = tl;
                    inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
                    t_min = 2e-3f;
                    t_max = dist - 2e-3f;
                    phase = 1;
                    occluded = false;
                    visits = 0;
                    sp = 0;
                    if (slab_enter(a.ws.root_min, a.ws.root_max, o, inv, t_min, t_max) >= 0.0f) {
                        cur = a.ws.root_ref;
                        has = true;
                    }
                }
            }
        }
        if (!has) a.shadow[pix] = sh_state;
    };

    // One internal node of the lane's query: descend into the nearer child box, push the farther,
    // or pop; ends the query when the stack runs dry.
    auto node_step = [&]() {
        if (++visits > MAX_VISITS_FAST) {
            atomicOr(a.err, ERR_TRAVERSAL_LIMIT);
            sp = 0;
            end_phase();
            return;
        }
        if (COUNT) ++(phase ? wsh : wp).nodes;
        const float4* bx = a.ws.boxes + 4ull * cur;
        float4 lmin = __ldg(bx), lmax = __ldg(bx + 1), rmin = __ldg(bx + 2), rmax = __ldg(bx + 3);
        uint2 rf = __ldg(a.ws.refs + cur);
        float tl = slab_enter(lmin, lmax, o, inv, t_min, t_max);
        float tr = slab_enter(rmin, rmax, o, inv, t_min, t_max);
        bool hl = tl >= 0.0f, hr = tr >= 0.0f;
        // Primary rays cull boxes entered at or beyond the closest hit (bvh4d.rs:461); the
        // any-hit query has no such cull (bvh4d.rs:541-575) and visits left before right.
        const bool any = phase != 0;
        if (hl && hr) {
            bool left_near = any || tl <= tr;
            float tn = left_near ? tl : tr;
            if (any || tn < t_max) {
                if (sp < FAST_STACK) {
                    st_ref[sp] = left_near ? rf.y : rf.x;
                    st_t[sp] = left_near ? tr : tl;
                    ++sp;
                } else {
                    atomicOr(a.err, ERR_BAD_INDEX);
                }
                cur = left_near ? rf.x : rf.y;
                return;
            }
        } else if (hl && (any || tl < t_max)) {
            cur = rf.x;
            return;
        } else if (hr && (any || tr < t_max)) {
            cur = rf.y;
            return;
        }
        if (!pop()) end_phase();
    };

    for (;;) {
        // Refill.
        unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && idle != 0u && (idle == FULL || (uint32_t)__popc(idle) >= a.refill_lanes)) {
            while (idle != 0u) {
                if (c_next == c_end) {
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(a.counter, a.chunk_rays);
                    base = __shfl_sync(FULL, base, 0);
                    if (base >= a.total_rays) {
                        exhausted = true;
                        break;
                    }
                    c_next = base;
                    c_end = min(base + a.chunk_rays, a.total_rays);
                }
                uint32_t take = min(c_end - c_next, (uint32_t)__popc(idle));
                bool mine = ((idle >> lane) & 1u) && (uint32_t)__popc(idle & lanes_below) < take;
                if (mine) {
                    uint32_t r = c_next + (uint32_t)__popc(idle & lanes_below);
                    uint32_t px, py;
                    if (ray_pixel(a, r, &obs, &px, &py, &pix)) {
                        const Cam cam = cam_of(a.cam, obs);
                        float sx, sy;
                        camera_ray(a.U[obs], cam, px, py, &o, &d, &sx, &sy);
                        inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
                        t_min = 1e-3f;
                        t_max = 180.0f;
                        slot = -1;
                        phase = 0;
                        visits = 0;
                        sp = 0;
                        float re = a.ws.empty ? -1.0f : slab_enter(a.ws.root_min, a.ws.root_max, o, inv, t_min, t_max);
                        if (re >= 0.0f && re < t_max) {
                            cur = a.ws.root_ref;
                            has = true;
                        } else {  // the ray misses the scene's box (bvh4d.rs:451)
                            a.hits[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            a.slots[pix] = 0xFFFFFFFFu;
                            a.shadow[pix] = 0;
                        }
                    }
                }
                idle &= ~__ballot_sync(FULL, mine);
                c_next += take;
            }
        }

        // One internal node for every lane that stands on one.
        if (has && !(cur & REF_LEAF)) node_step();

        // Leaves: postponed until `leaf_batch` lanes stand on one, or no lane is on an internal node.
        const bool at_leaf = has && (cur & REF_LEAF);
        const unsigned lm = __ballot_sync(FULL, at_leaf);
        const unsigned nm = __ballot_sync(FULL, has && !(cur & REF_LEAF));
        if (lm == 0u) {
            if (nm == 0u && exhausted) break;
            continue;
        }
        if (nm != 0u && (uint32_t)__popc(lm) < a.leaf_batch) continue;

        if (!COOP) {
            if (at_leaf) {
                if (++visits > MAX_VISITS_FAST) {
                    atomicOr(a.err, ERR_TRAVERSAL_LIMIT);
                    sp = 0;
                } else {
                    uint32_t first = cur & REF_FIRST_MASK, cnt = (cur >> REF_COUNT_SHIFT) & 63u;
                    if (COUNT) ++(phase ? wsh : wp).leaves;
                    for (uint32_t k = first; k < first + cnt; ++k) {
                        if (COUNT) ++(phase ? wsh : wp).tets;
                        GeomHit gh;
                        if (intersect_geom(a.ws.geoms + 5u * k, o, d, t_min, t_max, &gh)) {
                            if (phase == 0) {
                                t_max = gh.lambda;
                                best = gh;
                                slot = (int)k;
                            } else {
                                occluded = true;
                                sp = 0;
                                break;
                            }
                        }
                    }
                }
                if (!pop()) end_phase();
            }
            continue;
        }
        uint32_t first = 0, cnt = 0;
        if (at_leaf) {
            if (++visits > MAX_VISITS_FAST) {
                atomicOr(a.err, ERR_TRAVERSAL_LIMIT);
                sp = 0;
            } else {
                first = cur & REF_FIRST_MASK;
                cnt = (cur >> REF_COUNT_SHIFT) & 63u;
                if (COUNT) {
                    ++(phase ? wsh : wp).leaves;
                    (phase ? wsh : wp).tets += cnt;
                }
            }
            s_o[lane] = o;
            s_d[lane] = d;
            s_t[lane] = make_float4(t_min, t_max, 0.0f, 0.0f);
            s_key[lane] = ~0ull;
        }
        uint32_t incl = cnt;
#pragma unroll
        for (uint32_t s = 1; s < 32; s <<= 1) {
            uint32_t v = __shfl_up_sync(FULL, incl, s);
            if (lane >= s) incl += v;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        const uint32_t excl = incl - cnt;
        __syncwarp();
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t j = base + lane;
            // The owner: the first lane whose inclusive count exceeds j.
            uint32_t L = 0;
#pragma unroll
            for (uint32_t s = 16; s >= 1; s >>= 1) {
                uint32_t v = __shfl_sync(FULL, incl, L + s - 1);
                if (v <= j) L += s;
            }
            L = min(L, 31u);
            const uint32_t l_excl = __shfl_sync(FULL, excl, L);
            const uint32_t l_first = __shfl_sync(FULL, first, L);
            bool hit = false;
            unsigned long long key = 0;
            GeomHit gh;
            if (j < total) {
                const uint32_t i = j - l_excl;
                const float4 tt = s_t[L];
                if (intersect_geom(a.ws.geoms + 5u * (l_first + i), s_o[L], s_d[L], tt.x, tt.y, &gh)) {
                    key = ((unsigned long long)__float_as_uint(gh.lambda) << 32) | i;
                    atomicMin(s_key + L, key);
                    hit = true;
                }
            }
            __syncwarp();
            if (hit && s_key[L] == key) s_h[L] = make_float4(gh.u, gh.v, gh.w, 0.0f);
            __syncwarp();
        }
        if (at_leaf) {
            const unsigned long long k = s_key[lane];
            if (k != ~0ull) {
                if (phase == 0) {
                    const float4 h = s_h[lane];
                    best.lambda = __uint_as_float((uint32_t)(k >> 32));
                    best.u = h.x;
                    best.v = h.y;
                    best.w = h.z;
                    t_max = best.lambda;
                    slot = (int)(first + (uint32_t)(k & 0xFFFFFFFFull));
                } else {
                    occluded = true;
                    sp = 0;
                }
            }
            if (!pop()) end_phase();
        }
        __syncwarp();
    }
    if (COUNT) {
        add_work(a.work, wp);
        add_work(a.work + 3, wsh);
    }
}

// The main light's shadow query of a hit (compute_illumination's condition, renderer.rs:617-633).
struct ShadowQuery {
    float4 no, d, inv;
    float t_min, t_max;
    bool enters;  // the query's ray enters the scene's box
};
__device__ __forceinline__ bool casts_shadows(const SrGpuUniforms& U) {
    return U.mode == 0u && U.shadow_mode != 0u && U.num_flashes == 0u;
}
// Whether the hit at `lambda` of the ray (-no, d) of observer `obs` casts one; fills `q`.
__device__ __forceinline__ bool shadow_query(const TraceBatchArgs& a, uint32_t obs, uint32_t slot, float4 no, float4 d,
                                             float lambda, ShadowQuery* q) {
    const SrGpuUniforms& U = a.U[obs];
    if (!casts_shadows(U)) return false;
    const float4* at = a.attrs + 12u * slot;
    const uint32_t mat = __float_as_uint(__ldg(at + 10).z);
    if (__float_as_uint(__ldg(a.mats + 3u * mat + 2u).y) != 0u) return false;
    const float4 ev = sub4(mul4(d, lambda), no);  // o + d * lambda
    float4 tl;
    float dist;
    // The camera is read again here rather than kept in registers across the traversal.
    light_ray(U, cam_of(a.cam, obs), ev, &tl, &dist);
    if (!(fmaxf(rest_frame_cos(tl, __ldg(at + 8), __ldg(at + 9)), 0.0f) > 0.0f)) return false;
    // Bvh4D::is_occluded(hit.event, to_light, 2e-3, dist - 2e-3) (renderer.rs:636-641).
    q->no = neg4(ev);
    q->d = tl;
    q->inv = v4(safe_inv(tl.x), safe_inv(tl.y), safe_inv(tl.z), safe_inv(tl.w));
    q->t_min = 2e-3f;
    q->t_max = dist - 2e-3f;
    float en, ex;
    slab_interval(a.ws.root_min, a.ws.root_max, q->no, q->inv, q->t_min, q->t_max, &en, &ex);
    q->enters = ex >= en;
    return true;
}

// The default schedule (whole-tile refills, one tile per fetch, leaves tested per lane) in its lean
// form: a warp takes the next 32-ray tile when all its lanes are done, and each lane runs its
// primary query and then, when the main light needs it, its shadow query to the end, with no
// warp-wide bookkeeping per step.
__device__ __forceinline__ uint32_t sm_id() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
    return r;
}

// The next tile of a warp (called by one lane): its SM's band first, then the shared pool in
// frame order, then what is left in other SMs' bands. Returns ~0u when every tile is taken.
// `stage` and `steal` persist across calls (0: band, 1: pool, 2: stealing from band steal).
__device__ __forceinline__ uint32_t next_tile(const TraceBatchArgs& a, uint32_t home, uint32_t& stage, uint32_t& steal) {
    const uint32_t total_tiles = a.total_rays >> 5;
    if (stage == 0) {
        uint32_t v = atomicAdd(a.sched + home, 1u);
        if (v < a.band_tiles) return home * a.band_tiles + v;
        stage = 1;
    }
    const uint32_t pool_base = a.num_bands * a.band_tiles;
    if (stage == 1) {
        uint32_t v = atomicAdd(a.sched + a.num_bands, 1u);
        if (v < total_tiles - pool_base) return pool_base + v;
        stage = 2;
    }
    while (steal < a.num_bands) {
        const uint32_t b = (home + steal) % a.num_bands;
        if (*(volatile uint32_t*)(a.sched + b) < a.band_tiles) {
            uint32_t v = atomicAdd(a.sched + b, 1u);
            if (v < a.band_tiles) return b * a.band_tiles + v;
        }
        ++steal;
    }
    return ~0u;
}

// SS > 0: the first SS entries of each thread's traversal stack live in dynamic shared memory
// (SplitStack), the rest in local memory; SS == 0: all in local memory (LocalStack). OCT: the
// scene has the 16 sign-octant box copies; otherwise the compact layout (one copy). TOP: the first
// a.top_n wide nodes (the tree's top levels) are staged in shared memory after the stacks, their
// (min, max) boxes then their references.
template <bool COUNT, int SS, bool OCT, bool TOP>
__global__ void __launch_bounds__(512) k_trace_lean(const __grid_constant__ TraceBatchArgs a) {
    const uint32_t lane = threadIdx.x & 31u;
    Work wp{0, 0, 0}, wsh{0, 0, 0};
    uint2 lm[FAST_STACK];
    extern __shared__ uint2 sm_stack[];
    using Stack = typename std::conditional<(SS > 0), SplitStack<SS>, LocalStack>::type;
    Stack st;
    if constexpr (SS > 0) st = SplitStack<SS>{sm_stack + threadIdx.x * SplitStack<SS>::ROW, lm};
    else st = LocalStack{lm};
    TopStage top{nullptr, nullptr, 0u};
    if constexpr (TOP) {
        float4* tb = reinterpret_cast<float4*>(sm_stack + (SS > 0 ? blockDim.x * (uint32_t)SplitStack<SS>::ROW : 0u));
        uint2* tr = reinterpret_cast<uint2*>(tb + 4u * a.top_n);
        for (uint32_t i = threadIdx.x; i < 4u * a.top_n; i += blockDim.x) tb[i] = __ldg(a.ws.boxes + i);  // copy 0: (min, max)
        for (uint32_t i = threadIdx.x; i < a.top_n; i += blockDim.x) tr[i] = __ldg(a.ws.refs + i);
        __syncthreads();
        top = TopStage{tb, tr, a.top_n};
    }
    const uint32_t home = a.num_bands ? sm_id() % a.num_bands : 0u;
    uint32_t stage = a.num_bands ? 0u : 1u, steal = 0;
    for (;;) {
        uint32_t tile = 0;
        if (lane == 0) tile = next_tile(a, home, stage, steal);
        tile = __shfl_sync(0xFFFFFFFFu, tile, 0);
        if (tile == ~0u) break;
        const uint32_t base = tile << 5;
        uint32_t obs = 0, px = 0, py = 0, pix = 0;
        const bool valid = ray_pixel(a, base + lane, &obs, &px, &py, &pix);
        if (!valid) continue;
        float4 o, d;
        float sx, sy;
        camera_ray(a.U[obs], cam_of(a.cam, obs), px, py, &o, &d, &sx, &sy);
        const float4 no = neg4(o);  // the traversal and the hit event use the negated origin only
        const float4 inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
        float t_max = 180.0f;
        GeomHit best{0.0f, 0.0f, 0.0f, 0.0f};
        int slot = -1;
        if (!a.ws.empty) {
            float en, ex;
            slab_interval(a.ws.root_min, a.ws.root_max, no, inv, 1e-3f, t_max, &en, &ex);
            if (ex >= en && en < t_max)  // else the ray misses the scene's box (bvh4d.rs:451)
                slot = closest_lean<COUNT, OCT, TOP>(a.ws, a.ws.root_ref, no, d, inv, 1e-3f, t_max, best, st, a.err, wp, top);
        }
        a.hits[pix] = make_float4(best.lambda, best.u, best.v, best.w);
        a.slots[pix] = slot < 0 ? 0xFFFFFFFFu : (uint32_t)slot;
        uint8_t sh = 0;
        ShadowQuery q;
        if (slot >= 0 && shadow_query(a, obs, (uint32_t)slot, no, d, best.lambda, &q)) {
            sh = 1;
            if (q.enters && any_lean<COUNT, OCT, TOP>(a.ws, a.ws.root_ref, q.no, q.d, q.inv, q.t_min, q.t_max, st, a.err, wsh, top))
                sh = 2;
        }
        a.shadow[pix] = sh;
    }
    if (COUNT) {
        add_work(a.work, wp);
        add_work(a.work + 3, wsh);
    }
}

// ---------------------------------------------------------------------------------------------
// The packet form (SrTuning.packet): the walks of sr_fan.cuh in two persistent launches.
//
//   k_fan_trace    Every warp takes tiles of 64 pixels (two rays per lane; 8 pixels in small frames) until there are none. A walk
//                  of more than FAN_BUDGET steps is given up: its tile goes into a queue as eight
//                  groups of 8 pixels, which the warps walk from the hits found, as they run out of tiles.
//                  Pixels whose hits cast a shadow ray are listed, 32 (or a group) at a time.
//   k_fan_shadow   The main light's shadow queries of the listed pixels. What a walk of more than
//                  FAN_ANY_BUDGET steps leaves open goes into the queue, each query walked by a warp
//                  alone.
//
// Rays that spread (small frames, and the views away from a fast observer's motion, which aberration
// widens up to e^2|rapidity| times) make an interval that holds far more than they meet: one tile of a
// 471x163 frame took 1.1 ms alone. Splitting such tiles in launches of their own left each launch
// waiting for its last warps; from a queue the parts of a slow tile start while other tiles still run. One
// launch for both kinds of rays was slower: its code misses the instruction cache (1.4 of 11 stall
// cycles per instruction against 0.2 of 7).
//
// The queue: an entry is written at list[tail++]; a warp takes the ticket head++, and the entry of that
// number is its next task, or there is none once all first tasks and every entry are finished. Only the warps
// of the first blocks (`helpers`) do so while the queue is empty; the others leave then (a warp that queued
// something comes back for it itself). A warp waits only for work that running warps are doing, which never
// waits for it, and for at most q.polls polls. Where a wait runs out all the same, its ticket is given up and the
// entry written later at its place is taken by nobody: the frame is incomplete (ERR_QUEUE_WAIT, and `lost`, which
// outlives the frame's own flags until a call reports it) and the list is not zero at the end. `dirty` says so to
// the launches behind: the shadow launch leaves, the next batch's camera launch clears the list.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t FAN_BUDGET = 400, FAN_ANY_BUDGET = 160;
// Tests without a hit after which a tile's walk is given up. A walk given up costs more in parts (from
// the root again, fewer rays per test), so a launch with much to do per warp gives up late (the 8-frame
// launch of the 7.9M-tet workload: 2.10 ms of closest hits at 200 to 256, 2.40 at 128, 2.87 at 64), and a
// small one, which its slowest tiles hold up, early (471x163 pixels seen at rapidity 1.7: 0.40 ms at 256,
// 0.27 at 128).
constexpr uint32_t FAN_WASTE = 256, FAN_WASTE_SMALL = 128, FAN_SMALL_TILES = 48u << 10;
constexpr uint32_t FAN_UNLIMITED = 1u << 22;
constexpr uint32_t FAN_GROUP_LOG = 3, FAN_PAIR_LOG = 1;  // log2 of a group's and a pair's pixels
// Blocks that stay for the queue: one for every 4 SMs. Waiting warps hold the room that another stream's launch
// could use and their polls slow the working ones. With three engines' frames in turn, all blocks waiting against a
// quarter of the SMs' number against none: 1280x800 of the 7.9M-tet workload 738, 410 and 452 us a frame, five
// frames of 471x163 to 715x513 656, 338 and 358, 8 of 1280x800 3.02, 2.79 and 2.78 ms; one engine alone, trace
// time: 294, 259 and 251 us (1280x800, 16 bodies), 580, 608 and 623 (the five).
constexpr uint32_t FAN_HELPERS_PER = 4;
// A task: tile * 64 + part + 1 (0: no entry yet). Parts of a tile in k_fan_trace's queue: its 8 groups of 8
// pixels, then its 32 pairs; in the list of shadow rays: its two halves of 32 pixels, then its 8 groups, then
// its 32 pairs; in k_fan_shadow's queue: its 64 pixels.
constexpr uint32_t FAN_PARTS_LOG = 6, FAN_GROUPS = 8, FAN_HALVES = 2;
constexpr uint32_t FAN_MAX_TILES = 1u << (31u - FAN_PARTS_LOG);
constexpr uint32_t FAN_SHADOWS_PER_TILE = 32, FAN_QUEUED_PER_TILE = 64;

struct FanTasks {
    uint32_t* count;    // FAN_COUNTERS words of this launch, zero at the start
    uint32_t* list;     // the queue, zero at the start and again at the end
    uint32_t* dirty;    // entries were left in the list
    uint32_t* lost;     // a frame is incomplete (pinned host memory)
    uint32_t polls;     // a wait's limit
    uint32_t* shadows;  // the pixels that cast shadow rays, as tasks
    uint32_t* num_shadows;
    uint32_t waste;     // FAN_WASTE or FAN_WASTE_SMALL
    uint32_t helpers;   // the first blocks, whose warps wait for the queue's entries
};

// log2 of a tile's pixels: 64, or 8 where that leaves less than a tile per warp. Three engines' frames in turn, in
// tiles of 8, 16 and 64: 16 accelerated bodies at 120x78 102, 138 and 151 us a frame, at 320x200 130, 152 and
// 154, at 640x400 205, 181 and 163, at 1100x700 459, 285 and 185; 147k tetrahedra at 451x205 76, 82 and 93.
static uint32_t fan_tile_log(uint64_t pixels) { return pixels < (128u << 10) ? 3u : 6u; }

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The observer of a tile and the tile's corner pixel.
struct FanTile {
    uint32_t obs, x, y;
};
__device__ __forceinline__ FanTile fan_tile(const TraceBatchArgs& a, uint32_t tile) {
    FanTile t;
    t.obs = find_obs(a.tile_pre, a.n, tile);
    const uint32_t across = a.obs[t.obs].tiles_x, lt = tile - __ldg(a.tile_pre + t.obs), row = lt / across;
    t.x = (lt - row * across) * a.tile_w;
    t.y = row * a.tile_h;
    return t;
}
__device__ __forceinline__ uint32_t warp_next(uint32_t* counter) {
    uint32_t t = 0;
    if ((threadIdx.x & 31u) == 0) t = atomicAdd(counter, 1u);
    return __shfl_sync(FULL_WARP, t, 0);
}
__device__ __forceinline__ void store_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Puts a task (tile, part) for each lane that has one at the end of `list`, after all lanes' writes: the warp's
// barrier orders them before each lane's releasing store.
__device__ __forceinline__ void fan_list(uint32_t* list, uint32_t* tail, uint32_t tile, uint32_t part, bool has) {
    const uint32_t lane = threadIdx.x & 31u, which = __ballot_sync(FULL_WARP, has);
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(tail, (uint32_t)__popc(which));
    at = __shfl_sync(FULL_WARP, at, 0) + (uint32_t)__popc(which & ((1u << lane) - 1u));
    __syncwarp();
    if (has) store_release(list + at, (tile << FAN_PARTS_LOG) + part + 1u);
}
__device__ __forceinline__ void fan_push(const FanTasks& q, uint32_t tile, uint32_t part, bool has) {
    fan_list(q.list, q.count + FAN_TAIL, tile, part, has);
}
// A warp's first tasks are done: `mine` of them.
__device__ __forceinline__ void fan_first_done(const FanTasks& q, uint32_t mine) {
    __syncwarp();
    if ((threadIdx.x & 31u) == 0 && mine) {
        __threadfence();
        atomicAdd(q.count + FAN_FIRST_DONE, mine);
    }
}
__device__ __forceinline__ void fan_finished(const FanTasks& q) {
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) {
        __threadfence();
        atomicAdd(q.count + FAN_FINISHED, 1u);
    }
}
// The next task of the queue, or 0 when all work is done (`first`: the number of first tasks), of a launch of
// `tiles` tiles.
__device__ __forceinline__ uint32_t fan_take(const FanTasks& q, uint32_t first, uint32_t tiles, uint32_t* err) {
    uint32_t entry = 0;
    if ((threadIdx.x & 31u) == 0 &&
        (blockIdx.x < q.helpers || (int)(load_acquire(q.count + FAN_TAIL) - load_acquire(q.count + FAN_HEAD)) > 0)) {
        const uint32_t ticket = atomicAdd(q.count + FAN_HEAD, 1u);
        for (uint32_t polls = 0;; ++polls) {
            if (load_acquire(q.count + FAN_TAIL) > ticket) {
                entry = load_acquire(q.list + ticket);
                if (entry) {
                    q.list[ticket] = 0u;
                    break;
                }
            } else {
                // Finished entries are counted after what they queued: with every first task done and as
                // many entries finished as queued, nothing more will be.
                if (load_acquire(q.count + FAN_FIRST_DONE) == first) {
                    const uint32_t finished = load_acquire(q.count + FAN_FINISHED);
                    const uint32_t tail = load_acquire(q.count + FAN_TAIL);
                    if (finished == tail && tail <= ticket) break;
                }
                __nanosleep(200);
            }
            if (polls > q.polls) {
                atomicOr(err, ERR_QUEUE_WAIT);
                *(volatile uint32_t*)q.dirty = 1u;
                *(volatile uint32_t*)q.lost = 1u;
                break;
            }
        }
        if (entry && (entry - 1u) >> FAN_PARTS_LOG >= tiles) {  // not this launch's: never followed
            atomicOr(err, ERR_BAD_INDEX);
            entry = 0;
        }
    }
    // Lane 0 acquired the entry; the barrier orders the other lanes' reads of what its task left behind it.
    __syncwarp();
    return __shfl_sync(FULL_WARP, entry, 0);
}

// The ray of a pixel, and what is written of its hit: out of line, one copy for the rays of a lane (two in
// line make the tile's straight code too long for the instruction cache).
struct FanRay {
    float4 d, inv;
};
static __device__ __noinline__ FanRay fan_ray(const SrGpuUniforms* U, const float4* cam, uint32_t obs, uint32_t px, uint32_t py) {
    float4 o;
    FanRay r;
    float sx, sy;
    camera_ray(U[obs], cam_of(cam, obs), px, py, &o, &r.d, &sx, &sy);
    r.inv = v4(safe_inv(r.d.x), safe_inv(r.d.y), safe_inv(r.d.z), safe_inv(r.d.w));
    return r;
}
// The negated origin of an observer's rays: camera_ray's, the same for every pixel.
__device__ __forceinline__ float4 fan_origin(const SrGpuUniforms& U, const Cam& c) {
    float4 o = c.pos;
    if (U.slice_mode == 2u) o = sub4(o, mul4(c.e0, U.frontier_view_offset));
    if (U.slice_mode == 3u) o = add4(o, mul4(c.e0, U.prophecy_delta));
    return neg4(o);
}
// Returns whether the hit casts a shadow ray.
static __device__ __noinline__ bool fan_write(const TraceBatchArgs& a, uint32_t obs, uint32_t pix, uint32_t slot, float lambda,
                                              float4 d, float4 no) {
    // The barycentrics of the hit, as the test computed them (kept there, they would take registers
    // through the walk).
    const float4* g = a.ws.geoms + 5u * slot;
    const float4 v0 = __ldg(g);
    const float4 ev = sub4(mul4(d, lambda), no);
    const float2 q01 = add2(f2(ev.x, ev.y), f2(-v0.x, -v0.y)), q23 = add2(f2(ev.z, ev.w), f2(-v0.z, -v0.w));
    const float4 q = make_float4(q01.x, q01.y, q23.x, q23.y);
    a.hits[pix] = make_float4(lambda, edot_p(__ldg(g + 2), q), edot_p(__ldg(g + 3), q), edot_p(__ldg(g + 4), q));
    a.shadow[pix] = 0;
    ShadowQuery sq;
    return shadow_query(a, obs, slot, no, d, lambda, &sq);
}

// The closest hits of a rectangle of 2^(w_log + h_log) pixels of observer `obs` with corner (x0, y0);
// `resume`: the hits in memory are kept as bounds. Returns false when the walk was given up; `casts`: bit
// r set when one of the first (0) or second half (1) of the pixels has a hit that casts a shadow ray.
template <bool OCT>
__device__ __forceinline__ bool fan_pixels(const TraceBatchArgs& a, uint32_t obs, uint32_t x0, uint32_t y0, uint32_t w_log,
                                           uint32_t h_log, bool resume, uint32_t budget, uint32_t waste, FanQueue& f, uint2* st,
                                           uint32_t* casts) {
    const uint32_t lane = threadIdx.x & 31u, half = 1u << (w_log + h_log - 1u);
    const ObsDev& od = a.obs[obs];
    float4 d[FAN_RAYS];
    float t_max[FAN_RAYS];
    int slot[FAN_RAYS];
#pragma unroll
    for (int r = 0; r < FAN_RAYS; ++r) {
        d[r] = v4(0.0f, 0.0f, 0.0f, 0.0f);
        t_max[r] = 0.0f;
        slot[r] = -1;
    }
    {
        const Cam cam = cam_of(a.cam, obs);
        fan_bounds(a.U[obs], cam, fan_origin(a.U[obs], cam), x0, y0, w_log, h_log, f.rays);
    }
    auto rays = [&]() {
        const float4 no = f.rays.no;
#pragma unroll
        for (int r = 0; r < FAN_RAYS; ++r) {
            const uint32_t i = (uint32_t)r * half + lane;
            const uint32_t px = x0 + (i & ((1u << w_log) - 1u)), py = y0 + (i >> w_log);
            const FanRay ray = fan_ray(a.U, a.cam, obs, px, py);
            d[r] = ray.d;
            float en, ex;
            slab_interval(a.ws.root_min, a.ws.root_max, no, ray.inv, 1e-3f, 180.0f, &en, &ex);
            // Pixels outside the frame take no part, nor do rays that miss the scene's box (bvh4d.rs:451).
            const bool in = lane < half && px < od.width && py < od.height && ex >= en && en < 180.0f;
            t_max[r] = in ? 180.0f : 0.0f;
            if (resume && in) {
                const uint32_t pix = od.pix_base + py * od.width + px;
                slot[r] = (int)__ldcg(a.slots + pix);
                if (slot[r] >= 0) t_max[r] = __ldcg(&a.hits[pix].x);
            }
        }
    };
    bool done = true, ready = false;
    if (!a.ws.empty) {
        if (resume) {
            rays();
            ready = true;
        }
        done = closest_fan<OCT>(a.ws, rays, ready, d, 1e-3f, budget, waste, slot, t_max, f, st, a.err);
    }
    *casts = 0;
#pragma unroll
    for (int r = 0; r < FAN_RAYS; ++r) {
        const uint32_t i = (uint32_t)r * half + lane;
        const uint32_t px = x0 + (i & ((1u << w_log) - 1u)), py = y0 + (i >> w_log);
        bool query = false;
        if (lane < half && px < od.width && py < od.height) {
            const uint32_t pix = od.pix_base + py * od.width + px;
            a.slots[pix] = (uint32_t)slot[r];
            if (slot[r] >= 0) query = fan_write(a, obs, pix, (uint32_t)slot[r], t_max[r], d[r], f.rays.no) && done;
        }
        if (__any_sync(FULL_WARP, query)) *casts |= 1u << r;
    }
    return done;
}

// The shadow query of a pixel with a hit; false: it casts none.
__device__ __forceinline__ bool fan_query(const TraceBatchArgs& a, uint32_t obs, uint32_t px, uint32_t py, uint32_t pix,
                                          ShadowQuery* q) {
    const uint32_t slot = __ldcg(a.slots + pix);
    if (slot == 0xFFFFFFFFu) return false;
    float4 o, d;
    float sx, sy;
    camera_ray(a.U[obs], cam_of(a.cam, obs), px, py, &o, &d, &sx, &sy);
    return shadow_query(a, obs, slot, neg4(o), d, __ldcg(&a.hits[pix].x), q);
}

// The parts of 2^size_log pixels of a tile: the longer side halved (the height on a tie).
struct FanParts {
    uint32_t w_log, h_log, across;  // log2 of a part's size and of the parts in a row
};
__device__ __forceinline__ FanParts fan_parts(uint32_t tw_log, uint32_t th_log, uint32_t size_log) {
    FanParts g{tw_log, th_log, 0u};
    while (g.w_log + g.h_log > size_log) {
        if (g.w_log > g.h_log) --g.w_log;
        else --g.h_log;
    }
    g.across = tw_log - g.w_log;
    return g;
}
__device__ __forceinline__ uint32_t part_x(const FanParts& g, uint32_t part) { return (part & ((1u << g.across) - 1u)) << g.w_log; }
__device__ __forceinline__ uint32_t part_y(const FanParts& g, uint32_t part) { return (part >> g.across) << g.h_log; }

// 96 registers (it takes 114 unbounded, without a spill either way) leave room for 20 warps per SM instead of
// 16: the 8-frame launch's closest hits 2.10 ms against 2.29. At 80 it spills and takes 2.37.
template <bool OCT>
__global__ void __maxnreg__(96) k_fan_trace(const __grid_constant__ TraceBatchArgs a, const FanTasks q) {
    extern __shared__ FanQueue sm_queue[];
    FanQueue& sm = sm_queue[threadIdx.x >> 5];
    uint2 st[FAN_LEVELS];
    const uint32_t tiles = a.total_rays >> 5, tw_log = (uint32_t)__ffs((int)a.tile_w) - 1u, th_log = (uint32_t)__ffs((int)a.tile_h) - 1u;
    const uint32_t lane = threadIdx.x & 31u;
    // ahead: the next tile, asked for a tile early (lane 0). No tile belongs to a warp by its number: those
    // that wait must wait for running warps only, and a block may start late where other launches run.
    uint32_t mine = 0, ahead = 0;
    if (lane == 0) ahead = atomicAdd(q.count + FAN_NEXT, 1u);
    bool whole = true;  // whole tiles first, then the queue
    for (;;) {
        uint32_t tile, part = 0;
        if (whole) {
            tile = __shfl_sync(FULL_WARP, ahead, 0);
            if (lane == 0 && tile < tiles) ahead = atomicAdd(q.count + FAN_NEXT, 1u);
            if (tile >= tiles) {
                fan_first_done(q, mine);
                whole = false;
            }
        }
        if (!whole) {
            const uint32_t task = fan_take(q, tiles, tiles, a.err);
            if (!task) break;
            tile = (task - 1u) >> FAN_PARTS_LOG;
            part = (task - 1u) & ((1u << FAN_PARTS_LOG) - 1u);
        }
        const FanTile t = fan_tile(a, tile);
        const bool pair = part >= FAN_GROUPS;
        if (pair) part -= FAN_GROUPS;
        const uint32_t size_log = whole ? tw_log + th_log : (pair ? FAN_PAIR_LOG : FAN_GROUP_LOG);
        const FanParts g = fan_parts(tw_log, th_log, size_log);
        const uint32_t x0 = part_x(g, part), y0 = part_y(g, part);  // in the tile
        uint32_t casts;
        const bool done = fan_pixels<OCT>(a, t.obs, t.x + x0, t.y + y0, g.w_log, g.h_log, !whole, pair ? FAN_UNLIMITED : FAN_BUDGET,
                                          pair ? FAN_UNLIMITED : q.waste, sm, st, &casts);
        if (!done) {
            // A tile into groups; a group into its pairs, numbered over the tile.
            const FanParts p = fan_parts(tw_log, th_log, FAN_PAIR_LOG);
            // Pairs lie along rows (the last halving is of the height), as a group's pixels 2 k and 2 k + 1 do.
            const uint32_t px = x0 + ((2u * lane) & ((1u << g.w_log) - 1u)), py = y0 + ((2u * lane) >> g.w_log);
            if (pair) {
                if (lane == 0) atomicOr(a.err, ERR_TRAVERSAL_LIMIT);
            } else if (size_log > FAN_GROUP_LOG) {
                fan_push(q, tile, lane, lane < (1u << (size_log - FAN_GROUP_LOG)));
            } else {
                fan_push(q, tile, FAN_GROUPS + ((py >> p.h_log) << p.across) + (px >> p.w_log), lane < (1u << (FAN_GROUP_LOG - FAN_PAIR_LOG)));
            }
        } else if (casts) {
            fan_list(q.shadows, q.num_shadows, tile, whole ? lane : FAN_HALVES + part + (pair ? FAN_GROUPS : 0u),
                     lane < 2u && (whole ? (casts >> lane) & 1u : lane == 0u));
        }
        if (whole) ++mine;
        else fan_finished(q);
    }
}

__global__ void __launch_bounds__(512) k_fan_shadow(const __grid_constant__ TraceBatchArgs a, const FanTasks q) {
    extern __shared__ FanShadows sm_shadows[];
    FanShadows& sm = sm_shadows[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    uint2 st[FAN_LEVELS];
    const uint32_t tw_log = (uint32_t)__ffs((int)a.tile_w) - 1u, th_log = (uint32_t)__ffs((int)a.tile_h) - 1u;
    const uint32_t tasks = *q.num_shadows, part_mask = (1u << FAN_PARTS_LOG) - 1u;
    if (tasks == 0 || *q.dirty) return;
    uint32_t mine = 0;
    for (;;) {
        const uint32_t next = warp_next(q.count + FAN_NEXT);
        if (next >= tasks) break;
        const uint32_t task = q.shadows[next] - 1u, tile = task >> FAN_PARTS_LOG, part = task & part_mask;
        const bool half = part < FAN_HALVES, pair = part >= FAN_HALVES + FAN_GROUPS;
        const FanParts g = fan_parts(tw_log, th_log, half ? tw_log + th_log : (pair ? FAN_PAIR_LOG : FAN_GROUP_LOG));
        const uint32_t k = half ? 0u : part - FAN_HALVES - (pair ? FAN_GROUPS : 0u);
        const FanTile t = fan_tile(a, tile);
        const uint32_t n = 1u << (g.w_log + g.h_log - (half ? 1u : 0u));  // the task's pixels
        const uint32_t i = (half ? n * part : 0u) + lane;
        const uint32_t x = part_x(g, k) + (i & ((1u << g.w_log) - 1u)), y = part_y(g, k) + (i >> g.w_log);  // in the tile
        const ObsDev& od = a.obs[t.obs];
        const uint32_t px = t.x + x, py = t.y + y, pix = od.pix_base + py * od.width + px;
        ShadowQuery s;
        s.no = v4(0.0f, 0.0f, 0.0f, 0.0f);
        s.d = v4(0.0f, 0.0f, 1.0f, 0.0f);
        s.t_max = 0.0f;
        s.enters = false;
        const bool query = lane < n && px < od.width && py < od.height &&
                           fan_query(a, t.obs, px, py, pix, &s);
        const bool enters = query && s.enters;
        bool hit = false, done = true;
        if (__any_sync(FULL_WARP, enters))
            done = any_fan(a.ws, enters, s.no, s.d, 2.0f * (float)x / (float)(a.tile_w - 1u) - 1.0f,
                           2.0f * (float)y / (float)(a.tile_h - 1u) - 1.0f, 2e-3f, s.t_max, FAN_ANY_BUDGET, hit, sm, st);
        const bool pending = !done && enters && !hit;
        if (query) a.shadow[pix] = hit ? 2 : 1;
        if (__any_sync(FULL_WARP, pending)) fan_push(q, tile, (y << tw_log) + x, pending);
        ++mine;
    }
    fan_first_done(q, mine);
    for (;;) {
        const uint32_t task = fan_take(q, tasks, a.total_rays >> 5, a.err);
        if (!task) break;
        const uint32_t i = (task - 1u) & part_mask;
        const FanTile t = fan_tile(a, (task - 1u) >> FAN_PARTS_LOG);
        const ObsDev& od = a.obs[t.obs];
        const uint32_t px = t.x + (i & ((1u << tw_log) - 1u)), py = t.y + (i >> tw_log), pix = od.pix_base + py * od.width + px;
        ShadowQuery s;
        if (px < od.width && py < od.height && fan_query(a, t.obs, px, py, pix, &s)) {  // the same for every lane
            const bool hit = any_fan_one(a.ws, s.no, s.d, s.t_min, s.t_max, st, a.err);
            if (lane == 0) a.shadow[pix] = hit ? 2 : 1;
        }
        fan_finished(q);
    }
}

// Resident blocks per SM of k_fan_trace.
static cudaError_t fan_resident(int threads, int* blocks) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_fan_trace<true>, threads, (size_t)(threads / 32) * sizeof(FanQueue));
}

// The shared-memory stack depths the lean kernel is built for (SrTuning.stack_smem).
#define SR_LEAN_STACKS(X) X(0) X(8) X(10) X(12) X(16)

bool lean_stack_supported(uint32_t s) {
#define SR_ONE(S) if (s == (S)) return true;
    SR_LEAN_STACKS(SR_ONE)
#undef SR_ONE
    return false;
}

// The shared-memory stack and the staged top levels of the lean kernel can exceed the 48 KB
// default of one block.
template <bool COUNT, int SS, bool OCT, bool TOP>
static cudaError_t lean_attr(int max_smem) {
    return SS > 0 || TOP
               ? cudaFuncSetAttribute(k_trace_lean<COUNT, SS, OCT, TOP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      max_smem)
               : cudaSuccess;
}

template <int SS>
static cudaError_t lean_attrs_ss(int max_smem) {
    cudaError_t e = lean_attr<false, SS, true, false>(max_smem);
    if (e == cudaSuccess) e = lean_attr<true, SS, true, false>(max_smem);
    if (e == cudaSuccess) e = lean_attr<false, SS, false, false>(max_smem);
    if (e == cudaSuccess) e = lean_attr<true, SS, false, false>(max_smem);
    if constexpr (SS == 0 || SS == 12) {  // the depths built with staged top levels (octant layout)
        if (e == cudaSuccess) e = lean_attr<false, SS, true, true>(max_smem);
        if (e == cudaSuccess) e = lean_attr<true, SS, true, true>(max_smem);
    }
    return e;
}

static cudaError_t lean_kernel_attrs(int max_smem) {
    cudaError_t e = cudaSuccess;
#define SR_ONE(S) \
    if (e == cudaSuccess) e = lean_attrs_ss<(S)>(max_smem);
    SR_LEAN_STACKS(SR_ONE)
#undef SR_ONE
    return e;
}

template <int SS>
static void launch_lean_ss(bool count, bool oct, bool top, uint32_t blocks, uint32_t threads, size_t smem, cudaStream_t st,
                           const TraceBatchArgs& ta) {
    if constexpr (SS == 0 || SS == 12) {
        if (top && oct) {
            if (count) k_trace_lean<true, SS, true, true><<<blocks, threads, smem, st>>>(ta);
            else k_trace_lean<false, SS, true, true><<<blocks, threads, smem, st>>>(ta);
            return;
        }
    }
    if (oct) {
        if (count) k_trace_lean<true, SS, true, false><<<blocks, threads, smem, st>>>(ta);
        else k_trace_lean<false, SS, true, false><<<blocks, threads, smem, st>>>(ta);
    } else {
        if (count) k_trace_lean<true, SS, false, false><<<blocks, threads, smem, st>>>(ta);
        else k_trace_lean<false, SS, false, false><<<blocks, threads, smem, st>>>(ta);
    }
}

static void launch_lean(uint32_t ss, bool count, bool oct, bool top, uint32_t blocks, uint32_t threads, size_t smem,
                        cudaStream_t st, const TraceBatchArgs& ta) {
#define SR_ONE(S)                                                             \
    if (ss == (S)) {                                                          \
        launch_lean_ss<(S)>(count, oct, top, blocks, threads, smem, st, ta);  \
        return;                                                               \
    }
    SR_LEAN_STACKS(SR_ONE)
#undef SR_ONE
}

struct ShadeBatchArgs {
    SceneDev s;
    WideScene ws;
    const SrGpuUniforms* U;
    const float4* cam;
    const ObsDev* obs;
    const uint32_t* pix_pre;
    uint32_t n, total_px;
    const float4* hits;
    const uint32_t* slots;
    const uint8_t* shadow;
    float4* hdr;
    uint32_t* hit_id;
    float* lambda;
    float* tau;
    uint32_t* counters;  // [0] shadow rays, [1] errors
    unsigned long long* work;
    BBConst bb;
    uint32_t stars_binned;  // observers passing stars_binned_for get their stars from k_star_tiles
};

// The shadow queries of a pixel's shading: the main light's was traced by the trace kernel (its
// state must say so); with flashes in the frame every query is traced here. The SIMPLE kernel
// (no flashes in the batch) carries no traversal code.
template <bool COUNT, bool SIMPLE>
struct FrameOccluder {
    const WideScene* s;
    uint32_t* err;
    Work* work;
    uint8_t state;
    bool trace_here;
    __device__ bool operator()(float4 o, float4 d, float t0, float t1) {
        if (!SIMPLE && trace_here) return occluded_wide<COUNT>(*s, o, d, t0, t1, err, work);
        if (state == 0) atomicOr(err, ERR_SHADOW_MISMATCH);
        return state == 2;
    }
};

// SIMPLE: every observer of the batch is flash-free and gets its stars (if any) from the binned
// pass, so the kernel has neither shadow traversal nor the per-pixel star sum.
template <bool COUNT, bool SIMPLE>
__global__ void __launch_bounds__(256, SIMPLE ? 4 : 3) k_shade_batch(const __grid_constant__ ShadeBatchArgs a) {
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.total_px) return;
    uint32_t o = find_obs(a.pix_pre, a.n, p);
    uint32_t l = p - __ldg(a.pix_pre + o);
    const ObsDev& od = a.obs[o];
    uint32_t px = l % od.width, py = l / od.width;
    const SrGpuUniforms& U = a.U[o];
    const Cam cam = cam_of(a.cam, o);
    float4 ro, rd;
    float sx, sy;
    camera_ray(U, cam, px, py, &ro, &rd, &sx, &sy);
    uint32_t slot = a.slots[p];
    Work work{0, 0, 0};
    uint32_t shadow_rays = 0;
    Hit h;
    h.lambda = 0.0f;
    h.tau = 0.0f;
    F3 color;
    if (slot != 0xFFFFFFFFu) {
        float4 hr = a.hits[p];
        GeomHit gh{hr.x, hr.y, hr.z, hr.w};
        interpolate(a.s.attrs + 12u * slot, ro, rd, gh, &h);
        FrameOccluder<COUNT, SIMPLE> occ{&a.ws, a.counters + 1, &work, a.shadow[p], U.num_flashes != 0u};
        color = shade_hit(a.s, U, cam, rd, h, occ, &shadow_rays);
        if (U.num_haze > 0u) color = apply_haze(color, h.event, U);
    } else {
        color = shade_sky(rd);
    }
    if (!SIMPLE && U.mode == 0u && a.s.num_stars > 0u && !(a.stars_binned && stars_binned_for(U, a.s.num_stars)))
        color = add(color, stars_brute(a.s, U, cam, ro, rd, sx, sy, slot != 0xFFFFFFFFu ? h.lambda : INFINITY, a.bb));
    a.hdr[(size_t)od.pyr_base + l] = make_float4(color.x, color.y, color.z, 0.0f);
    if (a.hit_id)
        a.hit_id[p] = slot == 0xFFFFFFFFu ? 0xFFFFFFFFu : (a.s.leaf_to_orig ? __ldg(a.s.leaf_to_orig + slot) : slot);
    if (a.lambda) a.lambda[p] = h.lambda;
    if (a.tau) a.tau[p] = h.tau;
    if (shadow_rays) atomicAdd(a.counters, shadow_rays);
    if (COUNT && work.nodes) add_work(a.work + 3, work);
}

}  // namespace srk

#include "sr_batch_bloom.cuh"
#include "sr_stars.cuh"
#include "sr_adjoint.cuh"

namespace srk {

// ---------------------------------------------------------------------------------------------
// The batch sequence.
// ---------------------------------------------------------------------------------------------
namespace {

uint64_t mix(uint64_t h, uint64_t v) {
    h ^= v + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2);
    return h;
}

struct Shape {
    uint32_t n = 0, total_tiles = 0, total_px = 0, total_pyr = 0, total_star_tiles = 0;
    std::vector<ObsDev> obs;
    std::vector<uint32_t> pre;  // (SR_BLOOM_LEVELS + 3) rows of n + 1: tiles, levels 0..6, star tiles
};

Shape make_shape(const BatchRequest& r, uint32_t tile_w, uint32_t tile_h) {
    Shape s;
    s.n = r.n;
    s.obs.resize(r.n);
    // Rows of n + 1: trace tiles, bloom levels 0..6, 16x16 star tiles.
    const uint32_t rows = SR_BLOOM_LEVELS + 3, stride = r.n + 1;
    s.pre.assign((size_t)rows * stride, 0);
    uint32_t tiles = 0, px = 0, pyr = 0, star_tiles = 0;
    for (uint32_t i = 0; i < r.n; ++i) {
        ObsDev& o = s.obs[i];
        std::memset(&o, 0, sizeof(o));
        o.width = r.u[i].size[0];
        o.height = r.u[i].size[1];
        o.tiles_x = (o.width + tile_w - 1) / tile_w;
        o.tile_base = tiles;
        o.pix_base = px;
        o.pyr_base = pyr;
        o.has_cam64 = r.cam64 ? 1u : 0u;
        o.star_tile_base = star_tiles;
        s.pre[(size_t)(SR_BLOOM_LEVELS + 2) * stride + i] = star_tiles;
        star_tiles += ((o.width + STAR_TILE - 1) / STAR_TILE) * ((o.height + STAR_TILE - 1) / STAR_TILE);
        Pyramid p = make_pyramid(o.width, o.height);
        for (int k = 0; k <= SR_BLOOM_LEVELS; ++k) { o.lw[k] = p.w[k]; o.lh[k] = p.h[k]; o.loff[k] = p.off[k]; }
        o.loff[SR_BLOOM_LEVELS + 1] = p.off[SR_BLOOM_LEVELS + 1];
        s.pre[0 * stride + i] = tiles;
        for (int k = 0; k <= SR_BLOOM_LEVELS; ++k) {
            uint32_t* row = &s.pre[(size_t)(1 + k) * stride];
            row[i + 1] = row[i] + p.w[k] * p.h[k];
        }
        tiles += o.tiles_x * ((o.height + tile_h - 1) / tile_h);
        px += o.width * o.height;
        pyr += p.off[SR_BLOOM_LEVELS + 1];
    }
    s.pre[r.n] = tiles;
    s.pre[(size_t)(SR_BLOOM_LEVELS + 2) * stride + r.n] = star_tiles;
    s.total_star_tiles = star_tiles;
    s.total_tiles = tiles;
    s.total_px = px;
    s.total_pyr = pyr;
    return s;
}

}  // namespace

static WideScene wide_scene(const FastScene& s, const SceneDev& sd) {
    WideScene ws;
    ws.boxes = s.boxes.as<float4>();
    ws.oct_stride = 4ull * s.num_wide;
    ws.refs = s.refs.as<uint2>();
    ws.up = s.up.as<uint32_t>();
    ws.leafpar = s.leafpar.as<uint32_t>();
    ws.geoms = sd.geoms;
    ws.root_min = make_float4(s.root_min[0], s.root_min[1], s.root_min[2], s.root_min[3]);
    ws.root_max = make_float4(s.root_max[0], s.root_max[1], s.root_max[2], s.root_max[3]);
    ws.root_ref = s.root_ref;
    ws.empty = s.empty ? 1u : 0u;
    ws.fan_box = s.fan_box.as<float4>();
    ws.fan_ref = s.fan_ref.as<uint32_t>();
    ws.fan_root = s.fan_root;
    ws.leaf_bits = 0;
    while (s.max_leaf >> ws.leaf_bits) ++ws.leaf_bits;
    ws.oct_copies = s.copies == 16 ? 1u : 0u;
    return ws;
}

// Whether the node layouts give a ray trace_ref's hit bit for bit: their comparisons assume a range from 0 or
// beyond and finite values (no product of a coordinate, an inverse direction and a box overflows to a NaN).
__device__ __forceinline__ bool layout_ray(float4 o, float4 d, float t_min, float t_max) {
    const float lim = 1e12f;
    const auto in = [&](float v) { return fabsf(v) <= lim; };  // false for a NaN
    return t_min >= 0.0f && t_max > 0.0f && in(o.x) && in(o.y) && in(o.z) && in(o.w) && in(d.x) && in(d.y) && in(d.z) && in(d.w);
}

__device__ __forceinline__ void write_ray_hit(const SceneDev& s, double a0, double a1, double a2, double a3, float4 o, float4 d,
                                              int slot, const GeomHit& gh, SrRayHit* to) {
    SrRayHit out;
    out.id = 0xFFFFFFFFu;
    out.slot = 0xFFFFFFFFu;
    out.lambda = out.proper_time = 0.0f;
    for (int k = 0; k < 4; ++k) { out.event[k] = 0.0; out.tet_bary[k] = 0.0f; }
    out.uv[0] = out.uv[1] = 0.0f;
    out.material = out.pad = 0u;
    if (slot >= 0) {
        Hit h;
        interpolate(s.attrs + 12u * (uint32_t)slot, o, d, gh, &h);
        out.slot = (uint32_t)slot;
        out.id = s.leaf_to_orig ? __ldg(s.leaf_to_orig + slot) : (uint32_t)slot;
        out.lambda = h.lambda;
        out.proper_time = h.tau;
        out.event[0] = (double)h.event.x + a0;
        out.event[1] = (double)h.event.y + a1;
        out.event[2] = (double)h.event.z + a2;
        out.event[3] = (double)h.event.w + a3;
        out.tet_bary[0] = h.b0;
        out.tet_bary[1] = h.b1;
        out.tet_bary[2] = h.b2;
        out.tet_bary[3] = h.b3;
        out.uv[0] = h.uv_u;
        out.uv[1] = h.uv_v;
        out.material = h.material;
    }
    *to = out;
}

// Caller rays (sr_trace_rays), one thread per ray on the reference's nodes: scenes without the layouts, long lists,
// and the rays that the walk over the fan layout leaves (`rest`, counters[2] of them; null: all n).
__global__ void __launch_bounds__(64) k_trace_rays(const SceneDev s, double a0, double a1, double a2, double a3, const SrRay* rays,
                                                   uint32_t n, const uint32_t* rest, SrRayHit* hits, uint32_t* counters) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (rest ? counters[2] : n)) return;
    if (rest) i = rest[i];
    const SrRay r = rays[i];
    const float4 o = v4((float)(r.origin[0] - a0), (float)(r.origin[1] - a1), (float)(r.origin[2] - a2),
                        (float)(r.origin[3] - a3));
    const float4 d = v4(r.dir[0], r.dir[1], r.dir[2], r.dir[3]);
    GeomHit gh{0.0f, 0.0f, 0.0f, 0.0f};
    const int slot = trace_ref(s, o, d, r.t_min, r.t_max, &gh, counters + 1);
    write_ray_hit(s, a0, a1, a2, a3, o, d, slot, gh, hits + i);
}

// Caller rays on the fan layout, one warp per ray: boxes and records one per lane against the ray itself,
// nearest subtree first. A ray's own walk over binary nodes, one thread per ray, is a chain of dependent
// loads, and the call waits for its longest: 4096 rays into 1M tetrahedra took 670 us.
//
// The hit is the reference's. Of the records that the ray hits and whose leaf box it enters, let k have the
// smallest lambda; when the box's entry parameter as computed is not beyond it, every box on the way to
// k is entered before any hit so far (boxes hold their children's), so the reference tests k, and no
// nearer one. A hit before its box's entry is rounding against the build's padding; boxes are culled only
// 0.1% beyond the closest hit, so that one is met rather than culled, and the ray then takes the reference's own
// walk, as the rays that the layouts do not take: here, the whole warp doing the same, or, with `rest`, listed for a
// thread each (k_trace_rays). Of hits at equal lambda the reference keeps the one its order meets first
// (packet_precedes).
template <bool OCT>
__global__ void __launch_bounds__(128) k_trace_rays_fan(const SceneDev s, const __grid_constant__ WideScene ws, double a0, double a1,
                                                        double a2, double a3, const SrRay* rays, uint32_t n, uint32_t* rest,
                                                        SrRayHit* hits, uint32_t* counters) {
    const uint32_t i = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (i >= n) return;
    const SrRay r = rays[i];
    const float4 o = v4((float)(r.origin[0] - a0), (float)(r.origin[1] - a1), (float)(r.origin[2] - a2),
                        (float)(r.origin[3] - a3));
    const float4 d = v4(r.dir[0], r.dir[1], r.dir[2], r.dir[3]);
    const float4 no = neg4(o), inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
    GeomHit best{0.0f, 0.0f, 0.0f, 0.0f};
    int slot = -1;
    bool reference = !layout_ray(o, d, r.t_min, r.t_max);
    float en, ex;
    slab_interval(ws.root_min, ws.root_max, no, inv, r.t_min, r.t_max, &en, &ex);
    if (!reference && !ws.empty && ex >= en && en < r.t_max) {
        uint2 st[FAN_LEVELS];
        float t_max = r.t_max, limit = t_max;  // limit: boxes entered beyond it are culled
        uint32_t node = ws.fan_root, depth = 0, visits = 0;
        for (;;) {
            if (++visits > MAX_VISITS_FAST) {
                if (lane == 0) atomicOr(counters + 1, ERR_TRAVERSAL_LIMIT);
                break;
            }
            const float4* bx = ws.fan_box + (size_t)node * 64u;
            uint32_t ref = __ldg(ws.fan_ref + (size_t)node * 32u + lane);
            slab_interval(__ldg(bx + lane), __ldg(bx + 32u + lane), no, inv, r.t_min, limit, &en, &ex);
            const bool meets = ex >= en, leaf = (ref & REF_LEAF) != 0u;
            // en + 0: no sign bit on a zero entry.
            uint32_t key = meets && !leaf ? ((__float_as_uint(en + 0.0f) & ~31u) | lane) : FAN_NONE;
            FanDeal deal{__ballot_sync(FULL_WARP, meets && leaf), 0u, 0u, 0u};
            while (deal.leaves | deal.left) {
                uint32_t mine, from;
                const uint32_t held = fan_deal(deal, ref, lane, mine, from);
                const float entry = __shfl_sync(FULL_WARP, en, from);
                GeomHit gh;
                // Hits up to and including t_max, so that a hit at the closest hit's lambda is seen.
                const bool h = lane < held && intersect_lean(ws.geoms + 5u * mine, no, d, r.t_min,
                                                             __uint_as_float(__float_as_uint(t_max) + 1u), &gh);
                if (!__any_sync(FULL_WARP, h)) continue;
                if (__any_sync(FULL_WARP, h && !(gh.lambda >= entry))) reference = true;  // a NaN too
                const uint32_t nearest = redux_min(h ? __float_as_uint(gh.lambda) : FAN_NONE);
                for (uint32_t m = __ballot_sync(FULL_WARP, h && __float_as_uint(gh.lambda) == nearest); m; m &= m - 1u) {
                    const uint32_t c = (uint32_t)__ffs((int)m) - 1u, rec = __shfl_sync(FULL_WARP, mine, c);
                    const GeomHit g{__shfl_sync(FULL_WARP, gh.lambda, c), __shfl_sync(FULL_WARP, gh.u, c),
                                    __shfl_sync(FULL_WARP, gh.v, c), __shfl_sync(FULL_WARP, gh.w, c)};
                    if (g.lambda < t_max ||
                        (slot >= 0 && packet_precedes<OCT>(ws, rec, (uint32_t)slot, no, inv, r.t_min, counters + 1))) {
                        t_max = g.lambda;
                        best = g;
                        slot = (int)rec;
                    }
                }
                limit = fminf(r.t_max, t_max * 1.001f);
            }
            uint32_t k = redux_min(key);
            while ((k & ~31u) > __float_as_uint(limit) && depth > 0) {
                const uint2 e = st[--depth];
                key = e.x;
                ref = e.y;
                k = redux_min(key);
            }
            if ((k & ~31u) > __float_as_uint(limit)) break;
            const uint32_t c = k & 31u;
            node = __shfl_sync(FULL_WARP, ref, c);
            if (lane == c) key = FAN_NONE;
            st[depth++] = make_uint2(key, ref);
        }
    }
    if (reference && rest) {
        if (lane == 0) rest[atomicAdd(counters + 2, 1u)] = i;
        return;
    }
    if (reference) slot = trace_ref(s, o, d, r.t_min, r.t_max, &best, counters + 1);  // the same for every lane
    if (lane == 0) write_ray_hit(s, a0, a1, a2, a3, o, d, slot, best, hits + i);
}

// Lists longer than this walk a ray per thread: a warp per ray shortens the longest ray's chain of loads, which a
// short list waits for, and issues more for each, which a long one waits for. Whole calls, thread against warp per ray
// (us): 65,536 rays into 8 accelerated bodies 1362 and 817, into 64 of them 3429 and 1988 (neighbouring directions
// 1842 and 1192), into 147k tetrahedra 867 and 844; 262,144: 2766 and 2700, 7193 and 7129 (3261 and 4310), 2297 and
// 3105; a million: 12.7 and 13.5 ms, 29.5 and 30.8 (11.7 and 19.3), 11.2 and 14.9.
constexpr uint32_t RAYS_LONG = 1u << 16;
// Lists longer than this leave the rays that take the reference's walk to a second launch, a thread each; in a shorter
// one their warps walk them at once, alone in it as they are: lists of nothing else, warps against threads, 4096 rays
// into 8 accelerated bodies 616 and 845 us, into 64 of them 1039 and 2907; 16,384: 783 and 1031, 1816 and 2899; but
// 65,536: 1188 and 1356, 4910 and 3432. The launch costs 2 us of a 69 us call.
constexpr uint32_t RAYS_REST = 1u << 14;

cudaError_t fast_trace_rays(FastScene& s, const SceneDev& sd, const double anchor[4], const SrRay* rays, uint32_t n,
                            SrRayHit* hits, uint32_t* rest, uint32_t* counters, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const double *a = anchor;
    const uint32_t blocks = (n + 3) / 4;
    if (s.usable && n <= RAYS_LONG) {
        cudaError_t e = fan_ready(s, sd, st);
        if (e != cudaSuccess) return e;
    }
    if (!s.usable || s.fan_levels == 0 || n > RAYS_LONG) {
        k_trace_rays<<<(n + 63) / 64, 64, 0, st>>>(sd, a[0], a[1], a[2], a[3], rays, n, nullptr, hits, counters);
        return cudaGetLastError();
    }
    const WideScene ws = wide_scene(s, sd);
    if (n <= RAYS_REST) rest = nullptr;
    if (ws.oct_copies)
        k_trace_rays_fan<true><<<blocks, 128, 0, st>>>(sd, ws, a[0], a[1], a[2], a[3], rays, n, rest, hits, counters);
    else
        k_trace_rays_fan<false><<<blocks, 128, 0, st>>>(sd, ws, a[0], a[1], a[2], a[3], rays, n, rest, hits, counters);
    if (rest) k_trace_rays<<<(n + 63) / 64, 64, 0, st>>>(sd, a[0], a[1], a[2], a[3], rays, n, rest, hits, counters);
    return cudaGetLastError();
}

float4* fast_batch_hdr(FastCtx& c, uint32_t pyr_base) { return c.hdr.as<float4>() + pyr_base; }

cudaError_t fast_render_batch(FastCtx& c, FastScene& s, const SrTuning& t, const SceneDev& sd,
                              const double anchor[4], const BBConst& bb, uint32_t* counters, const BatchRequest& r,
                              cudaStream_t st) {
    if (r.n == 0) return cudaSuccess;
    c.adj_valid = false;  // the batch buffers the gradient's outcomes live in are about to change
    auto drop_graphs = [&]() {  // their last launches may still run
        cudaStreamSynchronize(st);
        fast_release(c);
    };
    // The packet walk; counting runs take the per-lane order, whose work counts are the reference's.
    uint64_t pixels = 0;
    for (uint32_t i = 0; i < r.n; ++i) pixels += (uint64_t)r.u[i].size[0] * r.u[i].size[1];
    cudaError_t e;
    bool packet = t.packet != 0 && !r.count_work && !lone_rays(sd.num_prims, pixels);
    if (packet && !s.empty) {
        if ((e = fan_ready(s, sd, st)) != cudaSuccess) return e;
        packet = s.fan_levels != 0;
    }
    Shape sh;
    uint32_t tile_w = t.tile_w, tile_h = t.tile_h;
    if (packet) {
        const uint32_t size_log = fan_tile_log(pixels);
        (tile_w < tile_h ? tile_w : tile_h) *= 2;
        while (tile_w * tile_h > (1u << size_log)) (tile_w > tile_h ? tile_w : tile_h) /= 2;
        sh = make_shape(r, tile_w, tile_h);
        const size_t old = c.fan_list.bytes, old_shadows = c.fan_shadows.bytes;
        // Without room for the queue the rays walk alone. The queue's own buffer: its entries are zero
        // between launches, whatever the next one's size, the list's are not.
        if (!c.fan_lost.p && c.fan_lost.ensure(64) == cudaSuccess) std::memset(c.fan_lost.p, 0, c.fan_lost.bytes);
        packet = sh.total_tiles < FAN_MAX_TILES && c.fan_lost.p &&
                 c.fan_list.ensure((size_t)sh.total_tiles * FAN_QUEUED_PER_TILE * 4) == cudaSuccess &&
                 c.fan_shadows.ensure((size_t)sh.total_tiles * FAN_SHADOWS_PER_TILE * 4) == cudaSuccess;
        if (c.fan_list.bytes != old || c.fan_shadows.bytes != old_shadows) drop_graphs();
        if (c.fan_list.bytes != old && c.fan_list.p) {
            cudaError_t z = cudaMemsetAsync(c.fan_list.p, 0, c.fan_list.bytes, st);
            if (z != cudaSuccess) return z;
        }
        if (!packet) cudaGetLastError();
    }
    if (!packet) {
        tile_w = t.tile_w;
        tile_h = t.tile_h;
        sh = make_shape(r, tile_w, tile_h);
    }
    const uint32_t n = r.n, stride = n + 1;
    if ((uint64_t)sh.total_tiles * 32 >= (1ull << 32)) return cudaErrorInvalidValue;
    // Buffers (grown on demand; a growth invalidates every captured graph).
    size_t old_hits = c.hits.bytes, old_hdr = c.hdr.bytes, old_U = c.inputs.bytes, old_sh = c.shadow.bytes, old_rgb = c.rgb.bytes;
    // The batch's inputs are one block, copied at once: uniforms, cameras, observers, prefix rows.
    const size_t at_cam = n * sizeof(SrGpuUniforms), at_obs = at_cam + n * sizeof(SrCameraF64);
    const size_t at_pre = at_obs + n * sizeof(ObsDev), in_bytes = at_pre + sh.pre.size() * 4;
    static_assert(sizeof(SrGpuUniforms) % 16 == 0 && sizeof(SrCameraF64) % 8 == 0 && sizeof(ObsDev) % 8 == 0, "the block's parts stay aligned");
    if ((e = c.inputs.ensure(in_bytes)) != cudaSuccess) return e;
    if ((e = c.cam.ensure(n * 6 * sizeof(float4))) != cudaSuccess) return e;
    if ((e = c.hits.ensure((size_t)sh.total_px * sizeof(float4))) != cudaSuccess) return e;
    if ((e = c.slots.ensure((size_t)sh.total_px * 4)) != cudaSuccess) return e;
    if ((e = c.shadow.ensure((size_t)sh.total_px)) != cudaSuccess) return e;  // shadow states
    if ((e = c.hdr.ensure((size_t)sh.total_pyr * sizeof(float4))) != cudaSuccess) return e;
    if (!c.sched.p) {
        if ((e = c.sched.ensure(std::max<size_t>((size_t)c.num_sms + 1, FAN_DIRTY + 1) * 4)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(c.sched.p, 0, c.sched.bytes, st)) != cudaSuccess) return e;
    }
    bool shadows = false;  // some observer casts shadow rays
    for (uint32_t i = 0; i < n; ++i)
        shadows = shadows || (r.u[i].mode == 0u && r.u[i].shadow_mode != 0u && r.u[i].num_flashes == 0u);
    bool binned = false;
    if (!r.star_brute && sd.num_stars > 0)
        for (uint32_t i = 0; i < n; ++i) binned = binned || stars_binned_for(r.u[i], sd.num_stars);
    // A flash-free batch whose stars all come from the binned pass shades with the SIMPLE kernel.
    bool simple = true;
    for (uint32_t i = 0; i < n; ++i) {
        const SrGpuUniforms& ui = r.u[i];
        if (ui.num_flashes != 0u ||
            (ui.mode == 0u && sd.num_stars > 0u && !(binned && stars_binned_for(ui, sd.num_stars))))
            simple = false;
    }
    const size_t old_star = c.star_r.bytes + c.star_box.bytes + c.star_count.bytes + c.star_list.bytes + c.star_scan.bytes;
    // Star lists: room for every (observer, star) in 8 tiles; tiles past the room sum every star.
    const uint32_t list_cap = (uint32_t)std::min<uint64_t>(
        c.star_room ? (uint64_t)c.star_room * n : std::max<uint64_t>(8ull * n * sd.num_stars, 1u << 20), 1u << 30);
    c.batch_list_cap = list_cap;
    size_t scan_bytes = 0;
    if (binned) {
        const size_t pairs = (size_t)n * sd.num_stars;
        const size_t tiles = sh.total_star_tiles;
        cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)tiles, st);
        if ((e = c.star_r.ensure(pairs * sizeof(float4))) != cudaSuccess) return e;
        if ((e = c.star_color.ensure(pairs * sizeof(float4))) != cudaSuccess) return e;
        if ((e = c.star_box.ensure(pairs * sizeof(float4))) != cudaSuccess) return e;
        if ((e = c.star_count.ensure(2 * tiles * 4)) != cudaSuccess) return e;
        if ((e = c.star_offset.ensure(tiles * 4)) != cudaSuccess) return e;
        if ((e = c.star_list.ensure((size_t)list_cap * 4)) != cudaSuccess) return e;
        if ((e = c.star_scan.ensure(scan_bytes)) != cudaSuccess) return e;
    }
    if (c.star_r.bytes + c.star_box.bytes + c.star_count.bytes + c.star_list.bytes + c.star_scan.bytes != old_star)
        drop_graphs();
    if (!r.rgb && (e = c.rgb.ensure((size_t)sh.total_px * 4)) != cudaSuccess) return e;
    if (c.hits.bytes != old_hits || c.hdr.bytes != old_hdr || c.inputs.bytes != old_U || c.shadow.bytes != old_sh ||
        c.rgb.bytes != old_rgb)
        drop_graphs();
    // Two pinned staging blocks in turn, so that a call does not wait for the batch before it: a block is
    // rewritten once the copy from it, two calls ago, has run.
    const int slot = c.staging_next;
    c.staging_next = 1 - slot;
    if (!c.staged[slot] && (e = cudaEventCreateWithFlags(&c.staged[slot], cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventSynchronize(c.staged[slot])) != cudaSuccess) return e;
    if ((e = c.staging[slot].ensure(in_bytes)) != cudaSuccess) return e;
    unsigned char* host = c.staging[slot].as<unsigned char>();
    std::memcpy(host, r.u, n * sizeof(SrGpuUniforms));
    if (r.cam64) std::memcpy(host + at_cam, r.cam64, n * sizeof(SrCameraF64));
    std::memcpy(host + at_obs, sh.obs.data(), n * sizeof(ObsDev));
    std::memcpy(host + at_pre, sh.pre.data(), sh.pre.size() * 4);
    unsigned char* dev = c.inputs.as<unsigned char>();
    if ((e = cudaMemcpyAsync(dev, host, in_bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(c.staged[slot], st)) != cudaSuccess) return e;
    struct {
        const SrGpuUniforms* U;
        const SrCameraF64* cam64;
        const ObsDev* obs;
        const uint32_t* pre;
    } in{reinterpret_cast<const SrGpuUniforms*>(dev), reinterpret_cast<const SrCameraF64*>(dev + at_cam),
         reinterpret_cast<const ObsDev*>(dev + at_obs), reinterpret_cast<const uint32_t*>(dev + at_pre)};
    c.batch_U = in.U;
    c.batch_obs = in.obs;

    uint32_t* rgb = r.rgb ? r.rgb : c.rgb.as<uint32_t>();
    const WideScene ws = wide_scene(s, sd);
    unsigned long long* work = reinterpret_cast<unsigned long long*>(counters + 4);
    const uint32_t* tile_pre = in.pre;
    const uint32_t* pix_pre = tile_pre + stride;

    auto sequence = [&](bool timed) -> cudaError_t {
        cudaError_t x;
        k_camera_batch<<<(n + 63) / 64, 64, 0, st>>>(n, in.U, in.cam64, in.obs, anchor[0], anchor[1], anchor[2], anchor[3],
                                                     c.cam.as<float4>(), counters, r.count_work ? 16u : 4u,
                                                     c.sched.as<uint32_t>(), (uint32_t)(c.sched.bytes / 4),
                                                     c.fan_list.as<uint32_t>(), c.fan_list.bytes / 4);
        if (timed) cudaEventRecord(r.ev[0], st);
        TraceBatchArgs ta;
        ta.top_n = 0;
        ta.ws = ws;
        ta.attrs = sd.attrs;
        ta.mats = sd.mats;
        ta.U = in.U;
        ta.cam = c.cam.as<float4>();
        ta.obs = in.obs;
        ta.tile_pre = tile_pre;
        ta.n = n;
        ta.total_rays = sh.total_tiles * 32u;
        ta.tile_w = tile_w;
        ta.tile_h = tile_h;
        ta.hits = c.hits.as<float4>();
        ta.slots = c.slots.as<uint32_t>();
        ta.shadow = c.shadow.as<uint8_t>();
        ta.chunk_rays = 32u * t.chunk_tiles;
        ta.refill_lanes = t.refill_lanes;
        ta.leaf_batch = t.leaf_batch;
        ta.counter = counters + 2;
        ta.sched = c.sched.as<uint32_t>();
        ta.num_bands = t.home_pct ? (uint32_t)c.num_sms : 0u;
        ta.band_tiles = ta.num_bands ? (uint32_t)((uint64_t)sh.total_tiles * t.home_pct / 100u / ta.num_bands) : 0u;
        if (ta.band_tiles == 0) ta.num_bands = 0;
        ta.err = counters + 1;
        ta.work = work;
        uint32_t blocks = (uint32_t)c.num_sms * t.blocks_per_sm;
        uint32_t need = (uint32_t)(((uint64_t)sh.total_tiles * 32 + t.block_threads - 1) / t.block_threads);
        // Blocks beyond the resident ones would start when the work is done; a small frame's slow tiles are
        // split among the warps that have none.
        if (packet) need = (uint32_t)c.num_sms * c.fan_blocks[t.block_threads / 128u];
        if (blocks > need) blocks = need;
        const size_t smem = t.leaf_coop ? (size_t)(t.block_threads / 32) * COOP_SMEM_PER_WARP : 0;
        const bool lean = !t.leaf_coop && t.leaf_batch == 1 && t.refill_lanes == 32 && t.chunk_tiles == 1;
        if (lean) {
            // Staged top levels need the octant layout (the compact layout's kernels stage none).
            const bool oct = s.copies == 16, top = oct && t.top_levels > 0;
            ta.top_n = top ? s.top_end[t.top_levels - 1] : 0u;
            const size_t ssm = lean_stack_bytes(t) + (size_t)ta.top_n * 72u;
            if (packet) {
                FanTasks ft;
                ft.count = c.sched.as<uint32_t>();
                ft.num_shadows = ft.count + 2 * FAN_COUNTERS;
                ft.dirty = ft.count + FAN_DIRTY;
                ft.list = c.fan_list.as<uint32_t>();
                ft.lost = c.fan_lost.as<uint32_t>();
                ft.polls = c.fan_polls;
                ft.shadows = c.fan_shadows.as<uint32_t>();
                ft.helpers = (uint32_t)c.num_sms / FAN_HELPERS_PER;
                ft.waste = sh.total_tiles < FAN_SMALL_TILES ? FAN_WASTE_SMALL : FAN_WASTE;
                const uint32_t warps = t.block_threads / 32;
                if (oct) k_fan_trace<true><<<blocks, t.block_threads, warps * sizeof(FanQueue), st>>>(ta, ft);
                else k_fan_trace<false><<<blocks, t.block_threads, warps * sizeof(FanQueue), st>>>(ta, ft);
                if (shadows) {
                    ft.count += FAN_COUNTERS;
                    k_fan_shadow<<<blocks, t.block_threads, warps * sizeof(FanShadows), st>>>(ta, ft);
                }
            } else {
                launch_lean(t.stack_smem, r.count_work, oct, top, blocks, t.block_threads, ssm, st, ta);
            }
        } else if (t.leaf_coop) {
            if (r.count_work) k_trace_batch<true, true><<<blocks, t.block_threads, smem, st>>>(ta);
            else k_trace_batch<false, true><<<blocks, t.block_threads, smem, st>>>(ta);
        } else {
            if (r.count_work) k_trace_batch<true, false><<<blocks, t.block_threads, 0, st>>>(ta);
            else k_trace_batch<false, false><<<blocks, t.block_threads, 0, st>>>(ta);
        }
        if ((x = cudaGetLastError()) != cudaSuccess) return x;
        if (timed) cudaEventRecord(r.ev[1], st);
        ShadeBatchArgs sa;
        sa.s = sd;
        sa.ws = ws;
        sa.U = ta.U;
        sa.cam = ta.cam;
        sa.obs = ta.obs;
        sa.pix_pre = pix_pre;
        sa.n = n;
        sa.total_px = sh.total_px;
        sa.hits = ta.hits;
        sa.slots = ta.slots;
        sa.shadow = ta.shadow;
        sa.hdr = c.hdr.as<float4>();
        sa.hit_id = r.hit_id;
        sa.lambda = r.lambda;
        sa.tau = r.tau;
        sa.counters = counters;
        sa.work = work;
        sa.bb = bb;
        sa.stars_binned = binned ? 1u : 0u;
        uint32_t gpx = (sh.total_px + 255) / 256;
        if (r.count_work) {
            if (simple) k_shade_batch<true, true><<<gpx, 256, 0, st>>>(sa);
            else k_shade_batch<true, false><<<gpx, 256, 0, st>>>(sa);
        } else {
            if (simple) k_shade_batch<false, true><<<gpx, 256, 0, st>>>(sa);
            else k_shade_batch<false, false><<<gpx, 256, 0, st>>>(sa);
        }
        if ((x = cudaGetLastError()) != cudaSuccess) return x;
        if (timed) cudaEventRecord(r.ev[2], st);
        if (binned) {
            const size_t tiles = sh.total_star_tiles;
            if ((x = cudaMemsetAsync(c.star_count.p, 0, 2 * tiles * 4, st)) != cudaSuccess) return x;  // counts and cursors
            StarBinArgs ba;
            ba.U = sa.U;
            ba.cam = sa.cam;
            ba.obs = sa.obs;
            ba.stars = sd.stars;
            ba.n = n;
            ba.num_stars = sd.num_stars;
            ba.r = c.star_r.as<float4>();
            ba.color = c.star_color.as<float4>();
            ba.box = c.star_box.as<float4>();
            ba.bb = bb;
            ba.count = c.star_count.as<uint32_t>();
            ba.offset = c.star_offset.as<uint32_t>();
            ba.fill = ba.count + tiles;
            ba.list = c.star_list.as<uint32_t>();
            ba.list_cap = list_cap;
            const uint64_t pairs = (uint64_t)n * sd.num_stars;
            const uint32_t gb = (uint32_t)((pairs + 255) / 256);
            k_star_bin<<<gb, 256, 0, st>>>(ba);
            size_t sb = scan_bytes;
            if ((x = cub::DeviceScan::ExclusiveSum(c.star_scan.p, sb, ba.count, c.star_offset.as<uint32_t>(), (int)tiles, st)) !=
                cudaSuccess)
                return x;
            k_star_fill<<<gb, 256, 0, st>>>(ba);
            k_star_sort<<<(uint32_t)tiles, 256, STAR_SORT_CAP * 4, st>>>(ba.count, ba.offset, ba.list, list_cap, sd.num_stars);
            StarTileArgs ta2;
            ta2.s = sd;
            ta2.U = sa.U;
            ta2.cam = sa.cam;
            ta2.obs = sa.obs;
            ta2.star_pre = tile_pre + (size_t)(SR_BLOOM_LEVELS + 2) * stride;
            ta2.n = n;
            ta2.hits = sa.hits;
            ta2.slots = sa.slots;
            ta2.r = ba.r;
            ta2.color = ba.color;
            ta2.box = ba.box;
            ta2.count = ba.count;
            ta2.offset = ba.offset;
            ta2.list = ba.list;
            ta2.list_cap = list_cap;
            ta2.hdr = sa.hdr;
            ta2.bb = bb;
            k_star_tiles<<<(uint32_t)tiles * STAR_BLOCKS, 64, 0, st>>>(ta2);
            if ((x = cudaGetLastError()) != cudaSuccess) return x;
        }
        if (timed) cudaEventRecord(r.ev[3], st);
        if (r.no_image) return cudaSuccess;
        int tail = 1;  // the first level that one block per observer takes
        for (uint32_t i = 0; i < n; ++i)
            while (tail <= SR_BLOOM_LEVELS && sh.obs[i].lw[tail] * sh.obs[i].lh[tail] > BLOOM_TAIL) ++tail;
        for (int k = 1; k < tail; ++k) {
            const uint32_t* pre = tile_pre + (size_t)(1 + k) * stride;
            uint32_t tot = sh.pre[(size_t)(1 + k) * stride + n];
            k_bloom_down_batch<<<(tot + 255) / 256, 256, 0, st>>>(sa.hdr, sa.obs, pre, n, k);
        }
        if (tail <= SR_BLOOM_LEVELS) k_bloom_tail_batch<<<n, 1024, 0, st>>>(sa.hdr, sa.obs, tail);
        for (int k = std::min(tail, SR_BLOOM_LEVELS) - 1; k >= 1; --k) {
            const uint32_t* pre = tile_pre + (size_t)(1 + k) * stride;
            uint32_t tot = sh.pre[(size_t)(1 + k) * stride + n];
            k_bloom_up_batch<<<(tot + 255) / 256, 256, 0, st>>>(sa.hdr, sa.obs, pre, n, k);
        }
        const uint32_t gcomp = std::min<uint32_t>(gpx, (uint32_t)c.num_sms * 6u);
        k_bloom_composite_batch<<<gcomp, 256, 0, st>>>(sa.hdr, sa.obs, pix_pre, n, rgb, sd.tables);
        if ((x = cudaGetLastError()) != cudaSuccess) return x;
        if (timed) cudaEventRecord(r.ev[4], st);
        return cudaSuccess;
    };

    const bool timed = r.ev != nullptr;
    if (!r.use_graph || timed || r.count_work) return sequence(timed);

    uint64_t key = 0xC0FFEEull;
    key = mix(key, n);
    key = mix(key, r.cam64 ? 1 : 0);
    key = mix(key, reinterpret_cast<uintptr_t>(rgb));
    key = mix(key, reinterpret_cast<uintptr_t>(r.hit_id));
    key = mix(key, reinterpret_cast<uintptr_t>(r.lambda));
    key = mix(key, reinterpret_cast<uintptr_t>(r.tau));
    key = mix(key, reinterpret_cast<uintptr_t>(sd.geoms));
    key = mix(key, reinterpret_cast<uintptr_t>(ws.boxes));
    key = mix(key, ((uint64_t)t.block_threads << 32) | t.blocks_per_sm);
    key = mix(key, ((uint64_t)t.tile_w << 32) | t.tile_h);
    key = mix(key, ((uint64_t)t.chunk_tiles << 40) | ((uint64_t)t.refill_lanes << 24) | ((uint64_t)t.leaf_batch << 8) |
                       t.leaf_coop);
    key = mix(key, t.home_pct);
    key = mix(key, ((uint64_t)t.stack_smem << 32) | t.top_levels);
    key = mix(key, (packet ? 1u : 0u) | (shadows ? 2u : 0u));
    key = mix(key, binned ? 0x5354ull : 0ull);
    key = mix(key, (simple ? 0x51ull : 0ull) | (r.no_image ? 0x100ull : 0ull));
    for (auto& o : sh.obs) key = mix(key, ((uint64_t)o.width << 32) | o.height);
    auto it = c.graphs.find(key);
    if (it == c.graphs.end()) {
        if (c.graphs.size() > 64) drop_graphs();
        GraphEntry g;
        if ((e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return sequence(false);
        cudaError_t se = sequence(false);
        e = cudaStreamEndCapture(st, &g.graph);
        if (se != cudaSuccess || e != cudaSuccess) {
            if (g.graph) cudaGraphDestroy(g.graph);
            cudaGetLastError();
            return sequence(false);
        }
        if ((e = cudaGraphInstantiate(&g.exec, g.graph, 0)) != cudaSuccess) {
            cudaGraphDestroy(g.graph);
            cudaGetLastError();
            return sequence(false);
        }
        it = c.graphs.emplace(key, g).first;
    }
    return cudaGraphLaunch(it->second.exec, st);
}

// ---------------------------------------------------------------------------------------------
// The gradient of the image loss (sr_adjoint.cuh).
// ---------------------------------------------------------------------------------------------
// Whether kernels on the current device can read `bytes` at `p` as float4: aligned, memory of this device, and all
// of it within one allocation.
static bool readable_here(const void* p, size_t bytes) {
    typedef int (*RangeFn)(unsigned long long*, size_t*, unsigned long long);  // cuMemGetAddressRange
    static const RangeFn range = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<RangeFn>(f);
    }();
    const unsigned long long at = reinterpret_cast<unsigned long long>(p);
    cudaPointerAttributes a{};
    int dev = 0;
    unsigned long long base = 0;
    size_t size = 0;
    if (at % 16 != 0 || !range || cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == dev && range(&base, &size, at) == 0 && at - base <= size &&
           bytes <= size - (at - base);
}

cudaError_t fast_adjoint(FastCtx& c, FastScene& s, const SrTuning& t, const SceneDev& sd, const double anchor[4],
                         const BBConst& bb, uint32_t* counters, const SrGpuUniforms& u, const SrCameraF64& cam,
                         const float* target, uint32_t level, bool frozen, uint32_t row0, uint32_t row1,
                         double out[10], cudaStream_t st) {
    const uint32_t W = u.size[0], H = u.size[1];
    cudaError_t e;
    if (frozen) {
        if (!c.adj_valid || c.adj_w != W || c.adj_h != H || c.adj_geoms != sd.geoms || c.adj_level != level ||
            c.adj_r0 != row0 || c.adj_r1 != row1)
            return cudaErrorInvalidValue;
    } else {
        c.adj_valid = false;
    }
    // Pyramid geometry of the loss levels 0..level.
    uint32_t lw[8], lh[8];
    size_t loff[9];
    lw[0] = W;
    lh[0] = H;
    loff[0] = 0;
    for (uint32_t k = 1; k <= level; ++k) {
        lw[k] = (lw[k - 1] + 1) / 2;
        lh[k] = (lh[k - 1] + 1) / 2;
    }
    for (uint32_t k = 0; k <= level; ++k) loff[k + 1] = loff[k] + (size_t)lw[k] * lh[k];
    const size_t npx = (size_t)W * H;
    if ((e = c.adj_pyr.ensure(2 * loff[level + 1] * sizeof(float4))) != cudaSuccess) return e;
    float4* pyr = c.adj_pyr.as<float4>();  // image levels 0..level
    float4* tpyr = pyr + loff[level + 1];  // target levels 0..level
    // The target is the caller's. Kernels read it where it lies when they can; else it is copied, which takes any
    // float address and refuses memory that is not there. Copied always, a gradient took 550 against 546 us
    // (320x200, level 3) and 839 against 829 (1280x800, level 0).
    const float4* tgt0 = reinterpret_cast<const float4*>(target);
    if (!readable_here(target, npx * sizeof(float4))) {
        if ((e = cudaMemcpyAsync(tpyr, target, npx * sizeof(float4), cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
        tgt0 = tpyr;
    }
    if (!frozen) {
        // The forward frame: hits, shadow results, star lists and the HDR image the loss compares.
        BatchRequest br{};
        br.n = 1;
        br.u = &u;
        br.cam64 = &cam;
        br.use_graph = true;
        br.no_image = true;
        if ((e = fast_render_batch(c, s, t, sd, anchor, bb, counters, br, st)) != cudaSuccess) return e;
    }
    const uint32_t tx16 = (W + STAR_TILE - 1) / STAR_TILE, ty16 = (H + STAR_TILE - 1) / STAR_TILE;
    const uint32_t tiles = tx16 * ty16;
    const bool stars_on = sd.num_stars > 0 && stars_binned_for(u, sd.num_stars);
    const uint32_t rblocks = (uint32_t)((npx + 255) / 256);
    // The forward pass's: the buffer may be larger from a batch of more observers, its entries beyond unwritten.
    const size_t list_cap = stars_on ? c.batch_list_cap : 0;
    if ((e = c.adj_cam.ensure(sizeof(DCam))) != cudaSuccess) return e;
    if ((e = c.adj_partials.ensure((size_t)std::max(tiles, rblocks) * ADJ_SLOTS * sizeof(double))) != cudaSuccess) return e;
    if ((e = c.adj_out.ensure(2 * ADJ_SLOTS * sizeof(double))) != cudaSuccess) return e;
    if ((e = c.adj_weight.ensure(2 * npx * 3 * sizeof(double))) != cudaSuccess) return e;
    if ((e = c.adj_grid.ensure(npx)) != cudaSuccess) return e;
    if ((e = c.adj_hdr.ensure(npx * sizeof(float4))) != cudaSuccess) return e;
    if (stars_on && (e = c.adj_stars.ensure((size_t)sd.num_stars * ADJ_STAR * sizeof(float))) != cudaSuccess) return e;
    if (stars_on && (e = c.adj_star_sum.ensure(npx * ADJ_SUM * sizeof(float))) != cudaSuccess) return e;
    if (stars_on && (e = c.adj_star_n.ensure(npx * 4)) != cudaSuccess) return e;
    if (stars_on && (e = c.adj_pass.ensure(list_cap * 32)) != cudaSuccess) return e;
    double* g0 = c.adj_weight.as<double>();
    double* g1 = g0 + npx * 3;
    const dim3 b2(16, 16);
    // The loss at the chosen level of `image` against the target, and (gradient mode) its weights
    // on the full image.
    auto loss_pass = [&](const void* image) -> cudaError_t {
        // Level 0 is the image and the target themselves.
        auto at = [&](const float4* level0, float4* levels, uint32_t k) { return k ? (const float4*)(levels + loff[k]) : level0; };
        const float4* img0 = reinterpret_cast<const float4*>(image);
        for (uint32_t k = 1; k <= level; ++k) {
            const dim3 g2((lw[k] + 15) / 16, (lh[k] + 15) / 16, 2);
            k_adj_down<<<g2, b2, 0, st>>>(at(img0, pyr, k - 1), at(tgt0, tpyr, k - 1), lw[k - 1], lh[k - 1], pyr + loff[k],
                                         tpyr + loff[k], lw[k], lh[k]);
        }
        const size_t nl = (size_t)lw[level] * lh[level];
        double* gl = (level % 2 == 0) ? g0 : g1;  // ends in g0 after `level` transposes
        const uint32_t lblocks = (uint32_t)((nl + 255) / 256);
        k_adj_residual<<<lblocks, 256, 0, st>>>(at(img0, pyr, level), at(tgt0, tpyr, level), (uint32_t)nl, lw[level], row0,
                                                 row1, gl, c.adj_partials.as<double>());
        k_adjoint_reduce<<<ADJ_SLOTS, 256, 0, st>>>(c.adj_partials.as<double>(), lblocks, c.adj_out.as<double>() + ADJ_SLOTS);
        for (uint32_t k = level; k >= 1; --k) {
            double* src = (k % 2 == 0) ? g0 : g1;
            double* dst = (k % 2 == 0) ? g1 : g0;
            const dim3 g2((lw[k - 1] + 15) / 16, (lh[k - 1] + 15) / 16);
            k_adj_up<<<g2, b2, 0, st>>>(src, lw[k], lh[k], dst, lw[k - 1], lh[k - 1]);
        }
        return cudaGetLastError();
    };
    if (!frozen) {
        if ((e = loss_pass(c.hdr.p)) != cudaSuccess) return e;
        if (stars_on && (e = cudaMemsetAsync(c.adj_pass.p, 0, list_cap * 32, st)) != cudaSuccess) return e;
    }
    // The duals of the camera and of the stars' cone events, then the pixels.
    k_adjoint_camera<<<1, 1, 0, st>>>(cam, anchor[0], anchor[1], anchor[2], anchor[3], c.adj_cam.as<DCam>());
    if (stars_on)
        k_adjoint_stars<<<(sd.num_stars + 127) / 128, 128, 0, st>>>(sd.stars, sd.num_stars, c.star_box.as<float4>(),
                                                                  c.adj_cam.as<DCam>(), bb, c.adj_stars.as<float>());
    AdjointArgs a;
    a.s = sd;
    a.U = c.batch_U;
    a.obs = c.batch_obs;
    a.star_pre = nullptr;
    a.dcam = c.adj_cam.as<DCam>();
    a.hits = c.hits.as<float4>();
    a.slots = c.slots.as<uint32_t>();
    a.shadow = c.shadow.as<uint8_t>();
    a.star = stars_on ? c.adj_stars.as<float>() : nullptr;
    a.star_box = stars_on ? c.star_box.as<float4>() : nullptr;
    a.star_sum = stars_on ? c.adj_star_sum.as<float>() : nullptr;
    a.star_n = stars_on ? c.adj_star_n.as<uint32_t>() : nullptr;
    a.count = stars_on ? c.star_count.as<uint32_t>() : nullptr;
    a.offset = stars_on ? c.star_offset.as<uint32_t>() : nullptr;
    a.list = stars_on ? c.star_list.as<uint32_t>() : nullptr;
    a.list_cap = (uint32_t)list_cap;
    a.stars_on = stars_on ? 1u : 0u;
    a.hdr_fwd = c.hdr.as<float4>();
    a.weight = g0;
    a.partials = c.adj_partials.as<double>();
    a.bb = bb;
    a.grid = c.adj_grid.as<uint8_t>();
    a.pass = stars_on ? c.adj_pass.as<uint32_t>() : nullptr;
    a.frozen = frozen ? 1u : 0u;
    a.hdr_out = c.adj_hdr.as<float4>();
    // The band's pixel rows (level-`level` rows [row0, row1) cover rows row0 * 2^level on) and the
    // 16x16 tiles over them.
    a.y0 = std::min(H, row0 << level);
    a.y1 = std::min(H, row1 << level);
    const uint32_t ty0 = a.y0 / STAR_TILE, ty1 = (a.y1 + STAR_TILE - 1) / STAR_TILE;
    a.tile0 = ty0 * tx16;
    const uint32_t band_tiles = (ty1 - ty0) * tx16;
    if (band_tiles && stars_on) k_adjoint_star_sums<<<band_tiles * ADJ_STAR_BLOCKS, 256, 0, st>>>(a);
    if (band_tiles) k_adjoint_pixels<<<band_tiles, 256, 0, st>>>(a);
    k_adjoint_reduce<<<ADJ_SLOTS, 256, 0, st>>>(a.partials, band_tiles, c.adj_out.as<double>());
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (frozen && (e = loss_pass(c.adj_hdr.p)) != cudaSuccess) return e;
    double both[2 * ADJ_SLOTS];
    if ((e = cudaMemcpyAsync(both, c.adj_out.p, sizeof(both), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    for (int k = 0; k < ADJ_SLOTS; ++k) out[k] = frozen ? 0.0 : both[k];
    out[0] = both[ADJ_SLOTS];  // the loss, from the residual pass
    if (!frozen) {
        c.adj_valid = true;
        c.adj_w = W;
        c.adj_h = H;
        c.adj_geoms = sd.geoms;
        c.adj_level = level;
        c.adj_r0 = row0;
        c.adj_r1 = row1;
    }
    return cudaSuccess;
}

}  // namespace srk
