// The fan layout and the packet walk over it (included by sr_fast.cu after sr_traverse.cuh).
//
// A warp's rays walk the tree together. Over binary nodes (two boxes per step, every lane testing the same
// two against its own ray) the 8-frame launch of the 7.9M-tet workload was bound by issue: 17.9k warp
// instructions per 32-pixel tile, 60% of them box tests and most of the rest record tests that no ray
// passes. Neighbouring pixels' rays share their origin and differ little in direction, so one test against
// the interval of a tile's directions stands for all of them, and the lanes can test 32 DIFFERENT boxes, or
// 32 different records, at once: per 8x8 tile 25 to 45 fan nodes and 5 to 20 batches of records, of which
// 2 to 13 records are left to test against the rays. The fan layout regroups the reference's tree for that:
// one fan node holds up to 32 subtrees or leaves of it, box and reference per lane (1152 bytes; 173 MB for
// the 7.9M-tet scene). Measured on that launch: 9.57 ms -> 2.86 ms at the same clocks, bound by issue and
// fixed latencies still (47% of issue slots, 20 warps per SM).
#pragma once

namespace srk {

constexpr uint32_t FAN = 32;            // entries of a fan node
constexpr uint32_t FAN_LEVELS = 16;     // fan nodes on a path (a tree that needs more has no fan layout)
constexpr uint32_t FAN_EMPTY = REF_LEAF;  // a leaf of no records: an unused entry
constexpr uint32_t FAN_NONE = 0xFFFFFFFFu;
constexpr int FAN_RAYS = 2;             // rays per lane of a closest-hit walk

// ---------------------------------------------------------------------------------------------
// Build. Level by level from the leaves: the units of level 0 are the leaves; a unit of the next
// level is a maximal subtree holding at most 32 units of the one below (the counts climb the parent
// links, the last of a node's two children to arrive carrying the sum on). A subtree of one unit is that
// unit; one of 2 to 32 becomes a fan node. Cutting from the leaves keeps the fan nodes at the
// bottom, where nearly all are, well filled (20 entries on average on the 7.9M-tet scene); cutting every
// five levels from the root leaves whatever remains there.
// ---------------------------------------------------------------------------------------------
struct FanCounts {
    uint32_t fans, root_total;
    uint32_t conflict;                       // a child claimed twice, or a box that does not hold its children's
    uint32_t units[FAN_LEVELS + 2];          // per level
    uint32_t reached[FAST_MAX_DEPTH + 2];    // nodes per depth (the marking)
};

// parent[child] = i for both children of every internal node (of every reached node, when `reach` is
// given). A child claimed twice sets `conflict`, and so does a box that does not hold its children's: a fan node
// leaves out the boxes between it and its entries, which only hides nothing from a ray where boxes are nested
// (as every builder here makes them; an uploaded tree need not). Free room of an arena holds stale nodes whose
// links may point into the live tree: on a conflict the build marks what the root reaches and looks again.
__global__ void k_fan_parents(const SrGpuNode* nodes, uint32_t n, const uint32_t* reach, uint32_t* parent, FanCounts* fc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || nodes[i].count != 0 || (reach && !reach[i])) return;
    const uint32_t c[2] = {nodes[i].left, nodes[i].right_or_first};
    for (int k = 0; k < 2; ++k) {
        bool sound = c[k] < n && c[k] != 0 && atomicExch(parent + c[k], i) == FAN_NONE;
        for (int a = 0; a < 4 && sound; ++a)  // false for a NaN
            sound = nodes[c[k]].min[a] >= nodes[i].min[a] && nodes[c[k]].max[a] <= nodes[i].max[a];
        if (!sound) fc->conflict = 1;
    }
}

// One level of the breadth-first marking: the nodes of depth `level`, which lie in the queue behind those of
// the depths above, put their children behind them.
__global__ void k_fan_reach(const SrGpuNode* nodes, uint32_t n, uint32_t* reach, uint32_t* queue, uint32_t level,
                            FanCounts* fc) {
    uint32_t begin = 0;
    for (uint32_t l = 0; l < level; ++l) begin += fc->reached[l];
    const uint32_t count = level ? fc->reached[level] : 1u;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t i = level ? queue[begin + q] : 0u;
        if (level == 0) fc->reached[0] = 1;
        reach[i] = 1;
        if (nodes[i].count != 0) continue;
        const uint32_t at = begin + count + atomicAdd(&fc->reached[level + 1], 2u);
        if (at + 1 < n) {
            queue[at] = nodes[i].left;
            queue[at + 1] = nodes[i].right_or_first;
        }
    }
}

// Appends `v` to list[*count ...] for the lanes with `yes` (one atomic per warp); returns its place.
__device__ __forceinline__ uint32_t fan_append(bool yes, uint32_t v, uint32_t* list, uint32_t* count) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, yes), lane = threadIdx.x & 31u;
    uint32_t at = 0;
    if (m && lane == 0) at = atomicAdd(count, (uint32_t)__popc(m));
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (yes) list[at] = v;
    return at;
}

// The leaves are the units of level 0.
__global__ void k_fan_leaves(const SrGpuNode* nodes, uint32_t n, const uint32_t* reach, uint32_t* uref, uint32_t* units,
                             FanCounts* fc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool leaf = i < n && nodes[i].count != 0 && (!reach || reach[i]);
    fan_append(leaf, i, units, &fc->units[0]);
    if (leaf) uref[i] = pack_leaf(nodes[i].right_or_first, nodes[i].count);
}

// total[v] = the units below v where that is at most 32, else 0; acc: what the first child brought.
__global__ void k_fan_climb(const uint32_t* units, uint32_t level, const uint32_t* parent, uint32_t* acc, uint32_t* total,
                            const FanCounts* fc) {
    const uint32_t num_units = fc->units[level];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < num_units; i += gridDim.x * blockDim.x) {
        uint32_t v = units[i], c = 1;
        total[v] = 1;
        for (uint32_t up = 0; v != 0 && up <= FAST_MAX_DEPTH; ++up) {
            const uint32_t p = parent[v];
            if (p == FAN_NONE) break;
            const uint32_t other = atomicAdd(acc + p, c);
            if (other == 0) break;
            c += other;
            if (c > FAN) break;
            total[p] = c;
            v = p;
        }
    }
}

// The units of the next level: the topmost counted nodes. Those of more than one unit become fan
// nodes, numbered behind the ones of the levels below.
__global__ void k_fan_units(uint32_t n, uint32_t level, const uint32_t* parent, const uint32_t* total, uint32_t* uref,
                            uint32_t* units, uint32_t* fan_root, FanCounts* fc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool unit = i < n && total[i] != 0 && (i == 0 || parent[i] == FAN_NONE || total[parent[i]] == 0);
    fan_append(unit, i, units, &fc->units[level + 1]);
    if (i == 0) fc->root_total = total[0];
    const bool fan = unit && total[i] > 1;
    const uint32_t at = fan_append(fan, i, fan_root, &fc->fans);
    if (fan) uref[i] = at;
}

// One warp per fan node: the entries below its root, in the reference's order, down to the units of
// the level below (the topmost nodes under the root that have a reference).
__global__ void __launch_bounds__(128) k_fan_fill(const SrGpuNode* nodes, uint32_t fans, const uint32_t* fan_root,
                                                  const uint32_t* uref, float4* box, uint32_t* ref) {
    __shared__ uint32_t next[4][FAN];
    const uint32_t w = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (w >= fans) return;
    uint32_t* nx = next[threadIdx.x >> 5];
    uint32_t node = fan_root[w], count = 1;
    for (uint32_t step = 0; step <= FAST_MAX_DEPTH; ++step) {
        const bool open = lane < count && (step == 0 || uref[node] == FAN_NONE);
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, open);
        if (!m) break;
        const uint32_t at = lane + (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (lane < count && at < FAN) nx[at] = open ? nodes[node].left : node;
        if (open && at + 1u < FAN) nx[at + 1u] = nodes[node].right_or_first;
        count = min(count + (uint32_t)__popc(m), FAN);
        __syncwarp();
        node = nx[lane];
        __syncwarp();
    }
    const bool used = lane < count;
    float4 lo = make_float4(3e37f, 3e37f, 3e37f, 3e37f), hi = neg4(lo);
    uint32_t r = FAN_EMPTY;
    if (used) {
        const SrGpuNode& nd = nodes[node];
        lo = make_float4(nd.min[0], nd.min[1], nd.min[2], nd.min[3]);
        hi = make_float4(nd.max[0], nd.max[1], nd.max[2], nd.max[3]);
        r = uref[node];
    }
    box[(size_t)w * 64u + lane] = lo;
    box[(size_t)w * 64u + 32u + lane] = hi;
    ref[(size_t)w * 32u + lane] = r;
}

static size_t fan_scratch(uint32_t n) { return 6 * (size_t)n * 4 + sizeof(FanCounts); }

// Builds the layout (s.fan_*); s.fan_levels stays 0 where there is none: memory short, a tree that needs more than
// FAN_LEVELS levels, or boxes that are not nested.
static cudaError_t fan_build(FastScene& s, const SrGpuNode* nodes, uint32_t n, cudaStream_t st) {
    s.fan_levels = 0;
    if (s.scratch.ensure_grow(fan_scratch(n)) != cudaSuccess) {
        cudaGetLastError();
        return cudaStreamSynchronize(st);
    }
    uint32_t* scratch = s.scratch.as<uint32_t>();
    uint32_t *parent = scratch, *acc = parent + n, *total = acc + n, *uref = total + n, *units = uref + n, *roots = units + n;
    FanCounts* fc = reinterpret_cast<FanCounts*>(roots + n);
    const uint32_t blocks = (n + 255) / 256;
    FanCounts h{};
    const uint32_t* reach = nullptr;
    cudaError_t e;
    auto look = [&]() -> cudaError_t {
        cudaError_t x = cudaMemcpyAsync(&h, fc, offsetof(FanCounts, units), cudaMemcpyDeviceToHost, st);
        return x == cudaSuccess ? cudaStreamSynchronize(st) : x;
    };
    if ((e = cudaMemsetAsync(parent, 0xFF, (size_t)n * 4, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(uref, 0xFF, (size_t)n * 4, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(fc, 0, sizeof(FanCounts), st)) != cudaSuccess) return e;
    k_fan_parents<<<blocks, 256, 0, st>>>(nodes, n, nullptr, parent, fc);
    if ((e = look()) != cudaSuccess) return e;
    if (h.conflict) {
        if ((e = cudaMemsetAsync(parent, 0xFF, (size_t)n * 4, st)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(fc, 0, sizeof(FanCounts), st)) != cudaSuccess) return e;
        // The marks lie in `roots`, which the fan numbering writes only after the leaves are listed; `total` is
        // the queue.
        if ((e = cudaMemsetAsync(roots, 0, (size_t)n * 4, st)) != cudaSuccess) return e;
        for (uint32_t l = 0; l < s.depth && l <= FAST_MAX_DEPTH; ++l)
            k_fan_reach<<<148, 256, 0, st>>>(nodes, n, roots, total, l, fc);
        reach = roots;
        k_fan_parents<<<blocks, 256, 0, st>>>(nodes, n, reach, parent, fc);
    }
    k_fan_leaves<<<blocks, 256, 0, st>>>(nodes, n, reach, uref, units, fc);
    // As many levels as a tree of this size usually has before the first look (each is a few launches, and a
    // look waits for them), then one by one.
    uint32_t levels = 0, usual = 1;
    for (uint64_t k = n / 2; k > FAN; k /= 18) ++usual;
    do {
        if ((e = cudaMemsetAsync(acc, 0, (size_t)n * 8, st)) != cudaSuccess) return e;  // acc and total
        k_fan_climb<<<std::min(blocks, 148u * 16u), 256, 0, st>>>(units, levels, parent, acc, total, fc);
        k_fan_units<<<blocks, 256, 0, st>>>(n, levels, parent, total, uref, units, roots, fc);
        ++levels;
        if (levels < usual && levels < FAN_LEVELS) continue;
        if ((e = look()) != cudaSuccess) return e;
        if (h.conflict) return cudaSuccess;  // not a tree of nested boxes: no fan layout
    } while (h.root_total == 0 && levels < FAN_LEVELS);
    if (h.root_total == 0) return cudaSuccess;
    if (s.fan_box.ensure_grow((size_t)h.fans * 64 * sizeof(float4)) != cudaSuccess ||
        s.fan_ref.ensure_grow((size_t)h.fans * 32 * 4) != cudaSuccess) {
        cudaGetLastError();
        s.fan_box.release();
        s.fan_ref.release();
        return cudaSuccess;
    }
    k_fan_fill<<<(h.fans + 3) / 4, 128, 0, st>>>(nodes, h.fans, roots, uref, s.fan_box.as<float4>(), s.fan_ref.as<uint32_t>());
    if ((e = cudaMemcpyAsync(&s.fan_root, uref, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    s.fan_levels = levels;
    s.num_fans = h.fans;
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// The walk: bounds of a warp's rays, and the tests of a box and of a record against them.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t FULL_WARP = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t redux_min(uint32_t v) { return __reduce_min_sync(FULL_WARP, v); }
__device__ __forceinline__ uint32_t redux_max(uint32_t v) { return __reduce_max_sync(FULL_WARP, v); }
// The largest |v| over the lanes `in`.
__device__ __forceinline__ float redux_abs(bool in, float v) {
    return __uint_as_float(redux_max(in ? __float_as_uint(fabsf(v)) : 0u));
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 pa, pb, pc, pr;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\tmov.b64 pc, {%6, %7};\n\t"
        "fma.rn.f32x2 pr, pa, pb, pc;\n\tmov.b64 {%0, %1}, pr;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
// A dot product for bounds (fused, any order: every use carries a margin).
__device__ __forceinline__ float dot_b(float4 a, float4 b) {
    const float2 p = fma2(f2(a.z, a.w), f2(b.z, b.w), mul2(f2(a.x, a.y), f2(b.x, b.y)));
    return p.x + p.y;
}
__device__ __forceinline__ float l1_b(float4 a) { return (fabsf(a.x) + fabsf(a.y)) + (fabsf(a.z) + fabsf(a.w)); }
__device__ __forceinline__ float max_b(float4 a) { return fmaxf(max3f(fabsf(a.x), fabsf(a.y), fabsf(a.z)), fabsf(a.w)); }
__device__ __forceinline__ float4 abs_b(float4 a) { return make_float4(fabsf(a.x), fabsf(a.y), fabsf(a.z), fabsf(a.w)); }
__device__ __forceinline__ float4 shfl4(float4 v, uint32_t lane) {
    return make_float4(__shfl_sync(FULL_WARP, v.x, lane), __shfl_sync(FULL_WARP, v.y, lane),
                       __shfl_sync(FULL_WARP, v.z, lane), __shfl_sync(FULL_WARP, v.w, lane));
}

// What stands for the rays of one warp, in shared memory (read back as broadcasts).
// near_p .. far_n: per axis the smallest and largest of the positive inverse directions and of the
// negative ones (0 where there is none).
struct FanDirs {
    float4 near_p, near_n, far_p, far_n;
};
// Rays of one origin -no: every direction is mid + a du + b dv + c with |a|, |b| <= 1 and no component of
// c above res.
struct FanRays {
    FanDirs dirs;
    float4 mid, du, dv, no;
    float res, o_max, d_max, pad;  // the largest components of the origin and of the directions
};
// The records waiting to be tested against the rays: per entry the record and its leaf's box (the index
// of its minimum in fan_box).
constexpr uint32_t FAN_QUEUE = 128;
static __device__ __noinline__ float4 inverse(float4 d) { return v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w)); }
struct FanQueue {
    FanRays rays;
    uint2 queue[FAN_QUEUE];
};
// Rays of many origins: the origins lie in the box [-no_lo, -no_hi] and are o + a ou + b ov + c', |c'| <=
// ores, with the a and b of the direction.
struct FanShadows {
    FanDirs dirs;
    float4 mid, du, dv, res;
    float4 no_lo, no_hi, o, ou, ov, ores;
};

// The smallest and largest positive and negative inverse directions of one axis over the lanes `in`.
__device__ __forceinline__ void fan_axis(bool in, float inv, float* near_p, float* near_n, float* far_p, float* far_n) {
    const uint32_t mag = __float_as_uint(fabsf(inv));
    const bool pos = in && inv > 0.0f, neg = in && inv < 0.0f;
    const uint32_t lp = redux_min(pos ? mag : FAN_NONE), ln = redux_min(neg ? mag : FAN_NONE);
    *near_p = lp == FAN_NONE ? 0.0f : __uint_as_float(lp);
    *near_n = ln == FAN_NONE ? 0.0f : -__uint_as_float(ln);
    *far_p = __uint_as_float(redux_max(pos ? mag : 0u));
    *far_n = -__uint_as_float(redux_max(neg ? mag : 0u));
}
__device__ __forceinline__ FanDirs fan_dirs(bool in, float4 inv) {
    FanDirs r;
    fan_axis(in, inv.x, &r.near_p.x, &r.near_n.x, &r.far_p.x, &r.far_n.x);
    fan_axis(in, inv.y, &r.near_p.y, &r.near_n.y, &r.far_p.y, &r.far_n.y);
    fan_axis(in, inv.z, &r.near_p.z, &r.near_n.z, &r.far_p.z, &r.far_n.z);
    fan_axis(in, inv.w, &r.near_p.w, &r.near_n.w, &r.far_p.w, &r.far_n.w);
    return r;
}

// Entry and exit of a box for all the rays: none of them (origins in [-no_lo, -no_hi]) enters it before
// `en` or leaves it after `ex`, as slab_interval computes them for the ray, bit for bit: rounding is
// monotonic in the origin and in each factor of one sign. Against a positive direction the near corner
// is bmin, and (bmin - o) times the smallest inverse direction is at most the ray's product where that is
// positive (negative ones are below t_min > 0 and do not count); against a negative one it is bmax. A
// sign that no ray has on an axis gives 0 there, which bounds nothing. The far side likewise.
__device__ __forceinline__ void fan_interval(float4 bmin, float4 bmax, float4 no_lo, float4 no_hi, const FanDirs& f, float t_min,
                                             float t_max, float* en, float* ex) {
    const float2 l01 = add2(f2(bmin.x, bmin.y), f2(no_lo.x, no_lo.y)), l23 = add2(f2(bmin.z, bmin.w), f2(no_lo.z, no_lo.w));
    const float2 h01 = add2(f2(bmax.x, bmax.y), f2(no_hi.x, no_hi.y)), h23 = add2(f2(bmax.z, bmax.w), f2(no_hi.z, no_hi.w));
    const float4 np = f.near_p, nn = f.near_n, fp = f.far_p, fn = f.far_n;
    const float2 a01 = mul2(l01, f2(np.x, np.y)), a23 = mul2(l23, f2(np.z, np.w));
    const float2 b01 = mul2(h01, f2(nn.x, nn.y)), b23 = mul2(h23, f2(nn.z, nn.w));
    *en = max3f(max3f(max3f(t_min, a01.x, b01.x), a01.y, b01.y), max3f(a23.x, b23.x, a23.y), b23.y);
    const float2 c01 = mul2(h01, f2(fp.x, fp.y)), c23 = mul2(h23, f2(fp.z, fp.w));
    const float2 d01 = mul2(l01, f2(fn.x, fn.y)), d23 = mul2(l23, f2(fn.z, fn.w));
    *ex = min3f(min3f(t_max, fmaxf(c01.x, d01.x), fmaxf(c01.y, d01.y)), fmaxf(c23.x, d23.x), fmaxf(c23.y, d23.y));
}

// Whether some of the rays (one origin) may hit the record at `g` before t_max; if so *lam is at most
// the hit parameter. Lanes test different records.
//
// A ray d meets the record's hyperplane at lambda = num / (n . d), num = n . (v0 - o) shared by the
// rays, and its barycentric coordinate u there is U + lambda (B1 . d), U = B1 . (o - v0). Times the
// denominator, the test u >= -1e-5 reads (U + 1e-5)(n . d) + num (B1 . d) >= 0: linear in d, so its
// largest value over the rays is its value at `mid` plus the magnitudes along du, dv and the rest. The
// same for v, w and 1 - u - v - w. What a float test can differ by from these is bounded by
// 2^-18 |B|_1 |n|_1 D (|o| + |v0 - o| + lambda D), D the largest direction component: the products and
// sums of the test and of this function round at 2^-24 of such terms at most 36 times. Every comparison rejects
// only where it holds: a record with a NaN or an infinity goes on to the rays' own tests, whose comparisons a NaN
// passes likewise.
__device__ __forceinline__ bool fan_record(const float4* g, const FanRays& f, float t_max, float* lam) {
    const float4 n = __ldg(g + 1), v0 = __ldg(g), B1 = __ldg(g + 2), B2 = __ldg(g + 3), B3 = __ldg(g + 4);
    const float4 mid = f.mid, du = f.du, dv = f.dv, no = f.no;
    const float res = f.res, d_max = f.d_max;
    const float2 w01 = add2(f2(v0.x, v0.y), f2(no.x, no.y)), w23 = add2(f2(v0.z, v0.w), f2(no.z, no.w));
    const float4 w = make_float4(w01.x, w01.y, w23.x, w23.y);
    const float w_max = max_b(w), n1 = l1_b(n);
    float num = dot_b(n, w), nc = dot_b(n, mid), nu = dot_b(n, du), nv = dot_b(n, dv);
    const float nr = n1 * res;
    const float spread = fabsf(nu) + fabsf(nv) + nr;
    *lam = 0.0f;
    const float den_lo = fabsf(nc) - spread;
    const bool edge = !(den_lo > 0.0f);  // the rays see the record edge on: no bound
    const float sgn = nc < 0.0f ? -1.0f : 1.0f;
    num *= sgn;
    nc *= sgn;
    nu *= sgn;
    nv *= sgn;
    const float num_err = 1e-6f * n1 * w_max;
    const float lo = __fdividef(fmaxf(num - num_err, 0.0f), nc + spread) * 0.9999f;
    if (!edge) *lam = lo;
    const float hi = fminf(__fdividef(num + num_err, den_lo) * 1.0001f, t_max);
    const float err = 3.8147e-6f * n1 * d_max * (f.o_max + w_max + hi * d_max);
    bool may = !(num < -num_err) && !(lo >= t_max);  // not behind the rays, nor beyond their hits
    float us = 0.0f, bc = 0.0f, bu = 0.0f, bv = 0.0f, b1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 B = k == 0 ? B1 : (k == 1 ? B2 : B3);
        const float U = 1e-5f - dot_b(B, w), c = dot_b(B, mid), u = dot_b(B, du), v = dot_b(B, dv), l1 = l1_b(B);
        const float top = fmaf(U, nc, num * c) + fabsf(fmaf(U, nu, num * u)) + fabsf(fmaf(U, nv, num * v)) +
                          fmaf(fabsf(U), nr, fmaf(fabsf(num), res, err) * l1);
        may = may && !(top < 0.0f);
        us += U;
        bc += c;
        bu += u;
        bv += v;
        b1 += l1;
    }
    const float S = 1.00005f - us;  // 1 + 1e-5 - u - v - w (each U carries 1e-5), and the rounding of the three sums
    const float top = fmaf(S, nc, -num * bc) + fabsf(fmaf(S, nu, -num * bu)) + fabsf(fmaf(S, nv, -num * bv)) +
                      fmaf(fabsf(S), nr, fmaf(fabsf(num), res, err) * b1);
    return edge || (may && !(top < 0.0f));
}

// A quantity that is affine over the rays up to a remainder: c + a u + b v + e, |a|, |b| <= 1, |e| <= r.
struct FanAff {
    float c, u, v, r;
};
__device__ __forceinline__ float aff_top(const FanAff& p) { return p.c + fabsf(p.u) + fabsf(p.v) + p.r; }
// The largest value of p q + s t: the products' affine part, and a bound of the rest.
__device__ __forceinline__ float aff_top2(const FanAff& p, const FanAff& q, const FanAff& s, const FanAff& t) {
    const float pl = fabsf(p.u) + fabsf(p.v), ql = fabsf(q.u) + fabsf(q.v), sl = fabsf(s.u) + fabsf(s.v), tl = fabsf(t.u) + fabsf(t.v);
    const float c = fmaf(p.c, q.c, s.c * t.c);
    const float u = fmaf(p.c, q.u, fmaf(p.u, q.c, fmaf(s.c, t.u, s.u * t.c)));
    const float v = fmaf(p.c, q.v, fmaf(p.v, q.c, fmaf(s.c, t.v, s.v * t.c)));
    const float rest = fmaf(pl, ql, fmaf(fabsf(p.c) + pl + p.r, q.r, p.r * (fabsf(q.c) + ql))) +
                       fmaf(sl, tl, fmaf(fabsf(s.c) + sl + s.r, t.r, s.r * (fabsf(t.c) + tl)));
    return c + fabsf(u) + fabsf(v) + rest;
}

// fan_record for rays of many origins: num, U and the products are affine over the rays too, up to
// bounded remainders; the same inequalities and error bound.
__device__ __forceinline__ bool fan_record_any(const float4* g, const FanShadows& f, float o_max, float d_max, float t_max) {
    const float4 n = __ldg(g + 1), v0 = __ldg(g);
    const float4 w = sub4(v0, f.o);
    const float w_max = max_b(w) + max_b(f.ou) + max_b(f.ov) + max_b(f.ores), n1 = l1_b(n);
    const float4 an = abs_b(n);
    FanAff num{dot_b(n, w), -dot_b(n, f.ou), -dot_b(n, f.ov), dot_b(an, f.ores) + 1e-6f * n1 * w_max};
    FanAff den{dot_b(n, f.mid), dot_b(n, f.du), dot_b(n, f.dv), dot_b(an, f.res) + 1e-6f * n1 * d_max};
    const float spread = fabsf(den.u) + fabsf(den.v) + den.r;
    const float den_lo = fabsf(den.c) - spread;
    if (!(den_lo > 0.0f)) return true;
    if (den.c < 0.0f) {
        num.c = -num.c;
        num.u = -num.u;
        num.v = -num.v;
        den.c = -den.c;
        den.u = -den.u;
        den.v = -den.v;
    }
    const float num_hi = aff_top(num);
    if (num_hi < 0.0f) return false;
    const float num_lo = fmaxf(2.0f * num.c - num_hi, 0.0f);
    if (__fdividef(num_lo, den.c + spread) * 0.9999f >= t_max) return false;
    const float hi = fminf(__fdividef(num_hi, den_lo) * 1.0001f, t_max);
    const float err = 3.8147e-6f * n1 * d_max * (o_max + w_max + hi * d_max);
    bool may = true;
    FanAff us{-1.00005f, 0.0f, 0.0f, 0.0f}, bs{0.0f, 0.0f, 0.0f, 0.0f};
    float b1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 B = __ldg(g + 2 + k);
        const float4 ab = abs_b(B);
        const float l1 = l1_b(B);
        const FanAff U{1e-5f - dot_b(B, w), dot_b(B, f.ou), dot_b(B, f.ov), dot_b(ab, f.ores)};
        const FanAff E{dot_b(B, f.mid), dot_b(B, f.du), dot_b(B, f.dv), dot_b(ab, f.res)};
        may = may && !(aff_top2(U, den, num, E) < -err * l1);
        us.c += U.c;
        us.u += U.u;
        us.v += U.v;
        us.r += U.r;
        bs.c += E.c;
        bs.u += E.u;
        bs.v += E.v;
        bs.r += E.r;
        b1 += l1;
    }
    us.c = -us.c;  // 1 + 1e-5 - u - v - w
    us.u = -us.u;
    us.v = -us.v;
    bs.c = -bs.c;
    bs.u = -bs.u;
    bs.v = -bs.v;
    return may && !(aff_top2(us, den, num, bs) < -err * b1);
}

// The records of the leaves `leaves` (lanes holding their references) and of the leaf in progress, dealt
// one per lane, up to 32: returns how many lanes hold one; `rec` and `from`, the record and the lane of
// its leaf.
struct FanDeal {
    uint32_t leaves, first, left, owner;
};
__device__ __forceinline__ uint32_t fan_deal(FanDeal& q, uint32_t ref, uint32_t lane, uint32_t& rec, uint32_t& from) {
    uint32_t pos = 0;
    rec = from = 0;
    while (pos < 32u && (q.leaves | q.left)) {
        if (!q.left) {
            q.owner = (uint32_t)__ffs((int)q.leaves) - 1u;
            q.leaves &= q.leaves - 1u;
            const uint32_t r = __shfl_sync(FULL_WARP, ref, q.owner);
            q.first = r & REF_FIRST_MASK;
            q.left = (r & REF_COUNT_MASK) >> REF_COUNT_SHIFT;
        }
        if (lane - pos < q.left) {
            rec = q.first + (lane - pos);
            from = q.owner;
        }
        const uint32_t take = min(q.left, 32u - pos);
        pos += take;
        q.first += take;
        q.left -= take;
    }
    return pos;
}

// A float as an integer of the same order, and back.
__device__ __forceinline__ uint32_t ordered(float v) {
    const uint32_t b = __float_as_uint(v);
    return b ^ ((uint32_t)((int)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t o) { return __uint_as_float(o ^ ((uint32_t)((int)~o >> 31) | 0x80000000u)); }

// The bounds of one axis's inverse directions from the range of its directions (which holds every ray's,
// rounding included; the factors cover the rounding of the inverses). safe_inv never exceeds 1e12.
__device__ __forceinline__ void fan_range(float lo, float hi, float& near_p, float& near_n, float& far_p, float& far_n) {
    near_p = hi > 0.0f ? fminf(__fdividef(0.99999f, hi), 0.99999e12f) : 0.0f;
    far_p = hi > 0.0f ? (lo > 0.0f ? fminf(__fdividef(1.00001f, lo), 1.00001e12f) : 1.00001e12f) : 0.0f;
    near_n = lo < 0.0f ? fmaxf(__fdividef(0.99999f, lo), -0.99999e12f) : 0.0f;
    far_n = lo < 0.0f ? (hi < 0.0f ? fmaxf(__fdividef(1.00001f, hi), -1.00001e12f) : -1.00001e12f) : 0.0f;
}

// Sets up `f` for the rays of the 2^(w_log + h_log) pixels of a rectangle with corner (x0, y0), from
// directions computed in fast arithmetic (within `slack`, which the bounds include: a few roundings of the
// tetrad's largest component, and of the image plane's extent where a wide view cancels it): lane l samples pixels l and half + l of the rectangle's rows, the first `half` lanes all of them.
__device__ __forceinline__ void fan_bounds(const SrGpuUniforms& U, const Cam& cam, float4 no, uint32_t x0, uint32_t y0,
                                           uint32_t w_log, uint32_t h_log, FanRays& f) {
    const uint32_t lane = threadIdx.x & 31u, half = 1u << (w_log + h_log - 1u);
    const uint32_t sx = (1u << w_log) - 1u, sy = (1u << h_log) - 1u;
    const float kx = __fdividef(2.0f * U.half_wh[0], (float)U.size[0]), ky = __fdividef(-2.0f * U.half_wh[1], (float)U.size[1]);
    const float c0 = U.slice_mode == 0u ? -1.0f : (U.slice_mode == 2u ? 1.0f : 0.0f);
    const float slack = (6e-6f + 2e-6f * (fabsf(U.half_wh[0]) + fabsf(U.half_wh[1]))) * fmaxf(max3f(max_b(cam.e0), max_b(cam.e1), max_b(cam.e2)), max_b(cam.e3));
    float4 d[FAN_RAYS];
    const float ix = sx ? __fdividef(2.0f, (float)sx) : 0.0f, iy = sy ? __fdividef(2.0f, (float)sy) : 0.0f;
#pragma unroll
    for (int r = 0; r < FAN_RAYS; ++r) {
        const uint32_t i = (uint32_t)r * half + (lane & (half - 1u));
        const float u = fmaf(kx, (float)(x0 + (i & sx)) + 0.5f, -U.half_wh[0]), v = fmaf(ky, (float)(y0 + (i >> w_log)) + 0.5f, U.half_wh[1]);
        const float q = rsqrtf(fmaf(u, u, fmaf(v, v, 1.0f))), nx = u * q, ny = v * q;
        auto comp = [&](float e0, float e1, float e2, float e3) { return fmaf(nx, e1, fmaf(ny, e2, fmaf(q, e3, c0 * e0))); };
        d[r] = make_float4(comp(cam.e0.x, cam.e1.x, cam.e2.x, cam.e3.x), comp(cam.e0.y, cam.e1.y, cam.e2.y, cam.e3.y),
                           comp(cam.e0.z, cam.e1.z, cam.e2.z, cam.e3.z), comp(cam.e0.w, cam.e1.w, cam.e2.w, cam.e3.w));
    }
    static_assert(FAN_RAYS == 2, "the ranges below take two rays per lane");
    FanRays r;
    r.d_max = 0.0f;
    auto axis = [&](float a, float b, float& np, float& nn, float& fp, float& fn) {
        const float lo = unordered(redux_min(ordered(fminf(a, b)))) - slack, hi = unordered(redux_max(ordered(fmaxf(a, b)))) + slack;
        r.d_max = fmaxf(r.d_max, fmaxf(-lo, hi));
        fan_range(lo, hi, np, nn, fp, fn);
    };
    axis(d[0].x, d[1].x, r.dirs.near_p.x, r.dirs.near_n.x, r.dirs.far_p.x, r.dirs.far_n.x);
    axis(d[0].y, d[1].y, r.dirs.near_p.y, r.dirs.near_n.y, r.dirs.far_p.y, r.dirs.far_n.y);
    axis(d[0].z, d[1].z, r.dirs.near_p.z, r.dirs.near_n.z, r.dirs.far_p.z, r.dirs.far_n.z);
    axis(d[0].w, d[1].w, r.dirs.near_p.w, r.dirs.near_n.w, r.dirs.far_p.w, r.dirs.far_n.w);
    // The corners: the first and last pixel of the first row (in the first half unless the rectangle is one
    // row) and of the last.
    const float4 d00 = shfl4(d[0], 0u), d11 = shfl4(d[1], half - 1u);
    const float4 d10 = sx < half ? shfl4(d[0], sx) : d11, d01 = sx < half ? shfl4(d[1], half - 1u - sx) : d00;
    r.mid = mul4(add4(add4(d00, d10), add4(d01, d11)), 0.25f);
    r.du = mul4(sub4(add4(d10, d11), add4(d00, d01)), 0.25f);
    r.dv = mul4(sub4(add4(d01, d11), add4(d00, d10)), 0.25f);
    float res = 0.0f;
#pragma unroll
    for (int k = 0; k < FAN_RAYS; ++k) {
        const uint32_t i = (uint32_t)k * half + (lane & (half - 1u));
        const float x = fmaf((float)(i & sx), ix, sx ? -1.0f : 0.0f), y = fmaf((float)(i >> w_log), iy, sy ? -1.0f : 0.0f);
        const float4 e = make_float4(fmaf(x, r.du.x, fmaf(y, r.dv.x, r.mid.x)), fmaf(x, r.du.y, fmaf(y, r.dv.y, r.mid.y)),
                                     fmaf(x, r.du.z, fmaf(y, r.dv.z, r.mid.z)), fmaf(x, r.du.w, fmaf(y, r.dv.w, r.mid.w)));
        res = fmaxf(res, max_b(sub4(d[k], e)));
    }
    r.res = __uint_as_float(redux_max(__float_as_uint(res))) * 1.0001f + slack;
    r.no = no;
    r.o_max = max_b(no);
    __syncwarp();  // the reads of f before
    if (lane == 0) f = r;
    __syncwarp();
}

// The packet form of closest_lean over the fan layout, for the whole warp (all 32 lanes call it together,
// converged): the rays of a rectangle of 2^(w_log + h_log) pixels, bounded by `f`, two per lane of the first
// half of as many lanes: pixel i = r 2^(w_log + h_log - 1) + lane at row i >> w_log. The rays themselves
// (`d`, and `t_max` and `slot`, the closest hits so far; t_max 0: the ray takes no part) are made by
// `rays`, when first a record has to be tested against them (`ready`); a tile of sky never needs them.
// Returns false when the walk was given up, after `budget` steps or `waste` tests without a hit; what it
// found is kept.
//
// The warp walks one sequence: a fan node's 32 entries are tested at once, one per lane, against the
// interval of the directions (fan_interval); the subtrees that may hold a nearer hit wait, the nearest
// taken first; the records of the leaves that may are queued, and 32 at a time are tested one per lane
// against the directions (fan_record); those that remain are tested by every lane against its own rays,
// nearest first. A ray takes a hit when it also enters the record's leaf box, which is when the
// reference tests the record; of hits at equal lambda, the one the reference's near-first order meets
// first (packet_precedes).
//
// The result of each ray is closest_lean's: the closest hit so far is never nearer than the reference's
// final one, so no box the reference enters on the way to its hit is culled, and that hit is tested; no
// nearer hit exists among the records tested. This holds as long as every hit lies beyond the entry
// parameter of its leaf's box as computed. A hit's event passes the barycentric test, so it lies inside
// the record's box, which the build pads by 1e-4: in ray parameter a margin of 1e-4 / |d| on the
// entering axis, against a rounding of the computed entry of order 1e-7 lambda; only hits far along a
// fast axis (lambda ~ 100 or more with |d| ~ 8) bring the two within a factor of two.
template <bool OCT, class Rays>
__device__ __forceinline__ bool closest_fan(const WideScene& s, const Rays& rays, bool& ready, float4 (&d)[FAN_RAYS],
                                            float t_min, uint32_t budget, uint32_t waste, int (&slot)[FAN_RAYS],
                                            float (&t_max)[FAN_RAYS], FanQueue& f, uint2* st, uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u;
    auto farthest = [&]() {
        uint32_t m = __float_as_uint(t_max[0]);
#pragma unroll
        for (int k = 1; k < FAN_RAYS; ++k) m = max(m, __float_as_uint(t_max[k]));
        return redux_max(m);
    };
    uint32_t tile_t = ready ? farthest() : __float_as_uint(180.0f);  // the farthest closest hit, as bits
    uint32_t node = s.fan_root, depth = 0, key = FAN_NONE, ref = FAN_EMPTY, steps = 0, wasted = 0;
    uint32_t head = 0, waiting = 0;  // the queue
    bool fresh = true;
    for (;;) {
        uint32_t count = 0, before = 0, total = 0;
        if (fresh) {
            if (++steps > budget || wasted > waste) return false;
            const float4* bx = s.fan_box + (size_t)node * 64u;
            const float4 bmin = __ldg(bx + lane), bmax = __ldg(bx + 32u + lane);
            ref = __ldg(s.fan_ref + (size_t)node * 32u + lane);
            float en, ex;
            fan_interval(bmin, bmax, f.rays.no, f.rays.no, f.rays.dirs, t_min, __uint_as_float(tile_t), &en, &ex);
            const bool hit = ex >= en;
            const bool leaf = (ref & REF_LEAF) != 0u;
            key = hit && !leaf ? ((__float_as_uint(en) & ~31u) | lane) : FAN_NONE;
            count = hit && leaf ? (ref & REF_COUNT_MASK) >> REF_COUNT_SHIFT : 0u;
            if (__any_sync(FULL_WARP, count != 0u))
                for (uint32_t b = 0; b < s.leaf_bits; ++b) {  // prefix sum, a bit of the counts at a time
                    const uint32_t m = __ballot_sync(FULL_WARP, (count >> b) & 1u);
                    before += (uint32_t)__popc(m & ((1u << lane) - 1u)) << b;
                    total += (uint32_t)__popc(m) << b;
                }
            fresh = false;
        }
        // Queue the records of the leaves, test them 32 at a time; what is left waits for the next
        // node's, or, with nothing nearer to enter, is tested too.
        uint32_t placed = 0;
        const uint32_t k = redux_min(key);
        const bool idle = (k & ~31u) >= tile_t && depth == 0;
        for (;;) {
            if (placed < total) {
                const uint32_t take = min(total - placed, FAN_QUEUE - waiting);
                const uint32_t first = ref & REF_FIRST_MASK, box = node * 64u + lane;
                // This lane's records at places [before, before + count) of the node's, of which
                // [placed, placed + take) go into the queue now.
                const uint32_t lo = max(before, placed), hi = min(before + count, placed + take);
                for (uint32_t j = lo; j < hi; ++j)
                    f.queue[(head + waiting + (j - placed)) & (FAN_QUEUE - 1u)] = make_uint2(first + (j - before), box);
                placed += take;
                waiting += take;
                __syncwarp();
            }
            if (waiting < 32u && !(idle && waiting)) break;
            const uint32_t held = min(waiting, 32u);
            const uint2 mine = f.queue[(head + lane) & (FAN_QUEUE - 1u)];
            head += held;
            waiting -= held;
            float lam = 0.0f;
            const bool may = lane < held && fan_record(s.geoms + 5u * mine.x, f.rays, __uint_as_float(tile_t), &lam);
            uint32_t rkey = may ? ((__float_as_uint(lam) & ~31u) | lane) : FAN_NONE;
            __syncwarp();
            steps += 2;
            if (!ready && __any_sync(FULL_WARP, may)) {
                rays();
                ready = true;
                tile_t = farthest();
            }
            for (;;) {
                const uint32_t q = redux_min(rkey);
                if ((q & ~31u) >= tile_t) break;
                ++steps;
                ++wasted;
                const uint32_t c = q & 31u;
                if (lane == c) rkey = FAN_NONE;
                const uint32_t rec = __shfl_sync(FULL_WARP, mine.x, c);
                // intersect_lean's values, every lane to the end (its lanes would run the union of the
                // early exits anyway, one ray after the other): the rays' chains overlap, and the warp
                // leaves together where no ray is left.
                const float4* g = s.geoms + 5u * rec;
                const float4 n = __ldg(g + 1), v0 = __ldg(g), B1 = __ldg(g + 2), B2 = __ldg(g + 3), B3 = __ldg(g + 4);
                const float4 no = f.rays.no;
                const float2 w01 = add2(f2(v0.x, v0.y), f2(no.x, no.y)), w23 = add2(f2(v0.z, v0.w), f2(no.z, no.w));
                const float num = edot_p(n, make_float4(w01.x, w01.y, w23.x, w23.y));
                bool h[FAN_RAYS], some = false;
                float lambda[FAN_RAYS];
#pragma unroll
                for (int r = 0; r < FAN_RAYS; ++r) {
                    const float denom = edot_p(n, d[r]);
                    lambda[r] = num / denom;
                    // Hits up to and including t_max, so that a hit at the closest hit's lambda is seen.
                    h[r] = fabsf(denom) >= 1e-9f && lambda[r] > t_min && lambda[r] <= t_max[r];
                    some = some || h[r];
                }
                if (!__any_sync(FULL_WARP, some)) continue;
                some = false;
#pragma unroll
                for (int r = 0; r < FAN_RAYS; ++r) {
                    const float4 ev = sub4(mul4(d[r], lambda[r]), no);
                    const float2 q01 = add2(f2(ev.x, ev.y), f2(-v0.x, -v0.y)), q23 = add2(f2(ev.z, ev.w), f2(-v0.z, -v0.w));
                    const float4 p = make_float4(q01.x, q01.y, q23.x, q23.y);
                    const float eps = -1e-5f;
                    const float u = edot_p(B1, p), v = edot_p(B2, p), w = edot_p(B3, p);
                    h[r] = h[r] && !(u < eps || u > 1.0f - eps) && !(v < eps || u + v > 1.0f - eps) &&
                           !(w < eps || u + v + w > 1.0f - eps);
                    some = some || h[r];
                }
                if (!__any_sync(FULL_WARP, some)) continue;
                --wasted;
                const uint32_t box = __shfl_sync(FULL_WARP, mine.y, c);
                const float4 bmin = __ldg(s.fan_box + box), bmax = __ldg(s.fan_box + box + 32u);
#pragma unroll
                for (int r = 0; r < FAN_RAYS; ++r) {
                    if (!h[r]) continue;
                    const float4 ri = inverse(d[r]);  // kept, it would take registers through the walk
                    float be, bex;
                    slab_interval(bmin, bmax, no, ri, t_min, __uint_as_float(__float_as_uint(t_max[r]) - 1u), &be, &bex);
                    if (!(bex >= be)) continue;
                    if (lambda[r] < t_max[r] ||
                        (slot[r] >= 0 && rec != (uint32_t)slot[r] &&
                         packet_precedes<OCT>(s, rec, (uint32_t)slot[r], no, ri, t_min, err))) {
                        t_max[r] = lambda[r];
                        slot[r] = (int)rec;
                    }
                }
                tile_t = farthest();
            }
        }
        if ((k & ~31u) >= tile_t) {  // nothing nearer waits at this node
            if (depth == 0) {
                if (waiting) continue;
                return true;
            }
            const uint2 e = st[--depth];
            key = e.x;
            ref = e.y;
            continue;
        }
        const uint32_t c = k & 31u;
        node = __shfl_sync(FULL_WARP, ref, c);
        if (lane == c) key = FAN_NONE;
        st[depth++] = make_uint2(key, ref);
        fresh = true;
    }
}

// The packet form of any_lean over the fan layout, for the whole warp: which lanes' rays (origins -no,
// directions d, ranges [t_min, t_max]) hit anything. `in`: this lane has a query (some lane does); `hit`
// is set on those that hit. Returns false when the walk was given up after `budget` steps. A lane's
// answer is any_lean's: it tests the records whose leaf box its ray enters until one hits, in whatever
// order. `x`, `y` in [-1, 1]: the lane's place in the tile, over which origins and directions are fitted
// as affine (shadow rays of one surface nearly are).
__device__ __forceinline__ bool any_fan(const WideScene& s, bool in, float4 no, float4 d, float x, float y, float t_min,
                                        float t_max, uint32_t budget, bool& hit, FanShadows& f, uint2* st) {
    const uint32_t lane = threadIdx.x & 31u;
    const float4 inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
    const float o_max = redux_abs(in, max_b(no)), d_max = redux_abs(in, max_b(d));
    const float end = redux_abs(in, t_max);
    __syncwarp();  // the reads of f before
    {
        auto sum = [](float v) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_WARP, v, o);
            return v;
        };
        const float cnt = (float)__popc(__ballot_sync(FULL_WARP, in));
        const float k = 1.0f / cnt;
        const float xm = sum(in ? x : 0.0f) * k, ym = sum(in ? y : 0.0f) * k;
        const float px = in ? x - xm : 0.0f, py = in ? y - ym : 0.0f;
        const float sxx = sum(px * px), syy = sum(py * py), sxy = sum(px * py);
        // Least squares over the lanes: slopes from the 2x2 normal equations (along one axis, or none,
        // where the lanes do not span both).
        const float det = sxx * syy - sxy * sxy;
        const bool both = det > 1e-3f * sxx * syy;
        const float ixx = both ? syy / det : (sxx > 1e-6f && sxx >= syy ? 1.0f / sxx : 0.0f);
        const float iyy = both ? sxx / det : (syy > 1e-6f && syy > sxx ? 1.0f / syy : 0.0f);
        const float ixy = both ? -sxy / det : 0.0f;
        FanShadows r;
        r.dirs = fan_dirs(in, inv);
        auto fit = [&](float v, float* c, float* u, float* w, float* res, float slack) {
            const float m = sum(in ? v : 0.0f) * k;
            const float vx = sum(px * (v - m)), vy = sum(py * (v - m));
            *u = ixx * vx + ixy * vy;
            *w = ixy * vx + iyy * vy;
            *c = m - *u * xm - *w * ym;
            *res = redux_abs(in, v - (*c + *u * x + *w * y)) * 1.0001f + slack;
        };
        const float so = 1e-6f * o_max, sd = 1e-6f * d_max;
        fit(-no.x, &r.o.x, &r.ou.x, &r.ov.x, &r.ores.x, so);
        fit(-no.y, &r.o.y, &r.ou.y, &r.ov.y, &r.ores.y, so);
        fit(-no.z, &r.o.z, &r.ou.z, &r.ov.z, &r.ores.z, so);
        fit(-no.w, &r.o.w, &r.ou.w, &r.ov.w, &r.ores.w, so);
        fit(d.x, &r.mid.x, &r.du.x, &r.dv.x, &r.res.x, sd);
        fit(d.y, &r.mid.y, &r.du.y, &r.dv.y, &r.res.y, sd);
        fit(d.z, &r.mid.z, &r.du.z, &r.dv.z, &r.res.z, sd);
        fit(d.w, &r.mid.w, &r.du.w, &r.dv.w, &r.res.w, sd);
        // The origins' box.
        auto range = [&](float v, float* lo, float* hi) {
            *lo = unordered(redux_min(in ? ordered(v) : 0xFFFFFFFFu));
            *hi = unordered(redux_max(in ? ordered(v) : 0u));
        };
        range(no.x, &r.no_lo.x, &r.no_hi.x);
        range(no.y, &r.no_lo.y, &r.no_hi.y);
        range(no.z, &r.no_lo.z, &r.no_hi.z);
        range(no.w, &r.no_lo.w, &r.no_hi.w);
        if (lane == 0) f = r;
    }
    __syncwarp();
    bool live = in;
    uint32_t node = s.fan_root, depth = 0, ref = FAN_EMPTY, inner = 0, steps = 0;
    bool fresh = true;
    for (;;) {
        if (fresh) {
            fresh = false;
            if (++steps > budget) return false;
            const float4* bx = s.fan_box + (size_t)node * 64u;
            const float4 bmin = __ldg(bx + lane), bmax = __ldg(bx + 32u + lane);
            ref = __ldg(s.fan_ref + (size_t)node * 32u + lane);
            float en, ex;
            fan_interval(bmin, bmax, f.no_lo, f.no_hi, f.dirs, t_min, end, &en, &ex);
            const bool meets = ex >= en;
            const bool leaf = (ref & REF_LEAF) != 0u;
            inner = __ballot_sync(FULL_WARP, meets && !leaf);
            FanDeal deal{__ballot_sync(FULL_WARP, meets && leaf), 0u, 0u, 0u};
            while (deal.leaves | deal.left) {
                uint32_t mine, from;
                const uint32_t held = fan_deal(deal, ref, lane, mine, from);
                uint32_t may = __ballot_sync(FULL_WARP, lane < held && fan_record_any(s.geoms + 5u * mine, f, o_max, d_max, end));
                ++steps;
                while (may) {
                    const uint32_t c = (uint32_t)__ffs((int)may) - 1u;
                    may &= may - 1u;
                    ++steps;
                    const uint32_t rec = __shfl_sync(FULL_WARP, mine, c);
                    GeomHit gh;
                    const bool h = live && intersect_lean(s.geoms + 5u * rec, no, d, t_min, t_max, &gh);
                    if (!__any_sync(FULL_WARP, h)) continue;
                    const uint32_t b = __shfl_sync(FULL_WARP, from, c);
                    float be, bex;
                    slab_interval(__ldg(bx + b), __ldg(bx + 32u + b), no, inv, t_min, t_max, &be, &bex);
                    if (h && bex >= be) {
                        hit = true;
                        live = false;
                    }
                    if (!__any_sync(FULL_WARP, live)) return true;
                }
            }
        }
        if (!inner) {
            if (depth == 0) return true;
            const uint2 e = st[--depth];
            inner = e.x;
            ref = e.y;
            continue;
        }
        const uint32_t c = (uint32_t)__ffs((int)inner) - 1u;
        inner &= inner - 1u;
        node = __shfl_sync(FULL_WARP, ref, c);
        if (inner) st[depth++] = make_uint2(inner, ref);
        fresh = true;
    }
}

// One any-hit query walked by the whole warp (every lane has the same ray): boxes and records one per
// lane against the ray itself.
__device__ __forceinline__ bool any_fan_one(const WideScene& s, float4 no, float4 d, float t_min, float t_max, uint2* st,
                                            uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u;
    const float4 inv = v4(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z), safe_inv(d.w));
    uint32_t node = s.fan_root, depth = 0, visits = 0;
    for (;;) {
        if (++visits > MAX_VISITS_FAST) {
            if (lane == 0) atomicOr(err, ERR_TRAVERSAL_LIMIT);
            return false;
        }
        const float4* bx = s.fan_box + (size_t)node * 64u;
        uint32_t ref = __ldg(s.fan_ref + (size_t)node * 32u + lane);
        float en, ex;
        slab_interval(__ldg(bx + lane), __ldg(bx + 32u + lane), no, inv, t_min, t_max, &en, &ex);
        const bool meets = ex >= en;
        const bool leaf = (ref & REF_LEAF) != 0u;
        uint32_t inner = __ballot_sync(FULL_WARP, meets && !leaf);
        FanDeal deal{__ballot_sync(FULL_WARP, meets && leaf), 0u, 0u, 0u};
        while (deal.leaves | deal.left) {
            uint32_t mine, from;
            const uint32_t held = fan_deal(deal, ref, lane, mine, from);
            GeomHit gh;
            if (__any_sync(FULL_WARP, lane < held && intersect_lean(s.geoms + 5u * mine, no, d, t_min, t_max, &gh))) return true;
        }
        while (!inner) {
            if (depth == 0) return false;
            const uint2 e = st[--depth];
            inner = e.x;
            ref = e.y;
        }
        const uint32_t c = (uint32_t)__ffs((int)inner) - 1u;
        inner &= inner - 1u;
        node = __shfl_sync(FULL_WARP, ref, c);
        if (inner) st[depth++] = make_uint2(inner, ref);
    }
}

}  // namespace srk
