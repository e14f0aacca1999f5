// Binned star footprints for the batched fast path (star_light, star.rs:240-286).
//
// A star's cone event depends on the observer, not on the pixel, so it is computed once per
// (observer, star) and projected onto the image. Its footprint only reaches pixels whose direction
// is within atan(2.4 * spread) of the star's (the 4-sigma cut of star.rs:266-270, spread <= the
// pixel pitch), so each star is listed in the 16x16 tiles a generous radius around its projection
// covers (count, prefix sum, fill: compact lists of any length; then each list is sorted by star index).
// What a star's term has that does not depend on the pixel (its event in the observer's frame, its
// Doppler-shifted colour) is computed once with it. Every pixel sums the terms of its tile's list in
// index order: the stars it skips are exactly stars whose term the cut rejects, so the sum is the brute
// force sum bit for bit. A tile whose list does not fit (longer than STAR_SORT_CAP, or past the list
// buffer) sums every star instead. Observers outside the binning's assumptions (stars_binned_for in
// sr_kernels.h) keep the brute force in the shading kernel. Included by sr_fast.cu, which defines
// find_obs, cam_of and ObsDev.
#pragma once

namespace srk {

constexpr uint32_t STAR_SORT_CAP = 8192;  // entries of a tile sorted in shared memory (32 KB)

struct StarBinArgs {
    const SrGpuUniforms* U;
    const float4* cam;
    const ObsDev* obs;
    const float4* stars;  // headers then segments
    uint32_t n, num_stars;
    float4* r;            // per (observer, star): the cone event in the observer's space
    float4* color;        // its Doppler-shifted blackbody colour, and the flux
    float4* box;          // the pixels its footprint may reach: x0, x1, y0, y1 (x0 > x1: none)
    uint32_t* count;      // per star tile: listed stars
    const uint32_t* offset;  // per star tile: start of its list (exclusive prefix sum of count)
    uint32_t* fill;       // per star tile: entries written so far
    uint32_t* list;
    uint32_t list_cap;
    BBConst bb;
};

// The star tiles a box touches.
struct StarRect {
    int x0, x1, y0, y1;
};
__device__ __forceinline__ StarRect star_rect(float4 box, uint32_t width, uint32_t height) {
    const int tx16 = (int)((width + STAR_TILE - 1) / STAR_TILE), ty16 = (int)((height + STAR_TILE - 1) / STAR_TILE);
    return StarRect{max(0, (int)floorf(box.x / STAR_TILE)), min(tx16 - 1, (int)floorf(box.y / STAR_TILE)),
                    max(0, (int)floorf(box.z / STAR_TILE)), min(ty16 - 1, (int)floorf(box.w / STAR_TILE))};
}

// Pass 1: the cone event of (observer, star), its colour, its footprint's box, and the tile counts.
__global__ void __launch_bounds__(256) k_star_bin(StarBinArgs a) {
    const uint64_t gi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= (uint64_t)a.n * a.num_stars) return;
    const uint32_t o = (uint32_t)(gi / a.num_stars), i = (uint32_t)(gi % a.num_stars);
    a.box[gi] = make_float4(1.0f, 0.0f, 1.0f, 0.0f);
    const SrGpuUniforms& U = a.U[o];
    if (!stars_binned_for(U, a.num_stars)) return;
    const Cam cam = cam_of(a.cam, o);
    float4 ro, rd;
    float sx, sy;
    camera_ray(U, cam, 0, 0, &ro, &rd, &sx, &sy);  // the ray origin is the same for every pixel
    const float cone = U.slice_mode == 0u ? -1.0f : (U.slice_mode == 2u ? 1.0f : 0.0f);
    const float4 hd = __ldg(a.stars + i);
    float4 cd, cu;
    if (!cone_event(a.stars + a.num_stars, __float_as_uint(hd.z), __float_as_uint(hd.w), ro, cam.e0, cone, &cd, &cu))
        return;
    // The star's direction in the camera frame (star_term's r).
    const float tau = -mdot(cd, cam.e0);
    const float4 r = add4(cd, mul4(cam.e0, -tau));
    const float r1 = mdot(r, cam.e1), r2 = mdot(r, cam.e2), r3 = mdot(r, cam.e3);
    const float rn = sqrtf(r1 * r1 + r2 * r2 + r3 * r3);
    if (!(rn > 0.0f)) return;
    const float W = (float)U.size[0], H = (float)U.size[1];
    const float hw = U.half_wh[0], hh = U.half_wh[1];
    // Angles from the view axis: the star's alpha; the pixels' at most amax; the footprint's theta.
    const float alpha = acosf(fminf(fmaxf(r3 / rn, -1.0f), 1.0f));
    const float amax = atanf(sqrtf(hw * hw + hh * hh));
    const float theta = 2.4f * (2.0f * hh / H) * 1.1f + 1e-4f;
    if (alpha - theta > amax + 0.01f) return;  // no pixel direction comes within theta of the star
    const float ssx = r1 / r3, ssy = r2 / r3;
    // Radius in the tangent plane (the radial stretch is the worst case), then in pixels.
    const float rt = (tanf(alpha + theta) - tanf(alpha)) * 1.25f;
    const float rpx = rt / (2.0f * hw / W) + 2.0f, rpy = rt / (2.0f * hh / H) + 2.0f;
    const float cx = (ssx / hw + 1.0f) * 0.5f * W - 0.5f, cy = (1.0f - ssy / hh) * 0.5f * H - 0.5f;
    if (!(cx + rpx >= 0.0f && cx - rpx <= W - 1.0f && cy + rpy >= 0.0f && cy - rpy <= H - 1.0f)) return;
    const ObsDev& od = a.obs[o];
    const float4 box = make_float4(cx - rpx, cx + rpx, cy - rpy, cy + rpy);
    const StarRect t = star_rect(box, od.width, od.height);
    if (t.x0 > t.x1 || t.y0 > t.y1) return;
    float dop = 1.0f;  // star_term's Doppler factor
    if (cone < 0.0f) {
        const float lam = sqrtf(fmaxf(mdot(r, r), 0.0f));
        const float du = mdot(cd, cu);
        if (du > 0.0f) dop = lam / du;
    }
    const F3 c = blackbody_rgb(hd.x * dop, BB{a.bb.r5, a.bb.g5, a.bb.b5, a.bb.wr, a.bb.wg, a.bb.wb});
    a.r[gi] = r;
    a.color[gi] = make_float4(c.x, c.y, c.z, hd.y);
    a.box[gi] = box;
    const uint32_t tx16 = (od.width + STAR_TILE - 1) / STAR_TILE;
    for (int ty = t.y0; ty <= t.y1; ++ty)
        for (int tx = t.x0; tx <= t.x1; ++tx) atomicAdd(a.count + od.star_tile_base + (uint32_t)ty * tx16 + (uint32_t)tx, 1u);
}

// Pass 2: each (observer, star) writes its index into the lists of its tiles.
__global__ void __launch_bounds__(256) k_star_fill(StarBinArgs a) {
    const uint64_t gi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= (uint64_t)a.n * a.num_stars) return;
    const float4 box = a.box[gi];
    if (box.x > box.y) return;
    const uint32_t o = (uint32_t)(gi / a.num_stars), i = (uint32_t)(gi % a.num_stars);
    const ObsDev& od = a.obs[o];
    const uint32_t tx16 = (od.width + STAR_TILE - 1) / STAR_TILE;
    const StarRect t = star_rect(box, od.width, od.height);
    for (int ty = t.y0; ty <= t.y1; ++ty)
        for (int tx = t.x0; tx <= t.x1; ++tx) {
            const uint32_t tile = od.star_tile_base + (uint32_t)ty * tx16 + (uint32_t)tx;
            const uint64_t k = (uint64_t)__ldg(a.offset + tile) + atomicAdd(a.fill + tile, 1u);
            if (k < a.list_cap) a.list[k] = i;
        }
}

// Whether a tile's list is too long to be sorted or not all there: its pixels sum every star.
__device__ __forceinline__ bool star_list_short(uint32_t cnt, uint32_t off, uint32_t list_cap) {
    return cnt > STAR_SORT_CAP || (uint64_t)off + cnt > list_cap;
}

// Pass 3: one tile's list per block, sorted by star index (bitonic, in shared memory).
__global__ void __launch_bounds__(256) k_star_sort(uint32_t* count, const uint32_t* offset, uint32_t* list, uint32_t list_cap,
                                                   uint32_t num_stars) {
    extern __shared__ uint32_t keys[];  // STAR_SORT_CAP entries
    const uint32_t tile = blockIdx.x;
    const uint32_t cnt = count[tile], off = offset[tile];
    if (cnt == 0 || star_list_short(cnt, off, list_cap)) return;
    uint32_t p2 = 1;
    while (p2 < cnt) p2 <<= 1;
    int bad = 0;
    for (uint32_t k = threadIdx.x; k < p2; k += blockDim.x) {
        const uint32_t v = k < cnt ? list[off + k] : 0xFFFFFFFFu;
        if (k < cnt && v >= num_stars) bad = 1;  // a list this pass did not fill
        keys[k] = v;
    }
    if (__syncthreads_or(bad)) {
        if (threadIdx.x == 0) count[tile] = STAR_SORT_CAP + 1;  // sum every star
        return;
    }
    for (uint32_t size = 2; size <= p2; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t k = threadIdx.x; k < p2; k += blockDim.x) {
                const uint32_t j = k ^ stride;
                if (j > k) {
                    const bool up = (k & size) == 0;
                    const uint32_t x = keys[k], y = keys[j];
                    if ((x > y) == up) {
                        keys[k] = y;
                        keys[j] = x;
                    }
                }
            }
            __syncthreads();
        }
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) list[off + k] = keys[k];
}

struct StarTileArgs {
    SceneDev s;
    const SrGpuUniforms* U;
    const float4* cam;
    const ObsDev* obs;
    const uint32_t* star_pre;  // star-tile prefix over observers (n + 1)
    uint32_t n;
    const float4* hits;
    const uint32_t* slots;
    const float4* r;
    const float4* color;
    const float4* box;
    const uint32_t* count;
    const uint32_t* offset;
    const uint32_t* list;
    uint32_t list_cap;
    float4* hdr;
    BBConst bb;
};

// Pass 4: every pixel adds its star sum to the HDR colour the shading kernel wrote (the same `colour + stars`
// addition as the shading). A warp takes 8x4 pixels of a tile and 32 stars of its list at a time: lanes
// drop the stars whose box misses the warp's pixels (two of three) and hold the others' data, which is
// passed round by shuffles, so that the terms, which must be added one after the other, wait for no
// memory. It is bound by the densest tiles' chains: a block takes a quarter of a tile, so that they
// spread over the chip. 100k stars at 1280x800: 162 us for 16x16 pixels a block with the sort and a
// star's whole term per pixel; 51 us, and 20 for the sort, like this.
constexpr uint32_t STAR_BLOCKS = 4;  // blocks of two warps per tile
__global__ void __launch_bounds__(64) k_star_tiles(const __grid_constant__ StarTileArgs a) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t tile = blockIdx.x / STAR_BLOCKS, lane = threadIdx.x & 31u;
    const uint32_t sub = (blockIdx.x % STAR_BLOCKS) * 2u + (threadIdx.x >> 5);  // 8x4 pixels, two in a row of the tile
    const uint32_t cnt = a.count[tile];
    if (cnt == 0) return;
    const uint32_t o = find_obs(a.star_pre, a.n, tile);
    const SrGpuUniforms& U = a.U[o];
    if (!stars_binned_for(U, a.s.num_stars)) return;
    const ObsDev& od = a.obs[o];
    const uint32_t local = tile - __ldg(a.star_pre + o);
    const uint32_t tx16 = (od.width + STAR_TILE - 1) / STAR_TILE;
    const uint32_t x0 = (local % tx16) * STAR_TILE + (sub & 1u) * 8u, y0 = (local / tx16) * STAR_TILE + (sub >> 1) * 4u;
    const uint32_t px = x0 + (lane & 7u), py = y0 + (lane >> 3);
    const bool inside = px < od.width && py < od.height;
    const uint32_t off = a.offset[tile];
    const uint32_t l = py * od.width + px, p = od.pix_base + l;
    const Cam cam = cam_of(a.cam, o);
    float4 ro, rd;
    float sx, sy;
    camera_ray(U, cam, px, py, &ro, &rd, &sx, &sy);
    float lambda_max = INFINITY;
    if (inside && a.slots[p] != 0xFFFFFFFFu) lambda_max = a.hits[p].x;
    F3 total{0.0f, 0.0f, 0.0f};
    if (star_list_short(cnt, off, a.list_cap)) {
        if (!inside) return;
        total = stars_brute(a.s, U, cam, ro, rd, sx, sy, lambda_max, a.bb);
    } else {
        float4 n;
        float spread, cone;
        star_ray(U, cam, rd, sx, sy, &n, &spread, &cone);
        const size_t base = (size_t)o * a.s.num_stars;
        const float bx0 = (float)x0, bx1 = (float)(x0 + 7u), by0 = (float)y0, by1 = (float)(y0 + 3u);
        for (uint32_t k0 = 0; k0 < cnt; k0 += 32u) {
            bool near = false;
            float4 sr = v4(0.0f, 0.0f, 0.0f, 0.0f), sc = sr;
            if (k0 + lane < cnt) {
                const size_t i = base + a.list[off + k0 + lane];
                const float4 box = __ldg(a.box + i);
                near = box.x <= bx1 && box.y >= bx0 && box.z <= by1 && box.w >= by0;
                if (near) {
                    sr = __ldg(a.r + i);
                    sc = __ldg(a.color + i);
                }
            }
            for (uint32_t m = __ballot_sync(FULL, near); m; m &= m - 1u) {
                const uint32_t j = (uint32_t)__ffs((int)m) - 1u;
                const float4 r = make_float4(__shfl_sync(FULL, sr.x, j), __shfl_sync(FULL, sr.y, j), __shfl_sync(FULL, sr.z, j),
                                             __shfl_sync(FULL, sr.w, j));
                // star_term (star.rs:254-283) from r and the colour.
                const float along = mdot(r, n);
                const float4 perp = sub4(r, mul4(n, along));
                const float d2 = fmaxf(mdot(perp, perp), 0.0f);
                const float sigma = 0.6f * (0.0f + spread * along);
                const float cut = 4.0f * sigma;
                const bool in = inside && along > 0.0f && along < lambda_max && d2 < cut * cut;
                if (!__any_sync(FULL, in)) continue;
                const F3 rgb{__shfl_sync(FULL, sc.x, j), __shfl_sync(FULL, sc.y, j), __shfl_sync(FULL, sc.z, j)};
                const float cn = __shfl_sync(FULL, sc.w, j);
                if (in) {
                    const float inv = 1.0f / (2.0f * sigma * sigma);
                    const float kernel = expf(-d2 * inv) * inv * FRAC_1_PI_F;
                    total = add(total, mul(rgb, cn * kernel));
                }
            }
        }
        if (!inside) return;
    }
    float4* h = a.hdr + (size_t)od.pyr_base + l;
    const float4 v = *h;
    *h = make_float4(v.x + total.x, v.y + total.y, v.z + total.z, 0.0f);
}

}  // namespace srk
