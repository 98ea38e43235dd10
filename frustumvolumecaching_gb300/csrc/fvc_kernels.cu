/*
 * fvc_kernels.cu - the renderer's CUDA kernels for sm_103a.
 *
 *  (the renderer's wavefront kernels live in fvc_render.cu)
 *  cache_*_kernel          frustum cache build, one depth brick of every alive
 *                          8x8 tile per iteration (search, density network,
 *                          compositing, then deterministic slots):
 *                          CacheRenderer::initCacheBlockwise,
 *                          src/cache_renderer.cu:18-569,931-1051.
 *  inference_kernel        network at given inputs (NerfNetwork::inference).
 *
 * Every loop is bounded; guards set bits in a device word instead of
 * trapping.
 */
#include "fvc_kernels.h"

#include <cuda_fp16.h>

namespace fvc {

constexpr unsigned FULL = 0xffffffffu;

/* ------------------------------------------------------------------------- */
/* network at given inputs (testing / occupancy generation)                   */
/* ------------------------------------------------------------------------- */
template <int HEAD_HIDDEN>
__global__ void __launch_bounds__(128) inference_kernel(InferenceParams p)
{
    __shared__ uint2 Wsm[W_TOTAL];
    __shared__ float bsm[64];
    __shared__ __align__(16) __half tiles[4][32 * TILE_STRIDE];
    for (int i = threadIdx.x; i < W_TOTAL; i += blockDim.x) Wsm[i] = p.weights[i];
    for (int i = threadIdx.x; i < 64; i += blockDim.x) bsm[i] = p.bias3[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __half *tile = tiles[w];
    const int n_batches = (p.n + 31) / 32;
    for (int b = blockIdx.x * 4 + w; b < n_batches; b += gridDim.x * 4) {
        const int r = b * 32 + lane;
        __half *trow = tile + lane * TILE_STRIDE;
        if (r < p.n) {
            const float3 pos = make_float3(p.pos[3 * r], p.pos[3 * r + 1], p.pos[3 * r + 2]);
            hash_encode_any(p.grid, p.table, pos, reinterpret_cast<__half2 *>(trow));
            if (p.features)
                for (int j = 0; j < 32; ++j) p.features[32 * r + j] = __half2float(trow[j]);
            if (p.dir) sh16(make_float3(p.dir[3 * r], p.dir[3 * r + 1], p.dir[3 * r + 2]), reinterpret_cast<__half2 *>(trow + 32));
        } else {
            for (int c = 0; c < 24; ++c) reinterpret_cast<uint32_t *>(trow)[c] = 0u;
        }
        __syncwarp();
        density_mlp(tile, Wsm, lane);
        if (p.dir) {
            float lo[2][4];
            color_mlp<HEAD_HIDDEN>(tile, Wsm, bsm, lane, lo);
            const int g = lane >> 2, t = lane & 3;
            if (t < 2) {
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    __half *r0 = tile + (16 * mt + g) * TILE_STRIDE + 48 + 2 * t;
                    *reinterpret_cast<uint32_t *>(r0) = pack_h2(lo[mt][0], lo[mt][1]);
                    *reinterpret_cast<uint32_t *>(r0 + 8 * TILE_STRIDE) = pack_h2(lo[mt][2], lo[mt][3]);
                }
            }
        }
        __syncwarp();
        if (r < p.n) {
            if (p.out4) {
                p.out4[4 * r + 0] = p.dir ? __half2float(trow[48]) : 0.f;
                p.out4[4 * r + 1] = p.dir ? __half2float(trow[49]) : 0.f;
                p.out4[4 * r + 2] = p.dir ? __half2float(trow[50]) : 0.f;
                p.out4[4 * r + 3] = __half2float(trow[16]);
            }
            if (p.base_out)
                for (int j = 0; j < 16; ++j) p.base_out[16 * r + j] = __half2float(trow[16 + j]);
        }
        __syncwarp();
    }
}

cudaError_t launch_inference(const InferenceParams &p, int head_hidden, int n_sms, cudaStream_t s)
{
    const int n_batches = (p.n + 31) / 32;
    const int grid = max(1, min((n_batches + 3) / 4, n_sms * 8));
    if (head_hidden == 2) inference_kernel<2><<<grid, 128, 0, s>>>(p);
    else inference_kernel<1><<<grid, 128, 0, s>>>(p);
    return cudaGetLastError();
}

/* ------------------------------------------------------------------------- */
/* frustum cache build                                                       */
/* ------------------------------------------------------------------------- */

/* initPayloads_cache_init_kernel, src/cache_renderer.cu:18-81: one CTA of
 * 64 threads per 8x8 tile; the blocks past the tiles' write the occupancy
 * cells. */
__global__ void __launch_bounds__(64) cache_init_kernel(CacheBuildParams p, int n_tiles)
{
    const int tile = blockIdx.x;
    if (tile >= n_tiles) {
        cells_from_bits(p.bits, p.cells, tile - n_tiles);
        return;
    }
    const int k = threadIdx.x;
    const int tx = tile % p.bX, ty = tile / p.bX;
    const int px = tx * 8 + (k & 7), py = ty * 8 + (k >> 3);
    float3 o, d;
    generate_ray(p.cam, px, py, o, d);
    float tn, tf;
    const bool hits = ray_aabb(o, d, p.scene.aabb_from, p.scene.aabb_to, tn, tf);
    const int start_step = max(0, (int)F_SUB(step_from_t(p.steps, hits ? tn : p.steps.near_), p.steps.near_i));
    CacheRay cr;
    cr.o = o; cr.d = d;
    cr.far_ = hits ? fminf(tf, p.steps.far_) : p.steps.far_;
    cr.T = 1.0f;
    cr.alive = hits ? 1 : 0;
    p.rays[(size_t)tile * 64 + k] = cr;
    __shared__ int s_alive[2], s_min[2];
    const int wa = __reduce_add_sync(FULL, hits ? 1 : 0);
    const int wm = __reduce_min_sync(FULL, (unsigned)start_step);
    if ((k & 31) == 0) { s_alive[k >> 5] = wa; s_min[k >> 5] = wm; }
    __syncthreads();
    if (k == 0) {
        p.block_step[tile] = min(s_min[0], s_min[1]) / 8;
        p.tile_alive[tile] = (s_alive[0] + s_alive[1]) > 0;
    }
}

/* The blockwise cache build (CacheRenderer::initCacheBlockwise,
 * src/cache_renderer.cu:931-1051) as a wavefront per depth-brick iteration:
 *   cache_search_kernel    per alive tile: the next depth brick holding an
 *                          occupied sample, its samples appended to a row list
 *                          (sample_cache_init_first/second_kernel :83-287);
 *   cache_density_kernel   the density network on all rows of the iteration
 *                          (inferenceLatents), warp-level tensor-core MLP;
 *   cache_composite_kernel per processed tile: density-only compositing and
 *                          the brick's need of a slot
 *                          (accumulateNew_cache_init_second_kernel :289-528);
 * then cache_assign_kernel gives bricks their slots and cache_fill_kernel
 * writes their voxels. */
/* G groups of 64 threads, one per ray of the tile: group g examines the depth
 * brick g past the next, and the tile takes the first one that holds an
 * occupied sample.  A tile's search is a serial chain over its empty bricks
 * (up to 36 of them in one iteration of the 3-cascade scene at 323x181), so
 * with few alive tiles eight bricks are examined at once; with many, all but
 * the first group's work would be repeated in the next iteration. */
constexpr int SEARCH_GROUPS = 8;

template <bool VD, int G>
__global__ void __launch_bounds__(64 * G, G == 1 ? 16 : 2) cache_search_kernel(CacheBuildParams p)
{
    after_previous();
    __shared__ uint8_t s_flags[2][2 * G]; /* per warp: 1 an occupied sample, 2 a ray alive past the brick */
    __shared__ int2 red[2];
    __shared__ int row_base;
    const int group = threadIdx.x / 64, k = threadIdx.x % 64, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wid = warp & 1;
    const int n_alive_tiles = *p.n_alive_tiles;
    for (int ai = blockIdx.x; ai < n_alive_tiles; ai += gridDim.x) {
        __syncthreads();
        const int tile = p.alive_list[ai];
        const CacheRay cr = p.rays[(size_t)tile * 64 + k];
        int bstep = p.block_step[tile];
        uint32_t mask = 0;
        float t_brick = 0.f;
        bool ray_alive = false; /* past the group's brick: the midpoints grow, so the brick alone tells */
        int chosen = -1;
        bool stop = false, alive_before = __syncthreads_or(cr.alive);
        for (int guard = 0; guard < p.max_search && !stop; ++guard) {
            float t1 = t_brick = t_from_step(p.steps, F_ADD((float)((bstep + group) * 8), p.steps.near_i));
            mask = 0;
            ray_alive = cr.alive != 0;
#pragma unroll
            for (int s = 0; s < 8; s += 2) {
                float tm[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float t0 = t1;
                    t1 = F_ADD(t0, calc_step(p.steps, t0));
                    tm[c] = F_MUL(F_ADD(t0, t1), 0.5f);
                }
                /* the steps past the far bound are the last ones */
                const uint32_t in = (tm[0] > cr.far_ ? 0u : 1u) | (tm[1] > cr.far_ ? 0u : 2u);
                if (in != 3u) ray_alive = false;
                if (in) mask |= (occupied2(p.scene, p.bits, p.cells, cr.o, cr.d, make_float2(tm[0], tm[1])) & in) << s;
            }
            const bool any_occ = __any_sync(FULL, mask != 0u), any_alive = __any_sync(FULL, ray_alive);
            if (lane == 0) s_flags[guard & 1][warp] = (any_occ ? 1 : 0) | (any_alive ? 2 : 0);
            __syncthreads();
            /* the bricks in order, as one group would have met them (the same in every thread) */
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (stop) break;
                const int f = s_flags[guard & 1][2 * g] | s_flags[guard & 1][2 * g + 1];
                if (!alive_before || bstep >= p.bZ) { /* no ray left, or beyond the frustum depth: the tile stops */
                    stop = true;
                } else if (f & 1) {
                    stop = true;
                    chosen = g;
                } else {
                    ++bstep;
                    alive_before = f & 2;
                }
            }
            if (!stop && guard == p.max_search - 1 && threadIdx.x == 0) atomicOr(p.guard, 4);
        }
        const bool mine = group == max(chosen, 0); /* the group that goes on with its brick */
        if (chosen < 0) mask = 0, ray_alive = false;
        const int cnt = __popc(mask);
        const int before = lanes_before(cnt); /* of this warp's rays */
        const int w_alive = __reduce_add_sync(FULL, ray_alive ? 1u : 0u);
        if (mine && lane == 31) red[wid] = make_int2(before + cnt, w_alive);
        __syncthreads();
        const int total = red[0].x + red[1].x, n_alive = red[0].y + red[1].y;
        const bool processed = total > 0 && n_alive > 0;
        if (mine && k == 0) {
            p.tile_n_samples[ai] = total;
            p.tile_processed[ai] = processed;
            p.tile_alive[tile] = n_alive > 0;
            p.block_step[tile] = bstep;
            if (processed) row_base = atomicAdd(p.build_row_counter, total);
        }
        if (mine) p.rays[(size_t)tile * 64 + k].alive = ray_alive;
        __syncthreads();
        if (!processed || !mine) continue;
        /* append the brick's samples to the iteration's rows, in (ray, step) order */
        int row = row_base + before + (wid ? red[0].x : 0);
        int *rof = p.build_row_of + (size_t)ai * 512;
        float t1 = t_brick;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const float t0 = t1;
            const float dt = calc_step(p.steps, t0);
            t1 = F_ADD(t0, dt);
            const float tm = F_MUL(F_ADD(t0, t1), 0.5f);
            if ((mask >> s) & 1u) {
                const float3 cp = contract(p.scene, at(cr.o, cr.d, tm));
                p.build_rows[row] = make_float4(cp.x, cp.y, cp.z, 0.f);
                if (VD) /* the build's network input direction (src/cache_renderer.cu:1026) */
                    p.build_dirs[row] = make_float4((cr.d.x + 1.0f) / 2.0f, (cr.d.y + 1.0f) / 2.0f, (cr.d.z + 1.0f) / 2.0f, 0.f);
                rof[s * 64 + k] = row++;
            } else {
                rof[s * 64 + k] = -1;
            }
        }
    }
}

/* density network on every row of the iteration: log-density and the 8
 * latents (fp16, as NerfNetwork::inferenceLatents stores them); VD: the view-dependent network's first head on the rows' ray
 * directions */
template <bool VD>
__global__ void __launch_bounds__(128) cache_density_kernel(CacheBuildParams p)
{
    after_previous();
    __shared__ uint2 Wsm[W_L3], Wfh[VD ? W_L3 : 1];
    __shared__ __align__(16) __half tiles[4][32 * TILE_STRIDE];
    const int n = *p.build_row_counter;
    if ((int)blockIdx.x * 128 >= n) return; /* no rows: no weights */
    for (int i = threadIdx.x; i < W_L3; i += blockDim.x) Wsm[i] = p.weights[i];
    if (VD)
        for (int i = threadIdx.x; i < W_L3; i += blockDim.x) Wfh[i] = p.weights_fh[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __half *tile = tiles[w];
    __half *trow = tile + lane * TILE_STRIDE;
    const int lo = p.latent_offset;
    for (int b = blockIdx.x * 4 + w; b < (n + 31) / 32; b += gridDim.x * 4) {
        const int r = b * 32 + lane;
        if (r < n) {
            const float4 rw = p.build_rows[r];
            hash_encode(p.grid, p.table, make_float3(rw.x, rw.y, rw.z), reinterpret_cast<__half2 *>(trow));
        } else {
            for (int c = 0; c < 16; ++c) reinterpret_cast<uint32_t *>(trow)[c] = 0u;
        }
        __syncwarp();
        density_mlp(tile, Wsm, lane);
        __half logd = trow[16];
        if (VD) {
            /* the first head (NerfNetwork::inferenceLatents, include/nerf_network.h:183-197) on
             * [density outputs | SH of the build ray's direction]; its outputs take rows 1.. of the
             * head input (row 0 keeps the log-density) */
            uint4 o0 = reinterpret_cast<const uint4 *>(trow + 16)[0], o1 = reinterpret_cast<const uint4 *>(trow + 16)[1];
            __half2 sh[8];
            if (r < n) {
                float3 d01;
                if (p.build_dirs) {
                    const float4 d = p.build_dirs[r];
                    d01 = make_float3(d.x, d.y, d.z);
                } else { /* the per-ray fill: the row's ray (src/cache_renderer.cu:899) */
                    const float4 d = p.dir_states[p.dir_slot[r]].dt;
                    d01 = make_float3((d.x + 1.0f) / 2.0f, (d.y + 1.0f) / 2.0f, (d.z + 1.0f) / 2.0f);
                }
                sh16(d01, sh);
            } else {
                for (int q = 0; q < 8; ++q) sh[q] = __floats2half2_rn(0.f, 0.f);
            }
            __syncwarp();
            reinterpret_cast<uint4 *>(trow)[0] = o0;
            reinterpret_cast<uint4 *>(trow)[1] = o1;
            reinterpret_cast<uint4 *>(trow)[2] = *reinterpret_cast<const uint4 *>(sh);
            reinterpret_cast<uint4 *>(trow)[3] = *reinterpret_cast<const uint4 *>(sh + 4);
            __syncwarp();
            density_mlp(tile, Wfh, lane); /* the same 32 -> 64 -> 16 shape */
            /* rows 1..16 <- first-head outputs 0..15 */
            __syncwarp();
            for (int j = 15; j >= 1; --j) trow[16 + j] = trow[16 + j - 1];
            trow[16] = logd;
        }
        if (r < n) {
            p.build_den[r] = trow[16];
            uint32_t lw[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                lw[q] = (uint32_t)__half_as_ushort(trow[16 + lo + 2 * q]) | ((uint32_t)__half_as_ushort(trow[17 + lo + 2 * q]) << 16);
            p.build_lat[r] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        }
        __syncwarp();
    }
}

/* grid: the alive tiles, as last known.  Groups of bricks below SEARCH_TILES of them: a search launch of the 3-cascade
 * scene's build takes, us with 1 / 8 groups, 44 / 30 at 323x181 (943 tiles) and 23 / 11 at 128x128 (256); thresholds of
 * 1024 to 4096 tiles measured alike. */
#ifndef FVC_SEARCH_TILES
#define FVC_SEARCH_TILES 1024
#endif
cudaError_t launch_cache_search(const CacheBuildParams &p, int grid, cudaStream_t s)
{
    if (grid <= FVC_SEARCH_TILES) {
        launch_after(p.view_dependent ? cache_search_kernel<true, SEARCH_GROUPS> : cache_search_kernel<false, SEARCH_GROUPS>, grid, 64 * SEARCH_GROUPS, 0, s, p);
    } else {
        launch_after(p.view_dependent ? cache_search_kernel<true, 1> : cache_search_kernel<false, 1>, grid, 64, 0, s, p);
    }
    return cudaGetLastError();
}

cudaError_t launch_cache_density(const CacheBuildParams &p, int grid, cudaStream_t s)
{
    launch_after(p.view_dependent ? cache_density_kernel<true> : cache_density_kernel<false>, grid, 128, 0, s, p);
    return cudaGetLastError();
}

/* One warp per processed tile, rays lane and lane + 32 per lane:
 * density-only compositing over the brick's 8 steps
 * (accumulateNew_cache_init_second_kernel :349-393) and whether the brick
 * needs a slot (a visible sample). */
__global__ void __launch_bounds__(128) cache_composite_kernel(CacheBuildParams p)
{
    after_previous();
    const int lane = threadIdx.x & 31;
    const int n_alive_tiles = *p.n_alive_tiles;
    const int n_warps = gridDim.x * (blockDim.x >> 5);
    for (int ai = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); ai < n_alive_tiles; ai += n_warps) {
        if (!p.tile_processed[ai]) continue; /* uniform over the warp */
        const int tile = p.alive_list[ai];
        const int bstep = p.block_step[tile];
        const int *rof = p.build_row_of + (size_t)ai * 512;
        const float t1s = t_from_step(p.steps, F_ADD((float)(bstep * 8), p.steps.near_i));
        int visible = 0, alive = 0;
        /* both rays' 16 row numbers, then their densities, before the first is composited: two memory
         * latencies a tile instead of two a step */
        CacheRay cr[2];
        int rows[2][8];
        float sigma[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            cr[h] = p.rays[(size_t)tile * 64 + h * 32 + lane];
#pragma unroll
            for (int s = 0; s < 8; ++s) rows[h][s] = rof[s * 64 + h * 32 + lane];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int s = 0; s < 8; ++s) sigma[h][s] = rows[h][s] >= 0 ? __half2float(p.build_den[rows[h][s]]) : 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float t1 = t1s;
            float T = cr[h].T;
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const float t0 = t1;
                const float dt = calc_step(p.steps, t0);
                t1 = F_ADD(t0, dt);
                const float tm = F_MUL(F_ADD(t0, t1), 0.5f);
                if (tm > cr[h].far_) { cr[h].alive = 0; continue; }
                if (rows[h][s] < 0) continue;
                const float alpha = fminf(1.0f, fmaxf(0.0f, 1.0f - expf(-expf(sigma[h][s]) * dt)));
                if (alpha > p.scene.alpha_thre) { T *= 1.0f - alpha; ++visible; }
                if (T < 1e-4f) cr[h].alive = 0;
            }
            alive += cr[h].alive;
            CacheRay *out = p.rays + (size_t)tile * 64 + h * 32 + lane;
            out->T = T;
            out->alive = cr[h].alive;
        }
        const int n_visible = (int)__reduce_add_sync(FULL, (unsigned)visible);
        const int n_alive_post = (int)__reduce_add_sync(FULL, (unsigned)alive);
        if (lane == 0) {
            p.tile_need[ai] = n_visible > 0;
            p.tile_n_alive[ai] = n_alive_post;
        }
    }
}

/* Exclusive scan over a 1024-thread block; *total receives the block sum.
 * s_w must hold 33 ints. */
__device__ __forceinline__ int block_exclusive_scan(int v, int &total, int *s_w)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int u = __shfl_up_sync(FULL, inc, off);
        if (lane >= off) inc += u;
    }
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int w = s_w[lane];
        int wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int u = __shfl_up_sync(FULL, wi, off);
            if (lane >= off) wi += u;
        }
        s_w[lane] = wi - w;
        if (lane == 31) s_w[32] = wi;
    }
    __syncthreads();
    const int excl = s_w[wid] + inc - v;
    total = s_w[32];
    __syncthreads();
    return excl;
}

/* Deterministic slot assignment for one iteration (replaces the atomicAdd of
 * accumulateNew_cache_init_second_kernel, src/cache_renderer.cu:419-426):
 * the tiles needing a brick get consecutive slots in alive-list (= tile
 * index) order.  Applies the per-tile updates of :518-527 (block step
 * advances unless the allocation overflowed; the tile stays alive while it
 * has alive rays and did not overflow), emits the (tile, slot) fill jobs and
 * the next alive list, counts the iteration and clears the next one's rows.
 * One CTA of 1024 threads, ASSIGN_TILES consecutive tiles a thread: a scan's
 * barriers are its whole cost, and 32,400 tiles (1080p) took 32 rounds of
 * three scans at one tile a thread (100 us), 8 rounds of one now.  A slot's
 * place among the round's slots is its job's place too, and both lists' counts
 * go through one scan as the halves of a 64-bit sum; only a round in which the
 * slots run out, where tiles die, scans the alive tiles again. */
constexpr int ASSIGN_TILES = 4;

__device__ __forceinline__ unsigned long long block_exclusive_scan64(unsigned long long v, unsigned long long &total, unsigned long long *s_w)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long inc = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long u = __shfl_up_sync(FULL, inc, off);
        if (lane >= off) inc += u;
    }
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const unsigned long long w = s_w[lane];
        unsigned long long wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned long long u = __shfl_up_sync(FULL, wi, off);
            if (lane >= off) wi += u;
        }
        s_w[lane] = wi - w;
        if (lane == 31) s_w[32] = wi;
    }
    __syncthreads();
    const unsigned long long excl = s_w[wid] + inc - v;
    total = s_w[32];
    __syncthreads();
    return excl;
}

__global__ void __launch_bounds__(1024) cache_assign_kernel(CacheBuildParams p)
{
    after_previous();
    __shared__ unsigned long long s_w[33];
    const int n = *p.n_alive_tiles;
    int slot0 = *p.slot_counter, jobs0 = 0, alive0 = 0; /* the same in every thread */
    for (int c0 = 0; c0 < n; c0 += 1024 * ASSIGN_TILES) {
        const int a0 = c0 + threadIdx.x * ASSIGN_TILES;
        int tile[ASSIGN_TILES];
        bool processed[ASSIGN_TILES], need[ASSIGN_TILES], stays[ASSIGN_TILES];
        unsigned long long mine = 0; /* low half: slots needed; high half: tiles alive when every slot is granted */
#pragma unroll
        for (int q = 0; q < ASSIGN_TILES; ++q) {
            const int ai = a0 + q;
            tile[q] = ai < n ? p.alive_list[ai] : 0;
            processed[q] = ai < n && p.tile_processed[ai];
            need[q] = processed[q] && p.tile_need[ai];
            stays[q] = ai < n && (processed[q] ? p.tile_n_alive[ai] > 0 : p.tile_alive[tile[q]] != 0);
            mine += (need[q] ? 1ull : 0ull) + (stays[q] ? 1ull << 32 : 0ull);
        }
        unsigned long long total;
        unsigned long long before = block_exclusive_scan64(mine, total, s_w);
        int slot = slot0 + (int)(before & 0xffffffffull);
        const int n_need = (int)(total & 0xffffffffull);
        const bool runs_out = slot0 + n_need > p.capacity; /* block-uniform */
        if (runs_out) {
            int sl = slot;
            mine = 0;
#pragma unroll
            for (int q = 0; q < ASSIGN_TILES; ++q) {
                if (need[q] && sl++ >= p.capacity) stays[q] = false;
                mine += stays[q] ? 1ull << 32 : 0ull;
            }
            before = block_exclusive_scan64(mine, total, s_w);
        }
        int apos = alive0 + (int)(before >> 32);
#pragma unroll
        for (int q = 0; q < ASSIGN_TILES; ++q) {
            const int ai = a0 + q;
            if (ai >= n) break;
            const bool overflow = need[q] && slot >= p.capacity;
            if (processed[q]) {
                const int bstep = p.block_step[tile[q]];
                if (need[q]) {
                    const int tx = tile[q] % p.bX, ty = tile[q] / p.bX;
                    if (bstep < p.bZ) {
                        const size_t bidx = ((size_t)bstep * p.bY + ty) * p.bX + tx;
                        if (!overflow) {
                            const int sx = slot / (p.dY * p.dZ), sy = (slot - sx * p.dY * p.dZ) / p.dZ;
                            const int sz = slot - sx * p.dY * p.dZ - sy * p.dZ;
                            p.packed_index[bidx] = (sx << 20) | (sy << 10) | sz;  /* pack3D(to3D(slot)) */
                        } else {
                            p.packed_index[bidx] = -1;
                        }
                    } else {
                        atomicOr(p.guard, 8);  /* brick beyond the frustum depth */
                    }
                }
                p.block_step[tile[q]] = bstep + (overflow ? 0 : 1);
                p.tile_alive[tile[q]] = stays[q];
            }
            if (need[q]) {
                if (!overflow) {
                    p.jobs[2 * (jobs0 + slot - slot0)] = ai;
                    p.jobs[2 * (jobs0 + slot - slot0) + 1] = slot;
                }
                ++slot;
            }
            if (stays[q]) p.alive_list_next[apos++] = tile[q];
        }
        jobs0 += max(0, min(n_need, p.capacity - slot0));
        slot0 += n_need;
        alive0 += (int)(total >> 32);
    }
    if (threadIdx.x == 0) {
        *p.slot_counter = slot0;
        *p.n_jobs = jobs0;
        *p.n_alive_next = alive0;
        *p.build_row_counter = 0;
        if (n > 0) ++*p.n_iterations;
    }
}

/* The 512 voxels of each brick that got a slot, written straight from the
 * iteration's network rows (zeros where the brick has no sample): density
 * slot and latent 0 per interpol_variant
 * (accumulateNew_cache_init_second_kernel :459-507).  Runs after
 * cache_assign_kernel, which advanced the tile's block step past the brick. */
__global__ void __launch_bounds__(256) cache_fill_kernel(CacheBuildParams p)
{
    after_previous();
    __shared__ float s_dt[8];
    const int n_jobs = *p.n_jobs;
    const bool by_alpha = p.variant == VARIANT_ALPHA || p.variant == VARIANT_ALPHA_INTERMEDIATES;
    const bool lat0 = p.variant == VARIANT_DENSITY_INTERMEDIATES || p.variant == VARIANT_ALPHA_INTERMEDIATES;
    for (int j = blockIdx.x; j < n_jobs; j += gridDim.x) {
        const int ai = p.jobs[2 * j], slot = p.jobs[2 * j + 1];
        __syncthreads();
        if (threadIdx.x == 0) {
            const int bstep = p.block_step[p.alive_list[ai]] - 1;
            float t1 = t_from_step(p.steps, F_ADD((float)(bstep * 8), p.steps.near_i));
            for (int s = 0; s < 8; ++s) {
                const float dt = calc_step(p.steps, t1);
                s_dt[s] = dt;
                t1 = F_ADD(t1, dt);
            }
        }
        __syncthreads();
        const int *rof = p.build_row_of + (size_t)ai * 512;
        Voxel *dst = reinterpret_cast<Voxel *>(p.voxels) + (size_t)slot * 512;
        for (int i = threadIdx.x; i < 512; i += blockDim.x) {
            const int row = rof[i];
            Voxel v;
            v.pad0 = v.pad1 = 0.f;
            if (row >= 0) {
                const float sigma = expf(__half2float(p.build_den[row]));
                const float alpha = fminf(1.0f, fmaxf(0.0f, 1.0f - expf(-sigma * s_dt[i >> 6])));
                v.density = p.variant == VARIANT_INTERMEDIATES ? 0.f : by_alpha ? alpha : sigma; /* Intermediates: slot unwritten */
                v.isset = 1.0f;
                v.lat = p.build_lat[row];
                if (lat0) v.lat.x = (v.lat.x & 0xffff0000u) | (uint32_t)__half_as_ushort(__float2half_rn(v.density));
            } else {
                v.density = 0.f;
                v.isset = 0.f;
                v.lat = make_uint4(0, 0, 0, 0);
            }
            __stcs(reinterpret_cast<float4 *>(dst + i), make_float4(v.density, v.isset, 0.f, 0.f));
            __stcs(reinterpret_cast<uint4 *>(dst + i) + 1, v.lat);
        }
    }
}

/* writeImageBuffer_cache_init_kernel2, src/cache_renderer.cu:530-569:
 * known_ranges_to = t at the start of the tile's final depth brick. */
__global__ void __launch_bounds__(64) cache_known_ranges_kernel(CacheBuildParams p)
{
    const int tile = blockIdx.x, k = threadIdx.x;
    const int tx = tile % p.bX, ty = tile / p.bX;
    const int px = tx * 8 + (k & 7), py = ty * 8 + (k >> 3);
    if (px >= p.fW || py >= p.fH) return;
    p.known_ranges[(size_t)py * p.fW + px] = t_from_step(p.steps, F_ADD((float)(p.block_step[tile] * 8), p.steps.near_i));
}

/* compaction of the initially alive tiles (single CTA of 1024 threads) */
__global__ void __launch_bounds__(1024) cache_compact_kernel(CacheBuildParams p, int n_tiles)
{
    __shared__ int s_w[33];
    __shared__ int s_carry;
    const int tid = threadIdx.x;
    if (tid == 0) s_carry = 0;
    __syncthreads();
    for (int c0 = 0; c0 < n_tiles; c0 += 1024) {
        const int t = c0 + tid;
        const int a = (t < n_tiles && p.tile_alive[t]) ? 1 : 0;
        int total;
        const int pos = s_carry + block_exclusive_scan(a, total, s_w);
        if (a) p.alive_list[pos] = t;
        __syncthreads();
        if (tid == 0) s_carry += total;
        __syncthreads();
    }
    if (tid == 0) *p.n_alive_tiles = s_carry;
}

/* ------------------------------------------------------------------------- */
/* per-ray cache fill (CacheRenderer::initCache, src/cache_renderer.cu:571-928) */
/* ------------------------------------------------------------------------- */
/* known_ranges_to starts at StepsizeInfo::far, the RayPayload
 * termination_depth of rays that end neither by opacity nor by overflow
 * (initRayPayloads_common_kernel, src/renderer.cu:62-78) */
__global__ void pr_known_init_kernel(PerRayFillParams p)
{
    const int n = p.W * p.H;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p.known_ranges[i] = p.steps.far_;
}

/* the froxel brick of a sample of pixel id at the midpoint tm, or -1 past the
 * frustum depth (bin = floor(step_from_t(t_mid) - near_i), :598-604) */
__device__ __forceinline__ int pr_brick(const PerRayFillParams &p, int id, float tm, int &bin)
{
    bin = (int)floorf(F_SUB(step_from_t(p.steps, tm), p.steps.near_i));
    const int bz = bin >> 3;
    if (bin < 0 || bz >= p.bZ) return -1;
    const int x = id % p.W, y = id / p.W;
    return (bz * p.bY + (y >> 3)) * p.bX + (x >> 3);
}

/* accumulate_cache_init_first_kernel (:571-623): per alive ray, the bricks of
 * its visible samples of this sub-iteration, until the transmittance falls
 * below 1e-4 (unclamped density) */
__global__ void __launch_bounds__(128) pr_mark_kernel(PerRayFillParams p, int it)
{
    after_previous();
    const int n_alive = p.counters[it & 1];
    const RayState *states = p.states[it & 1];
    for (int base = blockIdx.x * blockDim.x; base < n_alive; base += gridDim.x * blockDim.x) {
        const int i = base + threadIdx.x;
        const bool valid = i < n_alive;
        const int id = valid ? states[i].cnt.x : 0;
        float T = valid ? states[i].acc.w : 1.f;
        bool ended = false;
        int row;
        RowWalk walk(valid ? p.ray_rows[i] : make_int2(0, 0), valid, p.by_sample);
        while (walk.step(row)) {
            if (row < 0 || ended) continue;
            const float density = expf(__half2float(p.den[row]));
            const float t0 = p.row_t0[row];
            const float dt = calc_step(p.steps, t0);
            const float t1 = F_ADD(t0, dt);
            const float tm = F_MUL(F_ADD(t0, t1), 0.5f);
            const float alpha = fminf(1.0f, fmaxf(0.0f, 1.0f - expf(-density * dt)));
            if (alpha > p.scene.alpha_thre) {
                T *= 1.0f - alpha;
                int bin;
                const int b = pr_brick(p, id, tm, bin);
                if (b < 0) { /* beyond the frustum depth: pr_write ends the ray here */
                    ended = true;
                    continue;
                }
                p.flag[b] = 1;
            }
            if (T < 1e-4f) ended = true;
        }
    }
}

/* reserveNewBricks_kernel (:775-805) made deterministic: per brick column,
 * the number of bricks marked in this sub-iteration that hold no slot yet.  A
 * warp per column, a lane per depth: a thread that walked its column's 200
 * depths alone waited for each in turn (18 us a launch at 640x360, 53 with the
 * reservation below; 4 and 14 now). */
__global__ void __launch_bounds__(256) pr_count_kernel(PerRayFillParams p)
{
    after_previous();
    const int n_cols = p.bX * p.bY, lane = threadIdx.x & 31;
    const size_t plane = (size_t)n_cols;
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (c >= n_cols) return; /* the whole warp */
    int n = 0;
    for (int z = lane; z < p.bZ; z += 32) {
        const size_t b = (size_t)z * plane + c;
        n += p.flag[b] && !p.set[b];
    }
    n = __reduce_add_sync(FULL, n);
    if (lane == 0) p.col_count[c] = n;
}

/* exclusive scan of the column counts from the slot counter (one CTA of 1024) */
__global__ void __launch_bounds__(1024) pr_scan_kernel(PerRayFillParams p)
{
    after_previous();
    __shared__ int s_w[33];
    __shared__ int s_carry;
    const int n_cols = p.bX * p.bY;
    if (threadIdx.x == 0) {
        s_carry = p.slot_counter[0];
        p.slot_counter[1] = s_carry;
    }
    __syncthreads();
    for (int c0 = 0; c0 < n_cols; c0 += 1024) {
        const int c = c0 + threadIdx.x;
        const int v = c < n_cols ? p.col_count[c] : 0;
        int total;
        const int ex = block_exclusive_scan(v, total, s_w);
        if (c < n_cols) p.col_base[c] = s_carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) s_carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) p.slot_counter[0] = s_carry;
}

/* slots in (column, depth) order; a slot beyond the capacity leaves the brick
 * without one (packed index -1), as the reference's overflow does; clears the
 * marks for the next sub-iteration */
__global__ void __launch_bounds__(256) pr_reserve_kernel(PerRayFillParams p)
{
    after_previous();
    const int n_cols = p.bX * p.bY, lane = threadIdx.x & 31;
    const size_t plane = (size_t)n_cols;
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (c >= n_cols || p.col_count[c] == 0) {
        /* no new brick: the marks alone are cleared */
        for (int z = lane; c < n_cols && z < p.bZ; z += 32) p.flag[(size_t)z * plane + c] = 0;
        return;
    }
    int first = p.col_base[c];
    for (int z0 = 0; z0 < p.bZ; z0 += 32) {
        const int z = z0 + lane;
        const size_t b = (size_t)z * plane + c;
        const bool marked = z < p.bZ && p.flag[b];
        const bool fresh = marked && !p.set[b];
        const unsigned m = __ballot_sync(FULL, fresh);
        if (marked) p.flag[b] = 0;
        if (fresh) {
            const int slot = first + __popc(m & lanes_below());
            if (slot < p.capacity) {
                const int sx = slot / (p.dY * p.dZ), sy = (slot - sx * p.dY * p.dZ) / p.dZ;
                const int sz = slot - sx * p.dY * p.dZ - sy * p.dZ;
                p.packed_index[b] = (sx << 20) | (sy << 10) | sz;
                p.set[b] = 1;
            } else {
                p.packed_index[b] = -1;
            }
        }
        first += __popc(m);
    }
}

/* the slots reserved in this sub-iteration start out empty (Cache::
 * setDataArraysZero, src/cache_renderer.cu:854) */
__global__ void __launch_bounds__(256) pr_zero_kernel(PerRayFillParams p)
{
    after_previous();
    const int s0 = min(p.slot_counter[1], p.capacity), s1 = min(p.slot_counter[0], p.capacity);
    uint4 *v = reinterpret_cast<uint4 *>(p.voxels);
    const size_t n = (size_t)(s1 - s0) * 1024;
    const size_t base = (size_t)s0 * 1024;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        v[base + i] = make_uint4(0, 0, 0, 0);
}

/* accumulate_cache_init_second_kernel (:625-773): per alive ray, the voxels of
 * its visible samples (density clamped to exp(10)), the density slot and
 * latent 0 per interpol_variant; a sample whose brick got no slot (or lies
 * beyond the frustum depth) ends the ray at its t0, transmittance below 1e-4
 * at its t1.  Rays that end write their termination depth to known_ranges_to
 * (writeImageBuffer_cache_init_kernel, :807-827); the others are compacted
 * into the next alive list. */
__global__ void __launch_bounds__(128) pr_write_kernel(PerRayFillParams p, int it)
{
    after_previous();
    const int n_alive = p.counters[it & 1];
    RayState *states = p.states[it & 1];
    RayState *next = p.states[(it + 1) & 1];
    const bool by_alpha = p.variant == VARIANT_ALPHA || p.variant == VARIANT_ALPHA_INTERMEDIATES;
    const bool lat0 = p.variant == VARIANT_DENSITY_INTERMEDIATES || p.variant == VARIANT_ALPHA_INTERMEDIATES;
    Voxel *vox = reinterpret_cast<Voxel *>(p.voxels);
    for (int base = blockIdx.x * blockDim.x; base < n_alive; base += gridDim.x * blockDim.x) {
        const int i = base + threadIdx.x;
        const bool valid = i < n_alive;
        bool alive = false, ended = false;
        RayState st;
        int id = 0, row;
        float T = 1.f, term = p.steps.far_;
        int2 rr = make_int2(0, 0);
        if (valid) {
            st = states[i];
            rr = p.ray_rows[i];
            id = st.cnt.x;
            T = st.acc.w;
            alive = !window_done(rr.y); /* the march ended the ray past its far bound */
            if (p.max_samples_per_ray > 0) {
                st.cnt2.z += window_rows(rr.y);
                if (st.cnt2.z > p.max_samples_per_ray) atomicOr(p.guard, 1);
            }
        }
        const int ws = __reduce_add_sync(0xffffffffu, window_steps(rr.y));
        if ((threadIdx.x & 31) == 0 && ws) atomicAdd(&p.stats->n_steps, (unsigned long long)ws);
        RowWalk walk(rr, valid, p.by_sample);
        while (walk.step(row)) {
            if (row >= 0 && !ended) {
                const float density = expf(fminf(__half2float(p.den[row]), 10.0f));
                const float t0 = p.row_t0[row];
                const float dt = calc_step(p.steps, t0);
                const float t1 = F_ADD(t0, dt);
                const float tm = F_MUL(F_ADD(t0, t1), 0.5f);
                const float alpha = fminf(1.0f, fmaxf(0.0f, 1.0f - expf(-density * dt)));
                if (alpha > p.scene.alpha_thre) {
                    T *= 1.0f - alpha;
                    int bin;
                    const int b = pr_brick(p, id, tm, bin);
                    const int packed = b >= 0 ? p.packed_index[b] : -1;
                    if (packed < 0) { /* no slot: the cache overflowed here */
                        alive = false;
                        ended = true;
                        term = t0;
                        continue;
                    }
                    const int x = id % p.W, y = id / p.W;
                    const int slot = ((packed >> 20) & 1023) * (p.dY * p.dZ) + ((packed >> 10) & 1023) * p.dZ + (packed & 1023);
                    Voxel v;
                    v.density = p.variant == VARIANT_INTERMEDIATES ? 0.f : by_alpha ? alpha : density;
                    v.isset = 1.0f;
                    v.pad0 = v.pad1 = 0.f;
                    v.lat = p.lat[row];
                    if (lat0) v.lat.x = (v.lat.x & 0xffff0000u) | (uint32_t)__half_as_ushort(__float2half_rn(v.density));
                    vox[(size_t)slot * 512 + (bin & 7) * 64 + (y & 7) * 8 + (x & 7)] = v;
                }
                if (T < 1e-4f) {
                    alive = false;
                    ended = true;
                    term = t1;
                }
            }
        }
        if (valid) {
            st.acc.w = T;
            if (!alive) p.known_ranges[id] = term;
        }
        const unsigned m = __ballot_sync(0xffffffffu, alive);
        int wbase = 0;
        if ((threadIdx.x & 31) == 0 && m) wbase = atomicAdd(p.counters + ((it + 1) & 1), __popc(m));
        wbase = __shfl_sync(0xffffffffu, wbase, 0);
        if (alive) next[wbase + __popc(m & lanes_below())] = st;
    }
}

}  // namespace fvc
