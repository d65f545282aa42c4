// trace.cu — one-scene traversal, shading and ray-generation kernels for
// sm_103a (the device functions are in trace_dev.cuh).
#include <cuda_runtime.h>
#include <stdint.h>

#include "rt_internal.cuh"
#include "trace.cuh"
#include "trace_quad.cuh"

namespace rt {

// ---------------------------------------------------------------------------
// fused per-pixel Whitted path (Renderer::render_to_framebuffer, one pixel
// per lane, persistent warps fetching 32 pixels at a time)
// ---------------------------------------------------------------------------
template <int THREADS, int MINB, bool REFR = false>
__global__ void __launch_bounds__(THREADS, MINB) k_render(RenderArgs a) {
    const SceneView S = a.scene;
    __shared__ BvhHeader sH;
    __shared__ rt_lights sL;
    if (threadIdx.x == 0) sH = *S.hdr;
    for (int i = threadIdx.x; i < (int)(sizeof(rt_lights) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&sL)[i] = reinterpret_cast<const uint32_t*>(&a.lights)[i];
    __syncthreads();
    const BvhHeader& H = sH;
    const int lane = threadIdx.x & 31;
    const int pixels = a.width * a.height;
    uint64_t n_sec = 0, n_shadow = 0, n_hits = 0, n_prim = 0;
    const int chunk = a.chunk;   // pixels a warp takes per fetch (multiple of 32)
    for (;;) {
        int base0 = 0;
        if (lane == 0) base0 = (int)atomicAdd(a.work_counter, (unsigned)chunk);
        base0 = __shfl_sync(0xffffffffu, base0, 0);
        if (base0 >= pixels) break;
        for (int base = base0; base < base0 + chunk && base < pixels; base += 32) {
        const int gid = base + lane;
        if (gid < pixels) {
            int x, y;
            pixel_of(warp_tile_order(gid, a.width, a.height), a.width, a.height, 32, x, y);
            const PixelResult pr = render_pixel<REFR>(S, H, sL, a.cam, x, y, a.width,
                                                             a.height, a.max_bounces, a.status);
            const uint32_t acc_r = pr.r, acc_g = pr.g, acc_b = pr.b;
            ++n_prim;
            n_sec += pr.secondary;
            n_shadow += pr.shadow;
            n_hits += pr.hits;
            const int pix = a.width * y + x;
            if (a.image_rgb) {
                a.image_rgb[3 * (size_t)pix] = acc_r;
                a.image_rgb[3 * (size_t)pix + 1] = acc_g;
                a.image_rgb[3 * (size_t)pix + 2] = acc_b;
            }
            reinterpret_cast<uchar4*>(a.rgba)[pix] =
                rgba8_of(make_uint3(acc_r, acc_g, acc_b), a.inv1e6);
        }
        }
    }
    if (a.stats) {
        n_prim = __reduce_add_sync(0xffffffffu, (unsigned)n_prim);
        n_sec = __reduce_add_sync(0xffffffffu, (unsigned)n_sec);
        n_shadow = __reduce_add_sync(0xffffffffu, (unsigned)n_shadow);
        n_hits = __reduce_add_sync(0xffffffffu, (unsigned)n_hits);
        if (lane == 0) {
            atomicAdd((unsigned long long*)&a.stats->primary_rays, (unsigned long long)n_prim);
            atomicAdd((unsigned long long*)&a.stats->secondary_rays, (unsigned long long)n_sec);
            atomicAdd((unsigned long long*)&a.stats->shadow_rays, (unsigned long long)n_shadow);
            atomicAdd((unsigned long long*)&a.stats->hits, (unsigned long long)n_hits);
        }
    }
}

// The pixel's sum, as it is and as RGBA8.
__device__ __forceinline__ void write_pixel(const RenderArgs& a, int pix, uint3 sum) {
    if (a.image_rgb) {
        uint32_t* q = a.image_rgb + 3 * (size_t)pix;
        q[0] = sum.x;
        q[1] = sum.y;
        q[2] = sum.z;
    }
    reinterpret_cast<uchar4*>(a.rgba)[pix] = rgba8_of(sum, a.inv1e6);
}

// ---------------------------------------------------------------------------
// k_render_quad: the same rays as k_render, a pixel's path by four lanes
// (trace_quad.cuh), for frames with too few pixels to fill the SMs: these take as
// long as the chain of a path's rays.  A warp takes `chunk` (at most eight)
// neighbouring pixels at a time; its (hit, light) tasks are spread over all
// eight places, so that lights and places without a path do not lengthen the
// chain (against one light after the other, 64 x 64 of 1.2 M triangles: 400 ->
// 114 us).  Render of 64 x 64 / 256 x 256, pooled and this: 1k triangles 48 -> 30 /
// 55 -> 49 us, 10k 168 -> 64 / 221 -> 152, 200k 211 -> 96 / 275 -> 185, a terrain
// of 1.2 M 291 -> 114 / 389 -> 300.  Six blocks per SM: with eight, spills, +8 %.
// ---------------------------------------------------------------------------
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_render_quad(RenderArgs a) {
    const SceneView S = a.scene;
    __shared__ BvhHeader sH;
    __shared__ rt_lights sL;
    __shared__ QuadStack stacks[THREADS / 4];
    __shared__ uint8_t tasks[THREADS / 32][8 * RT_MAX_LIGHTS];
    __shared__ unsigned blocks[THREADS / 32][8];
    if (threadIdx.x == 0) sH = *S.hdr;
    for (int i = threadIdx.x; i < (int)(sizeof(rt_lights) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&sL)[i] = reinterpret_cast<const uint32_t*>(&a.lights)[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const bool writer = (lane & 3) == 0;   // of the ray's four lanes
    int2* st = stacks[threadIdx.x / 4].e;
    uint8_t* list = tasks[threadIdx.x / 32];
    unsigned* blocked = blocks[threadIdx.x / 32];
    const int per = a.chunk;   // pixels of a warp
    const int pixels = a.width * a.height;
    unsigned n_sec = 0, n_hits = 0, n_prim = 0;
    for (;;) {
        int base = 0;
        if (lane == 0) base = (int)atomicAdd(a.work_counter, (unsigned)per);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= pixels) break;
        const int gid = base + lane / 4;
        const bool valid = gid < pixels && lane / 4 < per;
        bool live = valid;
        int x, y;
        pixel_of(warp_tile_order(min(gid, pixels - 1), a.width, a.height), a.width, a.height, 32, x, y);
        f3 o = mk3(a.cam.pos[0], a.cam.pos[1], a.cam.pos[2]);
        f3 d = primary_dir(a.cam, x, y, a.width, a.height, 0.0f, 0.0f);
        float tmin = 0.0f, tmax = 1e36f, contribution = 1.0f;
        uint3 sum = make_uint3(0u, 0u, 0u);
        n_prim += valid;
        for (int bounce = 0;; ++bounce) {
            const TRay r = make_tray(o, d, mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z), tmin);
            const Hit hit = closest_hit_quad(S, sH, r, tmax, live, st, a.status);
            live = live && hit.id >= 0;
            HitInfo hi{};
            rt_material mat{};
            if (live) {
                hi = complete_hit(S, o, d, hit);
                mat = S.mats[__ldg(&S.map[hit.id])];
            }
            uint32_t mask = 0;
            int nt = 0;
            for (int l = 0; l < sL.count; ++l) {
                const bool counts = live && !light_vanishes(sL.light[l], mat, hi.hp, hi.n, d);
                f3 dir;
                const bool reaches = counts && shadow_dir(sL.light[l], hi.hp, dir);
                if (counts && !reaches) mask |= 1u << l;
                const unsigned m = __ballot_sync(0xffffffffu, reaches && writer);
                if (reaches && writer)
                    list[nt + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(lane / 4 | l << 3);
                nt += __popc(m);
            }
            if (lane < 8) blocked[lane] = 0u;
            __syncwarp();
            for (int t0 = 0; t0 < nt; t0 += 8) {
                const bool task = t0 + lane / 4 < nt;
                const int e = task ? list[t0 + lane / 4] : 0, from = (e & 7) * 4;
                const f3 hp = mk3(__shfl_sync(0xffffffffu, hi.hp.x, from),
                                  __shfl_sync(0xffffffffu, hi.hp.y, from),
                                  __shfl_sync(0xffffffffu, hi.hp.z, from));
                f3 dir = mk3(0.f, 0.f, 0.f);
                if (task) shadow_dir(sL.light[e >> 3], hp, dir);
                const TRay sr = make_tray(hp, dir, mk3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z), 0.01f);
                if (any_hit_quad(S, sH, sr, 1e37f, task, st, a.status) && writer)
                    atomicOr(&blocked[e & 7], 1u << (e >> 3));
            }
            __syncwarp();
            mask |= blocked[lane / 4];
            __syncwarp();
            if (live) {
                ++n_hits;
                const uint3 c = shade_hit(sL, mat, hi.hp, hi.n, d, contribution, mask);
                sum.x += c.x;
                sum.y += c.y;
                sum.z += c.z;
                live = bounce < a.max_bounces && mat.reflectiveness > 0.0f;
                if (live) {
                    f3 nd;
                    reflect_ray(d, hi.n, nd);
                    contribution = contribution * mat.reflectiveness * 1.0f;
                    o = hi.hp;
                    d = nd;
                    tmin = 0.0001f;
                    tmax = 1e37f;
                    ++n_sec;
                }
            }
            if (!__any_sync(0xffffffffu, live)) break;
        }
        if (valid && writer) write_pixel(a, a.width * y + x, sum);
    }
    if (a.stats) {
        n_prim = __reduce_add_sync(0xffffffffu, writer ? n_prim : 0u);
        n_sec = __reduce_add_sync(0xffffffffu, writer ? n_sec : 0u);
        n_hits = __reduce_add_sync(0xffffffffu, writer ? n_hits : 0u);
        if (lane == 0) {
            atomicAdd((unsigned long long*)&a.stats->primary_rays, (unsigned long long)n_prim);
            atomicAdd((unsigned long long*)&a.stats->secondary_rays, (unsigned long long)n_sec);
            atomicAdd((unsigned long long*)&a.stats->shadow_rays,
                      (unsigned long long)n_hits * (unsigned)sL.count);
            atomicAdd((unsigned long long*)&a.stats->hits, (unsigned long long)n_hits);
        }
    }
}

// ---------------------------------------------------------------------------
// k_render_pool: the same rays as k_render, scheduled so that a warp's lanes
// stay busy.  A warp takes a tile of 32 pixels and traces their primary rays
// together (coherent); the hits' shadow rays are traced as a dense list of
// (hit, light) tasks; each hit is shaded and, if the path continues, its
// reflection ray goes into the warp's pool in shared memory, which is traced
// 32 rays at a time whichever pixels they come from.  A pixel has one ray on
// the way at a time, so its fixed-point sum travels with the ray, and the lane
// that ends the path writes the pixel: no accumulation buffer to clear, add to
// and convert afterwards (11 % of a thumbnail, 0.5-1.5 % of 1920 x 1080 frames).
// Every ray is
// traversed and shaded exactly as in render_pixel, so the image is
// bit-identical to k_render's.
// ---------------------------------------------------------------------------
namespace {
constexpr int POOL = 64;   // rays a warp can hold: < 32 left + 32 of the current step

// The rays of a warp.  The ones left wait in the first places; those of
// the current step keep or take the places above, where a hit puts its point
// over its ray's origin, until the step's own reflection rays are written over
// them.  The L1 shares the SM's memory with this: a further 1.1 KB per warp (the
// hits in arrays of their own) cost 1-3 % of a frame.
struct WarpPool {
    float ro[3][POOL], rd[3][POOL], rc[POOL];   // origin or hit point, direction, contribution
    int rpix[POOL];
    uint8_t rbounce[POOL];                      // at most 64
    uint32_t racc[3][POOL];                     // the pixel's sum so far
    float hn[3][32];                            // hits of the current step
    int hid[32];
    unsigned hmask[32];
    uint8_t hslot[32];                          // their places
    uint8_t task[32 * RT_MAX_LIGHTS];           // shadow tasks that need a ray
};
}  // namespace

template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_render_pool(RenderArgs a) {
    const SceneView S = a.scene;
    __shared__ BvhHeader sH;
    __shared__ rt_lights sL;
    __shared__ WarpPool sQ[THREADS / 32];
    if (threadIdx.x == 0) sH = *S.hdr;
    for (int i = threadIdx.x; i < (int)(sizeof(rt_lights) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&sL)[i] = reinterpret_cast<const uint32_t*>(&a.lights)[i];
    const int lane = threadIdx.x & 31;
    WarpPool& Q = sQ[threadIdx.x >> 5];
    __syncthreads();
    const BvhHeader& H = sH;
    const int pixels = a.width * a.height;
    const unsigned lt = (1u << lane) - 1u;
    uint64_t n_sec = 0, n_shadow = 0, n_hits = 0, n_prim = 0;
    bool tiles = true;
    int pn = 0;   // rays waiting in the pool
    for (;;) {
        // 1. rays to trace: a full batch from the pool, else a new tile
        //    of primary rays, else what is left in the pool
        bool have = false;
        f3 o = mk3(0.f, 0.f, 0.f), d = o;
        float tmin = 0.0f, tmax = 1e36f;
        int tile_pix = -1;      // a primary ray's pixel
        int first = pn;         // place of the step's first ray
        if (pn >= 32 || (!tiles && pn > 0)) {
            const int k = min(32, pn);
            first = pn - k;
            have = lane < k;
            if (have) {
                const int j = first + lane;
                o = mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]);
                d = mk3(Q.rd[0][j], Q.rd[1][j], Q.rd[2][j]);
                tmin = 0.0001f;
                tmax = 1e37f;
            }
        } else if (tiles) {
            int base = 0;
            if (lane == 0) base = (int)atomicAdd(a.work_counter, 32u);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= pixels) {
                tiles = false;
                continue;
            }
            const int gid = base + lane;
            have = gid < pixels;
            if (have) {
                int x, y;
                pixel_of(warp_tile_order(gid, a.width, a.height), a.width, a.height, 32, x, y);
                tile_pix = a.width * y + x;
                o = mk3(a.cam.pos[0], a.cam.pos[1], a.cam.pos[2]);
                d = primary_dir(a.cam, x, y, a.width, a.height, 0.0f, 0.0f);
                ++n_prim;
            }
        } else {
            break;
        }
        // 2. closest hits; the hits are listed in the warp's hit slots
        bool hit_ok = false;
        Hit hit{-1, 0.f, 0.f, 0.f};
        if (have) {
            const TRay r = make_tray(o, d, mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z), tmin);
            hit = closest_hit<false, false>(S, H, r, tmax, a.status);
            hit_ok = hit.id >= 0;
        }
        const unsigned hm = __ballot_sync(0xffffffffu, hit_ok);
        const int nh = __popc(hm);
        const int at = first + lane;
        if (hit_ok) {
            const int k = __popc(hm & lt);
            const HitInfo hi = complete_hit(S, o, d, hit);
            Q.ro[0][at] = hi.hp.x; Q.ro[1][at] = hi.hp.y; Q.ro[2][at] = hi.hp.z;
            Q.hn[0][k] = hi.n.x; Q.hn[1][k] = hi.n.y; Q.hn[2][k] = hi.n.z;
            Q.hid[k] = hit.id;
            Q.hslot[k] = (uint8_t)at;
            Q.hmask[k] = 0u;
            if (tile_pix >= 0) {
                Q.rd[0][at] = d.x; Q.rd[1][at] = d.y; Q.rd[2][at] = d.z;
                Q.rc[at] = 1.0f;
                Q.rpix[at] = tile_pix;
                Q.rbounce[at] = 0;
                Q.racc[0][at] = Q.racc[1][at] = Q.racc[2][at] = 0u;
            }
        } else if (have) {   // the path ends in the void
            if (tile_pix >= 0)
                write_pixel(a, tile_pix, make_uint3(0u, 0u, 0u));
            else
                write_pixel(a, Q.rpix[at],
                            make_uint3(Q.racc[0][at], Q.racc[1][at], Q.racc[2][at]));
        }
        __syncwarp();
        // 3. shadow rays of every hit and light, 32 at a time
        const int nl = sL.count;
        // light-major (shadow_tasks): neighbouring lanes trace toward the same
        // light from neighbouring hits (coherent paths: 3 % faster on the
        // mid-scale frame with 2 lights, 10 % on the stress pose with 3, than
        // a hit's lights on neighbouring lanes); the tasks that need a ray
        // are traced densely
        shadow_tasks(
            nh, nl, Q.task,
            [&](int k, int l) {
                const int j = Q.hslot[k];
                return !light_vanishes(sL.light[l], S.mats[__ldg(&S.map[Q.hid[k]])],
                                       mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]),
                                       mk3(Q.hn[0][k], Q.hn[1][k], Q.hn[2][k]),
                                       mk3(Q.rd[0][j], Q.rd[1][j], Q.rd[2][j]));
            },
            [&](int k, int l) {
                const int j = Q.hslot[k];
                if (occluded<false, false, true>(S, H, sL.light[l],
                                                 mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]), a.status))
                    atomicOr(&Q.hmask[k], 1u << l);
            });
        __syncwarp();
        // 4. shading; continuing paths put their reflection ray into the pool
        bool push = false;
        f3 np = mk3(0.f, 0.f, 0.f), nd = np;
        float nc = 0.f;
        int npix = 0, nbounce = 0;
        uint3 sum = make_uint3(0u, 0u, 0u);
        if (lane < nh) {
            const int k = lane, j = Q.hslot[k];
            const f3 p = mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]);
            const f3 n = mk3(Q.hn[0][k], Q.hn[1][k], Q.hn[2][k]);
            const f3 dk = mk3(Q.rd[0][j], Q.rd[1][j], Q.rd[2][j]);
            const float ck = Q.rc[j];
            const rt_material mat = S.mats[__ldg(&S.map[Q.hid[k]])];
            const uint3 col = shade_hit(sL, mat, p, n, dk, ck, Q.hmask[k]);
            npix = Q.rpix[j];
            sum = make_uint3(Q.racc[0][j] + col.x, Q.racc[1][j] + col.y, Q.racc[2][j] + col.z);
            ++n_hits;
            n_shadow += (uint32_t)nl;
            const int bk = Q.rbounce[j];
            if (bk != a.max_bounces && mat.reflectiveness > 0.0f) {
                reflect_ray(dk, n, nd);
                np = p;
                nc = ck * mat.reflectiveness * 1.0f;
                nbounce = bk + 1;
                push = true;
                ++n_sec;
            } else {
                write_pixel(a, npix, sum);
            }
        }
        const unsigned pm = __ballot_sync(0xffffffffu, push);
        __syncwarp();   // every lane has read its hit's place
        if (push) {
            const int j = first + __popc(pm & lt);
            Q.ro[0][j] = np.x; Q.ro[1][j] = np.y; Q.ro[2][j] = np.z;
            Q.rd[0][j] = nd.x; Q.rd[1][j] = nd.y; Q.rd[2][j] = nd.z;
            Q.rc[j] = nc;
            Q.rpix[j] = npix;
            Q.rbounce[j] = (uint8_t)nbounce;
            Q.racc[0][j] = sum.x; Q.racc[1][j] = sum.y; Q.racc[2][j] = sum.z;
        }
        pn = first + __popc(pm);
        __syncwarp();
    }
    if (a.stats) {
        n_prim = __reduce_add_sync(0xffffffffu, (unsigned)n_prim);
        n_sec = __reduce_add_sync(0xffffffffu, (unsigned)n_sec);
        n_shadow = __reduce_add_sync(0xffffffffu, (unsigned)n_shadow);
        n_hits = __reduce_add_sync(0xffffffffu, (unsigned)n_hits);
        if (lane == 0) {
            atomicAdd((unsigned long long*)&a.stats->primary_rays, (unsigned long long)n_prim);
            atomicAdd((unsigned long long*)&a.stats->secondary_rays, (unsigned long long)n_sec);
            atomicAdd((unsigned long long*)&a.stats->shadow_rays, (unsigned long long)n_shadow);
            atomicAdd((unsigned long long*)&a.stats->hits, (unsigned long long)n_hits);
        }
    }
}

// ---------------------------------------------------------------------------
// k_render_pool_refr: k_render_pool for scenes with refracting materials.  A
// hit may continue two rays (the refracted one, contribution * reflectiveness
// * (1 - R), and the reflected one, * R, as generate_secondary_rays_disc
// makes them), and both go into the warp's pool.  The pool is taken from the
// top (last in, first out), so it holds at most 32 (max_bounces + 2) rays;
// it is sized for max_bounces <= MAXB (deeper frames use a larger pool or
// the ray-tree variant) and a push beyond it raises RT_DEV_OVERFLOW instead
// of writing.  Sums are integers, so the image is the ray-tree variant's.
// ---------------------------------------------------------------------------
namespace {
template <int RPOOL>
struct RefrPool {   // as WarpPool
    float ro[3][RPOOL], rd[3][RPOOL], rc[RPOOL];
    int rpix[RPOOL];
    uint8_t rbounce[RPOOL];
    float hn[3][32];
    int hid[32];
    unsigned hmask[32];
    uint8_t hslot[32], hinv[32];
    uint8_t task[32 * RT_MAX_LIGHTS];   // shadow tasks that need a ray
};
}  // namespace

template <int THREADS, int MINB, int MAXB>
__global__ void __launch_bounds__(THREADS, MINB) k_render_pool_refr(RenderArgs a) {
    constexpr int RPOOL = 32 * (MAXB + 2);
    static_assert(RPOOL <= 256, "places of the pool in 8 bits");
    const SceneView S = a.scene;
    __shared__ BvhHeader sH;
    __shared__ rt_lights sL;
    __shared__ RefrPool<RPOOL> sQ[THREADS / 32];
    if (threadIdx.x == 0) sH = *S.hdr;
    for (int i = threadIdx.x; i < (int)(sizeof(rt_lights) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&sL)[i] = reinterpret_cast<const uint32_t*>(&a.lights)[i];
    const int lane = threadIdx.x & 31;
    RefrPool<RPOOL>& Q = sQ[threadIdx.x >> 5];
    __syncthreads();
    const BvhHeader& H = sH;
    const int pixels = a.width * a.height;
    const unsigned lt = (1u << lane) - 1u;
    uint64_t n_sec = 0, n_shadow = 0, n_hits = 0, n_prim = 0;
    bool tiles = true;
    int pn = 0;   // rays waiting in the pool
    for (;;) {
        bool have = false;
        f3 o = mk3(0.f, 0.f, 0.f), d = o;
        float tmin = 0.0f, tmax = 1e36f;
        int tile_pix = -1;      // a primary ray's pixel
        int first = pn;         // place of the step's first ray
        if (pn >= 32 || (!tiles && pn > 0)) {
            const int k = min(32, pn);
            first = pn - k;
            have = lane < k;
            if (have) {
                const int j = first + lane;
                o = mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]);
                d = mk3(Q.rd[0][j], Q.rd[1][j], Q.rd[2][j]);
                tmin = 0.0001f;
                tmax = 1e37f;
            }
        } else if (tiles) {
            int base = 0;
            if (lane == 0) base = (int)atomicAdd(a.work_counter, 32u);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= pixels) {
                tiles = false;
                continue;
            }
            const int gid = base + lane;
            have = gid < pixels;
            if (have) {
                int x, y;
                pixel_of(warp_tile_order(gid, a.width, a.height), a.width, a.height, 32, x, y);
                tile_pix = a.width * y + x;
                o = mk3(a.cam.pos[0], a.cam.pos[1], a.cam.pos[2]);
                d = primary_dir(a.cam, x, y, a.width, a.height, 0.0f, 0.0f);
                ++n_prim;
            }
        } else {
            break;
        }
        bool hit_ok = false;
        Hit hit{-1, 0.f, 0.f, 0.f};
        if (have) {
            const TRay r = make_tray(o, d, mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z), tmin);
            hit = closest_hit<false, true>(S, H, r, tmax, a.status);
            hit_ok = hit.id >= 0;
        }
        const unsigned hm = __ballot_sync(0xffffffffu, hit_ok);
        const int nh = __popc(hm);
        const int at = first + lane;
        if (hit_ok) {
            const int k = __popc(hm & lt);
            const HitInfo hi = complete_hit(S, o, d, hit);
            Q.ro[0][at] = hi.hp.x; Q.ro[1][at] = hi.hp.y; Q.ro[2][at] = hi.hp.z;
            Q.hn[0][k] = hi.n.x; Q.hn[1][k] = hi.n.y; Q.hn[2][k] = hi.n.z;
            Q.hid[k] = hit.id;
            Q.hinv[k] = hi.inverse_n;
            Q.hslot[k] = (uint8_t)at;
            Q.hmask[k] = 0u;
            if (tile_pix >= 0) {
                Q.rd[0][at] = d.x; Q.rd[1][at] = d.y; Q.rd[2][at] = d.z;
                Q.rc[at] = 1.0f;
                Q.rpix[at] = tile_pix;
                Q.rbounce[at] = 0;
            }
        }
        __syncwarp();
        const int nl = sL.count;
        shadow_tasks(   // light-major, as k_render_pool
            nh, nl, Q.task,
            [&](int k, int l) {
                const int j = Q.hslot[k];
                return !light_vanishes(sL.light[l], S.mats[__ldg(&S.map[Q.hid[k]])],
                                       mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]),
                                       mk3(Q.hn[0][k], Q.hn[1][k], Q.hn[2][k]),
                                       mk3(Q.rd[0][j], Q.rd[1][j], Q.rd[2][j]));
            },
            [&](int k, int l) {
                const int j = Q.hslot[k];
                if (occluded<false, true>(S, H, sL.light[l],
                                          mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]), a.status))
                    atomicOr(&Q.hmask[k], 1u << l);
            });
        __syncwarp();
        bool push = false, push_t = false;
        f3 np = mk3(0.f, 0.f, 0.f), nd = np, td = np;
        float nc = 0.f, tc = 0.f;
        int npix = 0, nbounce = 0;
        if (lane < nh) {
            const int k = lane, j = Q.hslot[k];
            const f3 p = mk3(Q.ro[0][j], Q.ro[1][j], Q.ro[2][j]);
            const f3 n = mk3(Q.hn[0][k], Q.hn[1][k], Q.hn[2][k]);
            const f3 dk = mk3(Q.rd[0][j], Q.rd[1][j], Q.rd[2][j]);
            const float ck = Q.rc[j];
            const rt_material mat = S.mats[__ldg(&S.map[Q.hid[k]])];
            const uint3 col = shade_hit(sL, mat, p, n, dk, ck, Q.hmask[k]);
            npix = Q.rpix[j];
            if (col.x | col.y | col.z) {   // a zero colour adds nothing
                atomicAdd(&a.accum[3 * (size_t)npix], col.x);
                atomicAdd(&a.accum[3 * (size_t)npix + 1], col.y);
                atomicAdd(&a.accum[3 * (size_t)npix + 2], col.z);
            }
            ++n_hits;
            n_shadow += (uint32_t)nl;
            const int bk = Q.rbounce[j];
            if (bk < a.max_bounces) {
                float R = 1.0f;
                if (mat.refractive_index > 0.0f &&
                    refract_ray(dk, n, Q.hinv[k] != 0, mat.refractive_index, R, td)) {
                    tc = ck * mat.reflectiveness * (1.0f - R);
                    push_t = true;
                }
                if (mat.reflectiveness > 0.0f) {
                    reflect_ray(dk, n, nd);
                    nc = ck * mat.reflectiveness * R;
                    push = true;
                }
                np = p;
                nbounce = bk + 1;
            }
        }
        const unsigned pm = __ballot_sync(0xffffffffu, push);
        const unsigned pt = __ballot_sync(0xffffffffu, push_t);
        __syncwarp();   // every lane has read its hit's place
        auto put = [&](int j, f3 dir, float contribution) {
            if (j >= RPOOL) {
                atomicOr(a.status, RT_DEV_OVERFLOW);
                return;
            }
            Q.ro[0][j] = np.x; Q.ro[1][j] = np.y; Q.ro[2][j] = np.z;
            Q.rd[0][j] = dir.x; Q.rd[1][j] = dir.y; Q.rd[2][j] = dir.z;
            Q.rc[j] = contribution;
            Q.rpix[j] = npix;
            Q.rbounce[j] = (uint8_t)nbounce;
            ++n_sec;
        };
        if (push) put(first + __popc(pm & lt), nd, nc);
        if (push_t) put(first + __popc(pm) + __popc(pt & lt), td, tc);
        pn = min(RPOOL, first + __popc(pm) + __popc(pt));
        __syncwarp();
    }
    if (a.stats) {
        n_prim = __reduce_add_sync(0xffffffffu, (unsigned)n_prim);
        n_sec = __reduce_add_sync(0xffffffffu, (unsigned)n_sec);
        n_shadow = __reduce_add_sync(0xffffffffu, (unsigned)n_shadow);
        n_hits = __reduce_add_sync(0xffffffffu, (unsigned)n_hits);
        if (lane == 0) {
            atomicAdd((unsigned long long*)&a.stats->primary_rays, (unsigned long long)n_prim);
            atomicAdd((unsigned long long*)&a.stats->secondary_rays, (unsigned long long)n_sec);
            atomicAdd((unsigned long long*)&a.stats->shadow_rays, (unsigned long long)n_shadow);
            atomicAdd((unsigned long long*)&a.stats->hits, (unsigned long long)n_hits);
        }
    }
}

// ---------------------------------------------------------------------------
// stage-wise kernels on reference-layout buffers
// ---------------------------------------------------------------------------
// The stages' samples (80 B) and hits (64 B) are arrays of records that a lane
// handles one of.  Read or written word by word, each access of a warp falls
// into 32 sectors; the records of a warp go through shared memory instead, in
// accesses of 32 neighbouring words.  Words, because the callers' arrays need
// no more than a word's alignment.  A pitch of 20 words lets eight lanes' 16-byte
// parts meet each bank once.  k_gen_primary, 1000 x 701: 60 -> 14 us.
constexpr int STAGE_PITCH = 20;

// The first `cnt` (at most 32) records at g to the warp's stage.
template <int WORDS, int RECORDS = 32>
__device__ __forceinline__ void stage_in(float* sm, const void* g, int cnt) {
    const float* q = static_cast<const float*>(g);
    const int lane = threadIdx.x & 31;
    constexpr int TURNS = WORDS * RECORDS / 32;
    float v[TURNS];
#pragma unroll
    for (int k = 0; k < TURNS; ++k)
        if (32 * k + lane < cnt * WORDS) v[k] = q[32 * k + lane];
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int w = 32 * k + lane;
        if (w < cnt * WORDS) sm[w / WORDS * STAGE_PITCH + w % WORDS] = v[k];
    }
    __syncwarp();
}

// The records in `mask` (a bit for each, 32 / RECORDS bits apart) from the
// warp's stage to g.
template <int WORDS, int RECORDS = 32>
__device__ __forceinline__ void stage_out(const float* sm, void* g, unsigned mask) {
    float* q = static_cast<float*>(g);
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < WORDS * RECORDS / 32; ++k) {
        const int w = 32 * k + lane;
        if (mask >> (w / WORDS * (32 / RECORDS)) & 1) q[w] = sm[w / WORDS * STAGE_PITCH + w % WORDS];
    }
}

__device__ __forceinline__ void put4(float* sm, float x, float y, float z, float w) {
    *reinterpret_cast<float4*>(sm) = make_float4(x, y, z, w);
}

__global__ void __launch_bounds__(256) k_gen_primary(rt_camera cam, int w, int h, int q,
                                                     const rt_pixel_sample* ps, size_t count,
                                                     size_t offset, rt_sample* out) {
    __shared__ __align__(16) float stage[256 * STAGE_PITCH];
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const unsigned mask = __ballot_sync(0xffffffffu, k < count);
    float* sm = stage + threadIdx.x * STAGE_PITCH;
    if (k < count) {
        const int gid = (int)(offset + k);
        const int pixels = w * h;
        rt_pixel_sample p = {0.f, 0.f, 1.f};
        if (ps) p = ps[gid / pixels];
        int x, y;
        pixel_of(gid, w, h, q, x, y);
        const f3 d = primary_dir(cam, x, y, w, h, p.ox, p.oy);
        put4(sm, cam.pos[0], cam.pos[1], cam.pos[2], 0.f);
        put4(sm + 4, d.x, d.y, d.z, 0.f);
        put4(sm + 8, 1.0f / d.x, 1.0f / d.y, 1.0f / d.z, 0.f);
        put4(sm + 12, 0.0f, 1e36f, 0.f, 0.f);
        put4(sm + 16, __int_as_float(w * y + x), p.contribution, 0.f, 0.f);
    }
    const int lane = threadIdx.x & 31;
    if (mask) stage_out<20>(sm - lane * STAGE_PITCH, out + (k - lane), mask);
}

__device__ __forceinline__ f3 f3_of(const float* v) { return mk3(v[0], v[1], v[2]); }

// A warp takes `per` rays: 32, or with QUAD up to eight, by four lanes each
// (trace_quad.cuh).
template <bool QUAD>
__global__ void __launch_bounds__(128) k_trace(SceneView S, const rt_sample* __restrict__ smp,
                                               int n, rt_hit* __restrict__ hits,
                                               uint32_t* status, int per) {
    constexpr int RAYS = QUAD ? 8 : 32;   // places of a warp
    __shared__ BvhHeader sH;
    __shared__ __align__(16) float stage[4 * RAYS * STAGE_PITCH];
    __shared__ QuadStack stacks[QUAD ? 4 * RAYS : 1];
    if (threadIdx.x == 0) sH = *S.hdr;
    __syncthreads();
    const int lane = threadIdx.x & 31, ray_of = threadIdx.x / (32 / RAYS);   // in the block
    const int base = blockIdx.x * 4 * per + threadIdx.x / 32 * per;
    if (base >= n) return;
    n = min(per, n - base);   // this warp's rays (n may be the largest int)
    const int i = ray_of % RAYS;
    float* sm = stage + ray_of * STAGE_PITCH;
    float* warp = sm - ray_of % RAYS * STAGE_PITCH;
    hits += base;
    stage_in<20, RAYS>(warp, smp + base, n);
    const rt_ray& ray = *reinterpret_cast<const rt_ray*>(sm);
    const f3 o = f3_of(ray.ori), d = f3_of(ray.dir);
    bool hit = false;
    if (QUAD || i < n) {
        const TRay r = make_tray(o, d, f3_of(ray.inv_dir), ray.tmin);
        const float tmax = ray.tmax;
        Hit h;
        if (QUAD)
            h = closest_hit_quad(S, sH, r, tmax, i < n, stacks[QUAD ? ray_of : 0].e, status);
        else
            h = closest_hit<true, true, true>(S, sH, r, tmax, status);
        const bool mine = i < n && (!QUAD || lane % 4 == 0);   // one lane writes
        hit = mine && h.id >= 0;
        if (hit) {
            const HitInfo hi = complete_hit(S, o, d, h);
            const uint32_t head = 1u | (uint32_t)hits[i].shadow_hit << 8 | (uint32_t)hi.inverse_n << 16;
            put4(sm, __uint_as_float(head), h.t, __int_as_float(h.id), 0.f);
            put4(sm + 4, 0.f, 0.f, 0.f, 0.f);
            put4(sm + 8, hi.n.x, hi.n.y, hi.n.z, 0.f);
            put4(sm + 12, hi.hp.x, hi.hp.y, hi.hp.z, 0.f);
        } else if (mine) {
            hits[i].hit = 0;
        }
    }
    stage_out<16, RAYS>(warp, hits, __ballot_sync(0xffffffffu, hit));
}

template <bool QUAD>
__global__ void __launch_bounds__(128) k_shadow(SceneView S, rt_lights Ls, int n,
                                                rt_hit* __restrict__ hits, uint32_t* status, int per) {
    constexpr int RAYS = QUAD ? 8 : 32;   // places of a warp
    __shared__ BvhHeader sH;
    __shared__ __align__(16) float stage[4 * RAYS * STAGE_PITCH];
    __shared__ QuadStack stacks[QUAD ? 4 * RAYS : 1];
    if (threadIdx.x == 0) sH = *S.hdr;
    __syncthreads();
    const int lane = threadIdx.x & 31, ray_of = threadIdx.x / (32 / RAYS);   // in the block
    const int base = blockIdx.x * 4 * per + threadIdx.x / 32 * per;
    if (base >= n) return;
    n = min(per, n - base);   // this warp's rays (n may be the largest int)
    const int i = ray_of % RAYS;
    const float* sm = stage + ray_of * STAGE_PITCH;
    hits += base;
    stage_in<16, RAYS>(stage + (ray_of - ray_of % RAYS) * STAGE_PITCH, hits, n);
    const rt_hit& h = *reinterpret_cast<const rt_hit*>(sm);
    const bool hit = i < n && h.hit;
    const f3 hp = f3_of(h.hit_point);
    uint32_t mask = 0;
    if (QUAD) {
        for (int l = 0; l < Ls.count; ++l) {
            f3 dir = mk3(0.f, 0.f, 0.f);
            const bool live = hit && shadow_dir(Ls.light[l], hp, dir);
            const f3 inv = mk3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
            const TRay r = make_tray(hp, dir, inv, 0.01f);
            if (any_hit_quad(S, sH, r, 1e37f, live, stacks[QUAD ? ray_of : 0].e, status) || !live)
                mask |= 1u << l;
        }
        if (hit && lane % 4 == 0) hits[i].shadow_hit = (uint8_t)mask;
        return;
    }
    if (!hit) return;
    for (int l = 0; l < Ls.count; ++l)
        if (occluded<true, true, true>(S, sH, Ls.light[l], hp, status)) mask |= 1u << l;
    hits[i].shadow_hit = (uint8_t)mask;
}

__global__ void __launch_bounds__(128) k_shade(SceneView S, rt_lights Ls,
                                               const rt_sample* __restrict__ smp,
                                               const rt_hit* __restrict__ hits, int n,
                                               uint32_t* __restrict__ image) {
    __shared__ __align__(16) float stage[2][128 * STAGE_PITCH];
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, base = i - lane;
    if (base >= n) return;
    const int at = threadIdx.x * STAGE_PITCH, warp = at - lane * STAGE_PITCH;
    stage_in<16>(stage[0] + warp, hits + base, min(32, n - base));
    const rt_hit& h = *reinterpret_cast<const rt_hit*>(stage[0] + at);
    const bool hit = i < n && h.hit;
    if (!__any_sync(0xffffffffu, hit)) return;
    stage_in<20>(stage[1] + warp, smp + base, min(32, n - base));
    if (!hit) return;
    const rt_sample& sp = *reinterpret_cast<const rt_sample*>(stage[1] + at);
    const rt_material mat = S.mats[__ldg(&S.map[h.id])];
    const uint3 c = shade_hit(Ls, mat, f3_of(h.hit_point), f3_of(h.n), f3_of(sp.ray.dir),
                              sp.contribution, h.shadow_hit);
    uint32_t* px = image + 3 * (size_t)sp.pixel;
    atomicAdd(px, c.x);
    atomicAdd(px + 1, c.y);
    atomicAdd(px + 2, c.z);
}

// Secondary generation (the reference's mark / scan / generate of
// generate_secondary_rays_disc): flags -> per-block counts -> block offsets
// -> emit, in input order.  Reflected rays take the first slots, refracted
// rays the slots after all of them; a ray whose slot is at or beyond max_out
// is dropped, and a hit whose refracted slot is beyond it keeps R = 1 for its
// reflected ray, as in the kernel.
__device__ __forceinline__ void sec_flags(const SceneView& S, const rt_sample& smp, const rt_hit& h,
                                          bool& refl, bool& refr, rt_material& mat) {
    refl = refr = false;
    if (!h.hit) return;
    mat = S.mats[__ldg(&S.map[h.id])];
    refl = mat.reflectiveness > 0.0f;
    if (mat.refractive_index > 0.0f) {
        float R;
        f3 td;
        refr = refract_ray(f3_of(smp.ray.dir), f3_of(h.n), h.inverse_n != 0, mat.refractive_index,
                           R, td);
    }
}

// block_counts[b] = reflected rays of block b, block_counts[nb + b] =
// refracted ones; the scan over the 2 nb entries gives both slot bases.
__global__ void k_sec_count(SceneView S, const rt_sample* __restrict__ in,
                            const rt_hit* __restrict__ hits, int n,
                            uint32_t* __restrict__ block_counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool refl = false, refr = false;
    rt_material mat;
    if (i < n) sec_flags(S, in[i], hits[i], refl, refr, mat);
    const int cr = __syncthreads_count(refl);
    const int ct = __syncthreads_count(refr);
    if (threadIdx.x == 0) {
        block_counts[blockIdx.x] = (uint32_t)cr;
        block_counts[gridDim.x + blockIdx.x] = (uint32_t)ct;
    }
}

// Exclusive scan by one block, 4096 counts a turn (5,478 counts: 11 -> 5 us
// against a scan in shared memory with two barriers per doubling).
__global__ void __launch_bounds__(1024) k_sec_scan(uint32_t* __restrict__ block_counts, int nblocks,
                                                   int max_out, int32_t* __restrict__ d_count) {
    __shared__ uint32_t tot[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int b0 = 0, turn = 0; b0 < nblocks; b0 += 4096, turn ^= 1) {
        const int i = b0 + 4 * threadIdx.x;
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k < nblocks ? block_counts[i + k] : 0;
        const uint32_t own = v[0] + v[1] + v[2] + v[3];
        auto scan = [&](uint32_t x) {   // inclusive, over the warp
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, x, off);
                if (lane >= off) x += t;
            }
            return x;
        };
        const uint32_t in_warp = scan(own);
        if (lane == 31) tot[turn][w] = in_warp;
        __syncthreads();   // one barrier a turn: the next turn writes the other totals
        const uint32_t warps = scan(tot[turn][lane]);
        const uint32_t before = __shfl_sync(0xffffffffu, warps, (w + 31) & 31);
        uint32_t at = carry + (w ? before : 0) + in_warp - own;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i + k < nblocks) block_counts[i + k] = at;
            at += v[k];
        }
        carry += __shfl_sync(0xffffffffu, warps, 31);
    }
    if (threadIdx.x == 0) *d_count = (int32_t)min(carry, (uint32_t)max_out);
}

__device__ __forceinline__ rt_sample sec_sample(const rt_hit& h, f3 dir, int pixel,
                                                float contribution) {
    rt_sample o;
    o.ray.ori[0] = h.hit_point[0];
    o.ray.ori[1] = h.hit_point[1];
    o.ray.ori[2] = h.hit_point[2];
    o.ray.ori[3] = 0.f;
    o.ray.dir[0] = dir.x;
    o.ray.dir[1] = dir.y;
    o.ray.dir[2] = dir.z;
    o.ray.dir[3] = 0.f;
    o.ray.inv_dir[0] = 1.0f / dir.x;
    o.ray.inv_dir[1] = 1.0f / dir.y;
    o.ray.inv_dir[2] = 1.0f / dir.z;
    o.ray.inv_dir[3] = 0.f;
    o.ray.tmin = 0.0001f;
    o.ray.tmax = 1e37f;
    o.ray._pad[0] = o.ray._pad[1] = 0.f;
    o.pixel = pixel;
    o.contribution = contribution;
    o._pad[0] = o._pad[1] = 0;
    return o;
}

__global__ void k_sec_emit(SceneView S, const rt_sample* __restrict__ in,
                           const rt_hit* __restrict__ hits, int n,
                           const uint32_t* __restrict__ block_offsets, rt_sample* __restrict__ out,
                           int max_out) {
    __shared__ uint32_t warp_tot[2][32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool refl = false, refr = false;
    rt_material mat;
    if (i < n) sec_flags(S, in[i], hits[i], refl, refr, mat);
    const unsigned bal_l = __ballot_sync(0xffffffffu, refl);
    const unsigned bal_t = __ballot_sync(0xffffffffu, refr);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        warp_tot[0][w] = __popc(bal_l);
        warp_tot[1][w] = __popc(bal_t);
    }
    __syncthreads();
    if (!refl && !refr) return;
    uint32_t wl = 0, wt = 0;
    for (int k = 0; k < w; ++k) {
        wl += warp_tot[0][k];
        wt += warp_tot[1][k];
    }
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t slot_l = block_offsets[blockIdx.x] + wl + __popc(bal_l & below);
    const uint32_t slot_t = block_offsets[gridDim.x + blockIdx.x] + wt + __popc(bal_t & below);
    const rt_hit& h = hits[i];
    const rt_sample& smp = in[i];
    float R = 1.0f;
    if (refr && slot_t < (uint32_t)max_out) {
        f3 td;
        refract_ray(f3_of(smp.ray.dir), f3_of(h.n), h.inverse_n != 0, mat.refractive_index, R, td);
        out[slot_t] = sec_sample(h, td, smp.pixel, smp.contribution * mat.reflectiveness * (1.0f - R));
    }
    if (refl && slot_l < (uint32_t)max_out) {
        f3 dir;
        reflect_ray(f3_of(smp.ray.dir), f3_of(h.n), dir);
        out[slot_l] = sec_sample(h, dir, smp.pixel, smp.contribution * mat.reflectiveness * R);
    }
}

__global__ void k_fb_copy(const uint32_t* __restrict__ img, uchar4* __restrict__ rgba, size_t px,
                          float inv1e6) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= px) return;
    rgba[i] = rgba8_of(make_uint3(img[3 * i], img[3 * i + 1], img[3 * i + 2]), inv1e6);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
static unsigned blocks(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// Kernel variants the autotuner chooses from: block size x minimum resident
// blocks per SM (which bounds the registers per thread).
struct RenderVariant {
    int threads, min_blocks;
    void (*fn)(RenderArgs);
    bool pooled;
    bool refract;     // follows the refracted rays of refracting materials
    int max_bounces;  // deepest frame it holds (0: any)
    // a pixel's sum is added up in RenderArgs::accum (several of its rays may
    // be on the way at once)
    bool sums() const { return pooled && refract; }
};
static const RenderVariant kVariants[] = {
    {64, 8, k_render<64, 8>, false},    {64, 12, k_render<64, 12>, false},
    {128, 4, k_render<128, 4>, false},  {128, 6, k_render<128, 6>, false},
    {128, 8, k_render<128, 8>, false},  {256, 2, k_render<256, 2>, false},
    {256, 3, k_render<256, 3>, false},  {256, 4, k_render<256, 4>, false},
    {128, 6, k_render_pool<128, 6>, true}, {128, 8, k_render_pool<128, 8>, true},
    {256, 3, k_render_pool<256, 3>, true}, {256, 4, k_render_pool<256, 4>, true},
    {128, 6, k_render<128, 6, true>, false, true},
    {128, 4, k_render_pool_refr<128, 4, 6>, true, true, 6},
    {128, 5, k_render_pool_refr<128, 5, 4>, true, true, 4},
    {128, 6, k_render_quad<128, 6>, false},
    // by the frame's size k_render_quad or this (against k_render_pool<128, 6>,
    // which holds 7 blocks, 4K of 17.7 M triangles 9.64 -> 9.28 ms, mid-scale
    // frame 2.51 -> 2.46)
    {128, 8, k_render_pool<128, 8>, true},
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);
static_assert(kAutoVariant == kNumVariants - 1 && kQuadVariant == kNumVariants - 2 && kPoolVariant == 9,
              "the variants' numbers");
static_assert(kNumVariants <= kMaxRenderVariants, "per-variant context arrays");

int render_variant_count() { return kNumVariants; }

int render_variant_info(int v, int* threads, int* min_blocks, const void** fn) {
    if (v < 0 || v >= kNumVariants) return -1;
    if (threads) *threads = kVariants[v].threads;
    if (min_blocks) *min_blocks = kVariants[v].min_blocks;
    if (fn) *fn = (const void*)kVariants[v].fn;
    return 0;
}

bool render_variant_pooled(int v) { return v >= 0 && v < kNumVariants && kVariants[v].pooled; }

bool render_variant_sums(int v) { return v >= 0 && v < kNumVariants && kVariants[v].sums(); }

bool render_variant_refracts(int v) { return v >= 0 && v < kNumVariants && kVariants[v].refract; }

bool render_variant_fits(int v, int max_bounces) {
    if (v < 0 || v >= kNumVariants) return false;
    return kVariants[v].max_bounces == 0 || max_bounces <= kVariants[v].max_bounces;
}

int render_refract_variant(int max_bounces) {
    // the pooled variant with the smallest pool that holds the frame, else
    // the ray-tree walk
    int best = -1;
    for (int v = 0; v < kNumVariants; ++v) {
        if (!kVariants[v].refract || !render_variant_fits(v, max_bounces)) continue;
        if (best < 0 || (kVariants[v].pooled && (!kVariants[best].pooled ||
                                                 kVariants[v].max_bounces < kVariants[best].max_bounces)))
            best = v;
    }
    return best;
}

cudaError_t launch_render(const RenderArgs& a, int variant, int grid, cudaStream_t s) {
    if (variant < 0 || variant >= kNumVariants) return cudaErrorInvalidValue;
    const size_t px = (size_t)a.width * a.height;
    if (kVariants[variant].sums()) {
        if (!a.accum) return cudaErrorInvalidValue;
        cudaError_t e = cudaMemsetAsync(a.accum, 0, 3 * sizeof(uint32_t) * px, s);
        if (e != cudaSuccess) return e;
    }
    kVariants[variant].fn<<<grid, kVariants[variant].threads, 0, s>>>(a);
    if (kVariants[variant].sums() && px)
        k_fb_copy<<<blocks(px, 256), 256, 0, s>>>(a.accum, reinterpret_cast<uchar4*>(a.rgba), px,
                                                  a.inv1e6);
    return cudaGetLastError();
}

cudaError_t launch_gen_primary(const rt_camera& cam, int w, int h, int q, const rt_pixel_sample* ps,
                               size_t count, size_t offset, rt_sample* out, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    k_gen_primary<<<blocks(count, 256), 256, 0, s>>>(cam, w, h, q, ps, count, offset, out);
    return cudaGetLastError();
}

// Launches with few rays take four lanes per ray (trace_quad.cuh).  Up to 768
// (kQuadRaysPerSm) rays per SM (primary rays of 10k / 200k triangles, trace and shadow: 65k rays
// 140 -> 117 / 185 -> 153 us, 131k 150 -> 141 / 216 -> 192, 262k 181 -> 187 /
// 262 -> 269); and of these, fewer than eight to a warp as long as that leaves
// no more than 16 warps per SM (2k to 20k rays, whole pipeline 532 -> 520 us).
static int quad_rays_per_warp(int n, int sms) {
    if (n > kQuadRaysPerSm * sms) return 0;
    int per = 8;
    while (per > 1 && n <= 16 * sms * (per / 2)) per /= 2;
    return per;
}

cudaError_t launch_trace(const SceneView& S, const rt_sample* smp, int n, rt_hit* hits,
                         uint32_t* status, int sms, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (const int per = quad_rays_per_warp(n, sms))
        k_trace<true><<<blocks(n, 4 * per), 128, 0, s>>>(S, smp, n, hits, status, per);
    else
        k_trace<false><<<blocks(n, 128), 128, 0, s>>>(S, smp, n, hits, status, 32);
    return cudaGetLastError();
}

cudaError_t launch_shadow(const SceneView& S, const rt_lights& L, int n, rt_hit* hits,
                          uint32_t* status, int sms, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (const int per = quad_rays_per_warp(n, sms))
        k_shadow<true><<<blocks(n, 4 * per), 128, 0, s>>>(S, L, n, hits, status, per);
    else
        k_shadow<false><<<blocks(n, 128), 128, 0, s>>>(S, L, n, hits, status, 32);
    return cudaGetLastError();
}

cudaError_t launch_shade(const SceneView& S, const rt_lights& L, const rt_sample* smp,
                         const rt_hit* hits, int n, uint32_t* image, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_shade<<<blocks(n, 128), 128, 0, s>>>(S, L, smp, hits, n, image);
    return cudaGetLastError();
}

cudaError_t launch_gen_secondary(const SceneView& S, const rt_sample* in, int n, const rt_hit* hits,
                                 rt_sample* out, int max_out, int32_t* d_count,
                                 uint32_t* block_scratch, cudaStream_t s) {
    if (n <= 0) return cudaMemsetAsync(d_count, 0, sizeof(int32_t), s);
    const int nb = (int)blocks(n, 256);
    k_sec_count<<<nb, 256, 0, s>>>(S, in, hits, n, block_scratch);
    k_sec_scan<<<1, 1024, 0, s>>>(block_scratch, 2 * nb, max_out, d_count);
    k_sec_emit<<<nb, 256, 0, s>>>(S, in, hits, n, block_scratch, out, max_out);
    return cudaGetLastError();
}

cudaError_t launch_fb_copy(const uint32_t* img, uint8_t* rgba, size_t px, float inv1e6,
                           cudaStream_t s) {
    if (px == 0) return cudaSuccess;
    k_fb_copy<<<blocks(px, 256), 256, 0, s>>>(img, reinterpret_cast<uchar4*>(rgba), px, inv1e6);
    return cudaGetLastError();
}

size_t gen_secondary_scratch_bytes(int n) { return sizeof(uint32_t) * (2 * blocks(n, 256) + 1); }

}  // namespace rt
