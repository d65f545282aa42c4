// lbvh_dev.cuh — device-side stages of the LBVH build, shared by the
// one-scene kernels (lbvh.cu) and the persistent many-scene kernel
// (batch.cu).  Each function works on one scene whose arrays are passed
// already offset to that scene, so the same code serves both.
//
// Reference: BVHBuilder::build_lbvh (src/rt/bvh-builder.cpp:201-741) and
// src/kernel/bvh-builder.cl (citations per function).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rt_internal.cuh"

namespace rt {

constexpr int SORT_MINB = 3;   // radix tiles resident per SM (register budget)
constexpr int SORT_THREADS = 256;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_ITEMS = 16;   // keys per thread of a radix tile
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;   // 4096 keys per tile
constexpr uint32_t LB_AGG = 1u << 30, LB_PREFIX = 2u << 30, LB_MASK = (1u << 30) - 1;
constexpr uint32_t LB_SPIN_LIMIT = 1u << 22;
// Look-back words read per round trip.  A poll that meets an unpublished
// word reads its whole window again, so a wide window costs more in polls
// than it saves in round trips: 2 to 6 words measured best (32 words: a
// build of 17.7 M triangles 7 % slower; a sleep between polls changed
// nothing).
constexpr int LB_WINDOW = 4;

// float <-> order-preserving uint32 (min/max of the integers == fmin/fmax of
// the floats for non-NaN values).
__device__ __forceinline__ uint32_t f2o(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
    uint32_t u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
    return __uint_as_float(u);
}

// Relaxed GPU-scope accesses: coherent in L2, no ordering of other memory.
// For words that carry their whole message (the radix look-back's flag and
// count).
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Plain loads of what an earlier kernel of a build wrote.  The build's kernels
// start while their predecessor still runs, so its results are not read-only
// for the kernel's lifetime, as the non-coherent loads that __ldg and const
// __restrict__ give require: such a load may be moved above the wait for the
// predecessor.  A volatile asm stays behind it.  What the build's kernels read of
// one another goes through these: bounds (morton_params), digit counts (tile 0 of
// a pass), sorted keys, order, item counts and items, the header's status.  The
// radix tiles' keys and values are read at places that follow from a counter
// taken after the wait; vertices, indices, materials and ids are no kernel's of
// the build.
__device__ __forceinline__ uint32_t ld_dep(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_dep(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// build_primitive_bbox (bvh-builder.cl:100-130) of one triangle.
__device__ __forceinline__ void tri_aabb(const float4* __restrict__ pos,
                                         const uint32_t* __restrict__ idx, uint32_t i,
                                         float lo[3], float hi[3]) {
    const uint32_t a = __ldg(&idx[3 * (size_t)i]), b = __ldg(&idx[3 * (size_t)i + 1]),
                   c = __ldg(&idx[3 * (size_t)i + 2]);
    const float4 p0 = __ldg(&pos[a]), p1 = __ldg(&pos[b]), p2 = __ldg(&pos[c]);
    hi[0] = fmaxf(fmaxf(p0.x, p1.x), p2.x);
    hi[1] = fmaxf(fmaxf(p0.y, p1.y), p2.y);
    hi[2] = fmaxf(fmaxf(p0.z, p1.z), p2.z);
    lo[0] = fminf(fminf(p0.x, p1.x), p2.x);
    lo[1] = fminf(fminf(p0.y, p1.y), p2.y);
    lo[2] = fminf(fminf(p0.z, p1.z), p2.z);
}

// Scene bounds as six words that start at zero: the complements of the lower
// corner's ordered integers and the upper corner's, both maxima.
__device__ __forceinline__ void bounds_add(uint32_t* bounds, int c, float lo, float hi) {
    atomicMax(&bounds[c], ~f2o(lo));
    atomicMax(&bounds[3 + c], f2o(hi));
}

// Per-scene constants of morton_encode (bvh-builder.cl:181-252).
struct MortonParams {
    float glo[3], inv[3];
    float scale;          // pow(2, ceil(depth / 3.0))
    int depth, offset;    // offset = depth % 3 ? 3 - depth % 3 : 0
};

__device__ __forceinline__ MortonParams morton_params(const uint32_t* bounds, int depth) {
    MortonParams m;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        m.glo[c] = o2f(~ld_dep(&bounds[c]));
        const float ghi = o2f(ld_dep(&bounds[3 + c]));
        m.inv[c] = 1.0f / (ghi - m.glo[c]);
    }
    m.scale = (float)(1u << ((depth + 2) / 3));
    m.depth = depth;
    m.offset = depth % 3 ? 3 - (depth % 3) : 0;
    return m;
}

// Spreads the low 21 bits of v to every third bit (bit t to bit 3t): the
// mask-and-shift bit interleave ("magic numbers") of Morton encoders.
__device__ __forceinline__ uint64_t spread3(uint64_t v) {
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// spread3 of 10 bits in 32-bit arithmetic: the codes of up to 30 bits.
__device__ __forceinline__ uint32_t spread3_10(uint32_t v) {
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// morton_encode's bit loop takes, for code bit b (b < depth), bit (b+off)/3
// of the slice of axis (b+off+1) % 3.  With j = b + off, that is the
// interleave I whose bit j is bit j/3 of axis (j+1) % 3 (y, z, x for
// j = 0, 1, 2 mod 3), shifted down by off; the slices keep their low
// ceil(depth/3) bits (a slice of 2^ceil(depth/3), from a centroid at the
// upper bound, contributes nothing).
__device__ __forceinline__ uint32_t morton_code(const MortonParams& P, const float lo[3],
                                                const float hi[3]) {
    uint32_t m[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float center = (hi[k] + lo[k]) * 0.5f;
        float slice = (center - P.glo[k]) * P.inv[k];
        slice = fmaxf(0.0f, fminf(1.0f, slice));
        slice *= P.scale;
        m[k] = (uint32_t)slice;   // truncation
    }
    const int bits = (P.depth + 2) / 3;
    const uint32_t keep = (1u << bits) - 1u;
    if (bits <= 10) {
        // the 64-bit interleave is about half of k_morton_hist's instructions:
        // without it the build of 17.7 M triangles takes 1.997 against 2.017 ms
        // (1.24 M: no change, the kernel waits for its gathers there)
        const uint32_t I = spread3_10(m[1] & keep) | (spread3_10(m[2] & keep) << 1) |
                           (spread3_10(m[0] & keep) << 2);
        return (I >> P.offset) & ((1u << P.depth) - 1u);
    }
    const uint64_t I = spread3(m[1] & keep) | (spread3(m[2] & keep) << 1) |
                       (spread3(m[0] & keep) << 2);
    const uint64_t code = I >> P.offset;
    return P.depth >= 32 ? (uint32_t)code : (uint32_t)code & ((1u << P.depth) - 1u);
}

// Exclusive scan of one value per thread over a 256-thread block; one barrier
// (each warp sums the earlier warps' totals itself).
__device__ __forceinline__ uint32_t block_excl_scan_256(uint32_t v, uint32_t* s_warp) {
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (l >= o) x += y;
    }
    if (l == 31) s_warp[w] = x;
    __syncthreads();
    const uint32_t before = __reduce_add_sync(0xffffffffu, l < w ? s_warp[l] : 0u);
    return before + x - v;
}

template <int ITEMS>
struct __align__(16) SortSmemT {
    uint32_t keys[SORT_THREADS * ITEMS];
    uint32_t vals[SORT_THREADS * ITEMS];
    uint32_t whist[SORT_WARPS][256];
    uint32_t goff[256];
    uint32_t scan[2][SORT_WARPS];
    uint32_t tile;
};
using SortSmem = SortSmemT<SORT_ITEMS>;

// One tile of a stable LSD radix pass (8-bit digit at `shift`, one digit per
// thread): warp-striped keys, ballot ranking in index order, the tile in digit
// order in shared memory, decoupled look-back over the earlier tiles of the
// same sequence, and a coalesced scatter.  Must be called by all SORT_THREADS
// threads of a block; a tile holds SORT_THREADS * ITEMS keys (WHOLE: all of
// them; the last tile of a sequence may hold fewer).  A null `vin` stands for
// the values 0, 1, 2, ... (the first pass of a build).  `hist` holds the pass's
// 256 digit counts, `lookback` 256 words per tile: tile 0 publishes the global
// offset of each digit with its count, so the later tiles' prefixes are
// scatter offsets as they are.  A look-back that polls an unpublished word
// more than SPIN_LIMIT times gives up: it sets RT_DEV_TIMEOUT in *status and, if
// there is one, in *failed (the scene's BvhHeader::status), and goes on with the
// counts it has, so every block ends; its writes stay inside
// [0, n): a partial prefix only lowers the offsets, a key's place in its tile is
// added, and what would lie at or beyond n is dropped.  What the pass leaves is
// arbitrary then: some places keep what the memory held before, so neither its
// keys nor its values may be used as a sorted order (see emit_level).
//
// What bounds it: the chain of one tile, about 14 us of load and ranking
// (6.0-6.6), staging (1.3-1.7), look-back (3.4-4.0: 8 to 11 round trips) and
// scatter (1.3), which the look-back ties to the tiles before it.  Without bound
// checks in whole tiles, a scan of the digit counts in every tile and two of
// three barriers per scan, and with the first look-back words requested before
// the staging: build of 1.24 M triangles 213 -> 210 us, 10k-triangle frame 381 ->
// 376; at 17.7 M pairs (9.5 waves of tiles) no change.
template <int ITEMS, uint32_t SPIN_LIMIT, bool WHOLE>
__device__ __forceinline__ void onesweep_tile_body(SortSmemT<ITEMS>& S, uint32_t tile,
                                                   const uint32_t* __restrict__ kin,
                                                   const uint32_t* __restrict__ vin,
                                                   uint32_t* __restrict__ kout,
                                                   uint32_t* __restrict__ vout, uint32_t n,
                                                   int shift, const uint32_t* __restrict__ hist,
                                                   uint32_t* __restrict__ lookback,
                                                   uint32_t* __restrict__ status,
                                                   uint32_t* __restrict__ failed) {
    constexpr uint32_t TILE = SORT_THREADS * ITEMS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = tile * TILE;                 // n < 2^30
    const uint32_t valid = WHOLE ? TILE : n - base;    // keys of this tile
    const uint32_t mine = (uint32_t)warp * (ITEMS * 32) + lane;   // this thread's first key
    const uint32_t lanemask_lt = (1u << lane) - 1u;
    uint32_t k[ITEMS], v[ITEMS], rank[ITEMS];
    static_assert(ITEMS % 4 == 0, "whole 128-bit words per thread");
    // a whole, 16-byte aligned tile: 128-bit loads into shared memory, then
    // the warp-striped layout the ranking needs from there
    const bool vec =
        WHOLE && ((reinterpret_cast<uintptr_t>(kin) | reinterpret_cast<uintptr_t>(vin)) & 15u) == 0;
    if (vec) {
        const uint4* k4 = reinterpret_cast<const uint4*>(kin + base);
        const uint4* v4 = reinterpret_cast<const uint4*>(vin + base);
#pragma unroll
        for (int j = 0; j < ITEMS / 4; ++j) {
            const int e = j * SORT_THREADS + tid;
            reinterpret_cast<uint4*>(S.keys)[e] = __ldcs(&k4[e]);
            if (vin) reinterpret_cast<uint4*>(S.vals)[e] = __ldcs(&v4[e]);
        }
    }
    for (int i = tid; i < SORT_WARPS * 64; i += SORT_THREADS)
        reinterpret_cast<uint4*>(&S.whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    if (vec) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) k[j] = S.keys[mine + j * 32];
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            k[j] = WHOLE || mine + j * 32 < valid ? __ldcs(&kin[base + mine + j * 32]) : 0xffffffffu;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const bool ok = WHOLE || mine + j * 32 < valid;
        const uint32_t d = (k[j] >> shift) & 255u;
        // lanes holding the same digit: one ballot per digit bit (a fixed
        // cost, where a match instruction grows with the distinct digits)
        uint32_t peers = WHOLE ? 0xffffffffu : __ballot_sync(0xffffffffu, ok);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const uint32_t bit = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= ((d >> b) & 1u) ? bit : ~bit;
        }
        uint32_t prev = 0;
        if (ok) prev = S.whist[warp][d];
        __syncwarp();
        if (ok) {
            const uint32_t below = __popc(peers & lanemask_lt);
            rank[j] = prev + below;
            if (below == 0u) S.whist[warp][d] = prev + __popc(peers);
        }
        __syncwarp();
    }
    // the values, which the ranking does not need (its registers)
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t e = mine + j * 32;
        v[j] = !vin ? base + e : vec ? S.vals[e] : WHOLE || e < valid ? __ldcs(&vin[base + e]) : 0u;
    }
    __syncthreads();

    // thread tid's digit: counts of the warps, summed in warp order
    uint32_t cnt = 0;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) cnt += S.whist[w][tid];
    uint32_t excl = 0;
    uint32_t* my = &lookback[(size_t)tile * 256 + tid];
    if (tile == 0) {
        excl = block_excl_scan_256(ld_dep(&hist[tid]), S.scan[1]);
        st_relaxed(my, LB_PREFIX | (excl + cnt));
    } else {
        st_relaxed(my, LB_AGG | cnt);   // as early as the count is known
    }
    const uint32_t lstart = block_excl_scan_256(cnt, S.scan[0]);
    uint32_t c = lstart;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) {   // first place in the tile of each warp's keys
        const uint32_t x = S.whist[w][tid];
        S.whist[w][tid] = c;
        c += x;
    }
    __syncthreads();
    // the first look-back words are on their way while the tile is staged
    uint32_t win[LB_WINDOW];
    auto read_window = [&](int32_t p) {
#pragma unroll
        for (int t = 0; t < LB_WINDOW; ++t)   // tile 0 is always a prefix: p - t < 0 is never summed
            win[t] = p - t >= 0 ? ld_relaxed(&lookback[(size_t)(p - t) * 256 + tid]) : LB_PREFIX;
    };
    int32_t p = (int32_t)tile - 1;
    if (tile > 0) read_window(p);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (WHOLE || mine + j * 32 < valid) {
            const uint32_t at = S.whist[warp][(k[j] >> shift) & 255u] + rank[j];
            S.keys[at] = k[j];
            S.vals[at] = v[j];
        }
    }
    // Decoupled look-back.  Each word holds its whole message (flag and
    // count), so relaxed accesses suffice; the words of LB_WINDOW earlier
    // tiles are read per round trip and summed nearest first, up to the first
    // inclusive prefix or the first tile that has not published.
    if (tile > 0) {
        uint32_t spins = 0;
        bool open = true;   // no inclusive prefix yet
        for (;;) {
            int used = 0;
            bool wait = false;
#pragma unroll
            for (int t = 0; t < LB_WINDOW; ++t) {
                if (open && !wait) {
                    if ((win[t] & ~LB_MASK) == 0u) {
                        wait = true;
                    } else {
                        excl += win[t] & LB_MASK;
                        open = (win[t] & ~LB_MASK) != LB_PREFIX;
                        ++used;
                    }
                }
            }
            if (!open) break;
            p -= used;
            if (wait && ++spins > SPIN_LIMIT) {
                atomicOr(status, RT_DEV_TIMEOUT);
                if (failed) atomicOr(failed, RT_DEV_TIMEOUT);
                break;
            }
            read_window(p);
        }
        st_relaxed(my, LB_PREFIX | (excl + cnt));
    }
    S.goff[tid] = excl - lstart;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = tid; i < valid; i += SORT_THREADS) {
        const uint32_t key = S.keys[i];
        const uint32_t dst = S.goff[(key >> shift) & 255u] + i;
        if (dst < n) {   // always, unless a wait gave up (RT_DEV_TIMEOUT)
            kout[dst] = key;
            vout[dst] = S.vals[i];
        }
    }
}

// A caller that takes several tiles with one S has a barrier between them.
template <int ITEMS = SORT_ITEMS, uint32_t SPIN_LIMIT = LB_SPIN_LIMIT>
__device__ __forceinline__ void onesweep_tile(SortSmemT<ITEMS>& S, uint32_t tile,
                                              const uint32_t* __restrict__ kin,
                                              const uint32_t* __restrict__ vin,
                                              uint32_t* __restrict__ kout,
                                              uint32_t* __restrict__ vout, uint32_t n, int shift,
                                              const uint32_t* __restrict__ hist,
                                              uint32_t* __restrict__ lookback,
                                              uint32_t* __restrict__ status,
                                              uint32_t* __restrict__ failed) {
    if ((size_t)(tile + 1) * (SORT_THREADS * ITEMS) <= n)
        onesweep_tile_body<ITEMS, SPIN_LIMIT, true>(S, tile, kin, vin, kout, vout, n, shift, hist,
                                                    lookback, status, failed);
    else
        onesweep_tile_body<ITEMS, SPIN_LIMIT, false>(S, tile, kin, vin, kout, vout, n, shift, hist,
                                                     lookback, status, failed);
}

// rearrange_indices / rearrange_map (bvh-builder.cl:49-72) of sorted slot i,
// plus the traversal's triangle record; returns the triangle's AABB
// (build_leaf_bbox's min / max of the three vertices).
struct PermuteIO {
    const uint32_t* vals;       // sorted slot -> triangle in the order before the build
    const uint32_t* idx_old;
    const uint32_t* map_old;
    const uint32_t* orig_old;
    const float4* pos;
    uint32_t* idx_new;
    uint32_t* map_new;
    uint32_t* orig_new;
    float4* tris;
};

// Triangle record (its `more` mark clear) and AABB of sorted triangle i with
// vertices a, b, c.
__device__ __forceinline__ void tri_record(uint32_t i, const PermuteIO& P, uint32_t a, uint32_t b,
                                           uint32_t c, float4& lo, float4& hi) {
    const float4 p0 = __ldg(&P.pos[a]), p1 = __ldg(&P.pos[b]), p2 = __ldg(&P.pos[c]);
    P.tris[3 * (size_t)i] = make_float4(p0.x, p0.y, p0.z, 0.f);
    P.tris[3 * (size_t)i + 1] = make_float4(p1.x - p0.x, p1.y - p0.y, p1.z - p0.z, 0.f);
    P.tris[3 * (size_t)i + 2] = make_float4(p2.x - p0.x, p2.y - p0.y, p2.z - p0.z, 0.f);
    hi.x = fmaxf(fmaxf(p0.x, p1.x), p2.x);
    hi.y = fmaxf(fmaxf(p0.y, p1.y), p2.y);
    hi.z = fmaxf(fmaxf(p0.z, p1.z), p2.z);
    lo.x = fminf(fminf(p0.x, p1.x), p2.x);
    lo.y = fminf(fminf(p0.y, p1.y), p2.y);
    lo.z = fminf(fminf(p0.z, p1.z), p2.z);
    lo.w = hi.w = 0.f;
}

// `sorted` false: there is no order to take (a wait of the sort gave up), the
// triangles stay where they are.
__device__ __forceinline__ void permute_tri(uint32_t i, const PermuteIO& P, bool sorted, float4& lo,
                                            float4& hi) {
    const uint32_t o = sorted ? ld_dep(&P.vals[i]) : i;
    const uint32_t a = __ldg(&P.idx_old[3 * (size_t)o]), b = __ldg(&P.idx_old[3 * (size_t)o + 1]),
                   c = __ldg(&P.idx_old[3 * (size_t)o + 2]);
    P.idx_new[3 * (size_t)i] = a;
    P.idx_new[3 * (size_t)i + 1] = b;
    P.idx_new[3 * (size_t)i + 2] = c;
    P.map_new[i] = __ldg(&P.map_old[o]);
    P.orig_new[i] = __ldg(&P.orig_old[o]);
    tri_record(i, P, a, b, c, lo, hi);
}

// Refit's counterpart of permute_tri: the triangle keeps its place, its
// record and AABB are made from the current vertex positions
// (refit_lbvh, bvh-builder.cpp:743-790).
__device__ __forceinline__ void refit_tri(uint32_t i, const PermuteIO& P, float4& lo, float4& hi) {
    const uint32_t* idx = P.idx_new;
    tri_record(i, P, __ldg(&idx[3 * (size_t)i]), __ldg(&idx[3 * (size_t)i + 1]),
               __ldg(&idx[3 * (size_t)i + 2]), lo, hi);
}

// delta(i): highest differing bit between sorted keys i and i+1, with the
// index appended so that equal keys still order (Karras' augmentation).
__device__ __forceinline__ uint64_t delta(const uint32_t* __restrict__ k, uint32_t i) {
    const uint32_t x = ld_dep(&k[i]) ^ ld_dep(&k[i + 1]);
    return ((uint64_t)x << 32) | (uint64_t)(i ^ (i + 1));
}


// ---------------------------------------------------------------------------
// Multi-level emit + refit, warp-synchronous.  The tree is built bottom-up
// in a few launches ("levels").  Within a block, runs of consecutive items
// are joined by warps: a warp holds up to 32 consecutive items, one per lane
// (at level 0 the items are the sorted triangles).  warp_join writes in one
// step every node whose range lies inside the warp's items: the levels of
// the boundaries between items, as seven ballots, give each node's range and
// parent, and sparse tables in shared memory give its children's boxes.  A
// run whose parent lies outside the warp's items is left over; the block
// gathers the leftovers of its warps in order and joins them again, at most
// 32 per warp, until one warp holds them all or no node inside the block is
// left.  What is left then has its parent outside the block and becomes an
// item of the next level, which gathers the items of EMIT_GROUP blocks,
// until one block reaches the root.  A block leaves at most EMIT_FMAX items:
// they hang off the chains of nodes crossing its two ends, each at most 64
// deep (32 key bits + 32 index bits).
//
// The tree is the binary radix tree of the sorted keys (Karras), collapsed
// to the reference's leaf rule: a node [L, R] is an interior node of the
// reference's tree iff R - L + 1 >= min_leaf + 3 (find_middle's unsigned test
// last - first - 1 <= min_leaf, bvh-builder.cl:501) and its keys are not all
// equal (the bit loop of :515-525); otherwise it is a leaf, or part of one.
// The reference's split (highest differing bit, first index with the bit
// set) is the radix tree's split, so both trees have the same ranges.  With
// d[j] the augmented delta of the boundary before item j of a chunk and d[c]
// the boundary after its last item (D(-1) = D(n-1) = max), a run j..b is a
// left child iff d[b+1] < d[j];
// its parent stays in the chunk iff max d[b+2..c] > d[b+1] (the parent's
// range ends at the first boundary above d[b+1]); a right child's parent
// stays iff max d[0..j-1] > d[j].  Above the leftovers of a chunk, the
// boundaries between consecutive items are exactly the splits of the
// remaining nodes (a node's inner boundaries all lie below its end
// boundaries), so chunks and levels compose.
// ---------------------------------------------------------------------------
constexpr int EMIT_FMAX = 128;   // items a block may leave
constexpr int EMIT_GROUP = 8;   // blocks of one level gathered by a block of the next
constexpr uint32_t EMIT_LEAVE0 = 128u;   // runs a level-0 block may leave unjoined
constexpr uint32_t EMIT_LEAVE1 = 64u;    // the same above level 0
constexpr int EMIT_C0 = 512;             // triangles per level-0 block
constexpr int EMIT_MINB0 = 3;            // level-0 blocks resident per SM (40 registers)
constexpr int EMIT_C1 = EMIT_GROUP * EMIT_FMAX;    // items per block above level 0
// Threads per block above level 0 (its warps take the items' chunks in
// rounds): 256 in a level of more blocks than SMs, where two blocks per SM
// hide each other's barriers, 512 in the last, narrow levels, which last as
// long as one block does.  Against one thread per item (1024, one block per
// SM) and three barriers per gather: level 1 of 17.7 M triangles 341 -> 239
// us, of 1.24 M 30.7 -> 24.2 us, the last level 11.5 -> 9.4 us.
constexpr int EMIT_T_WIDE = 256, EMIT_T_NARROW = 512;

// Blocks of level 0 of an n-triangle scene, and of the level above nb blocks.
__host__ __device__ __forceinline__ uint32_t emit_blocks0(uint32_t n) {
    return (n + EMIT_C0 - 1) / EMIT_C0;
}
__host__ __device__ __forceinline__ uint32_t emit_next_level(uint32_t nb) {
    return (nb + EMIT_GROUP - 1) / EMIT_GROUP;
}
// Runs a block of a level with `blocks` blocks may leave unjoined (a level of
// one block is the root's and joins everything).
__host__ __device__ __forceinline__ uint32_t emit_leave(int level, uint32_t blocks) {
    return blocks > 1 ? (level == 0 ? EMIT_LEAVE0 : EMIT_LEAVE1) : 32u;
}

// An item: leaf range, keys at its ends, box, ref / count, and the augmented
// delta of the boundary before it.
struct __align__(16) EmitItem {
    uint32_t l, r, kl, kr;
    float lo[3], hi[3];
    int32_t ref, cnt;
    uint64_t db;
    uint32_t pad[2];
};

// A scene's emit items in its emit scratch `base`: level 0 writes buffer A,
// level 1 B, level 2 A, ...; A holds up to EMIT_FMAX items per level-0 block,
// B per level-1 block, then the item counts of A and of B.
struct EmitBuffers {
    EmitItem* items[2];
    uint32_t* counts[2];
};
__host__ __device__ __forceinline__ EmitBuffers emit_buffers(uint32_t n, uint8_t* base) {
    const uint32_t nb0 = emit_blocks0(n), nb1 = emit_next_level(nb0);
    EmitBuffers b;
    b.items[0] = reinterpret_cast<EmitItem*>(base);
    b.items[1] = b.items[0] + (size_t)nb0 * EMIT_FMAX;
    b.counts[0] = reinterpret_cast<uint32_t*>(b.items[1] + (size_t)nb1 * EMIT_FMAX);
    b.counts[1] = b.counts[0] + nb0;
    return b;
}
__host__ __device__ __forceinline__ size_t emit_buffers_bytes(uint32_t n) {
    const size_t blocks = (size_t)emit_blocks0(n) + emit_next_level(emit_blocks0(n));
    return blocks * EMIT_FMAX * sizeof(EmitItem) + ((blocks * sizeof(uint32_t) + 255) & ~(size_t)255);
}

struct WarpItem {
    uint32_t l, r, kl, kr;
    float lox, loy, loz, hix, hiy, hiz;
    int32_t ref, cnt;
    uint64_t db;
};

__device__ __forceinline__ uint64_t delta_or_max(const uint32_t* __restrict__ k, int64_t i,
                                                 uint32_t n) {
    return (i < 0 || i >= (int64_t)n - 1) ? ~0ull : delta(k, (uint32_t)i);
}

// The items of an emit block in shared memory, by quarters (those of
// consecutive items lie side by side: a warp's accesses meet every bank once,
// where whole 64 B items met four banks eight times): build of 1.24 M triangles
// 210 -> 205 us, of 17.7 M 1821 -> 1777 us.
template <int C>
struct ItemList {
    uint4 range[C];          // l, r, kl, kr
    float4 box0[C], box1[C]; // lo, hi.x | hi.y, hi.z, ref, cnt
    uint64_t db[C];
    __device__ __forceinline__ void load(uint32_t e, WarpItem& w) const {
        const uint4 q = range[e];
        const float4 b0 = box0[e], b1 = box1[e];
        w.l = q.x; w.r = q.y; w.kl = q.z; w.kr = q.w;
        w.lox = b0.x; w.loy = b0.y; w.loz = b0.z; w.hix = b0.w;
        w.hiy = b1.x; w.hiz = b1.y;
        w.ref = __float_as_int(b1.z); w.cnt = __float_as_int(b1.w);
        w.db = db[e];
    }
    __device__ __forceinline__ void store(uint32_t e, const WarpItem& w) {
        range[e] = make_uint4(w.l, w.r, w.kl, w.kr);
        box0[e] = make_float4(w.lox, w.loy, w.loz, w.hix);
        box1[e] = make_float4(w.hiy, w.hiz, __int_as_float(w.ref), __int_as_float(w.cnt));
        db[e] = w.db;
    }
};

// An item to and from global memory.
__device__ __forceinline__ void write_item(EmitItem* p, const WarpItem& w) {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(w.l, w.r, w.kl, w.kr);
    q[1] = make_uint4(__float_as_uint(w.lox), __float_as_uint(w.loy), __float_as_uint(w.loz),
                      __float_as_uint(w.hix));
    q[2] = make_uint4(__float_as_uint(w.hiy), __float_as_uint(w.hiz), (uint32_t)w.ref, (uint32_t)w.cnt);
    q[3] = make_uint4((uint32_t)w.db, (uint32_t)(w.db >> 32), 0u, 0u);
}
__device__ __forceinline__ void read_item(const EmitItem* p, WarpItem& w) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    const uint4 a = ld_dep(q), b = ld_dep(q + 1), c = ld_dep(q + 2), d = ld_dep(q + 3);
    w.l = a.x; w.r = a.y; w.kl = a.z; w.kr = a.w;
    w.lox = __uint_as_float(b.x); w.loy = __uint_as_float(b.y); w.loz = __uint_as_float(b.z);
    w.hix = __uint_as_float(b.w); w.hiy = __uint_as_float(c.x); w.hiz = __uint_as_float(c.y);
    w.ref = (int32_t)c.z; w.cnt = (int32_t)c.w;
    w.db = (uint64_t)d.x | ((uint64_t)d.y << 32);
}

// Shared scratch of one warp for warp_join, 2048 bytes.  st is a sparse table of one axis of
// the items' boxes (level t at start i: min / max over items i .. i+2^t-1);
// the arrays hold the items' ranges, end keys and references.  At the end
// `stage`, in the same space, hands the runs left over to the lanes they start at.
struct __align__(16) WarpScratch {
    union {
        struct {
            float2 st[5][32];
            uint32_t il[32], ir[32], ikl[32], ikr[32];
            int32_t iref[32], icnt[32];
        };
        float4 stage[3][32];
    };
};

// Level of a boundary delta: its highest set bit (the radix tree's level),
// 64 for the virtual boundaries before the first and after the last
// triangle.  Two boundaries of one level always have a higher one between
// them, so the nearest boundary above another one is the same by level as
// by delta, and levels order every pair of boundaries the tree compares.
__device__ __forceinline__ uint32_t delta_level(uint64_t x) {
    return x == ~0ull ? 64u : 63u - (uint32_t)__clzll(x);
}

// Lanes of `valid` whose level (bit planes P, most significant last) is
// above L.
__device__ __forceinline__ uint32_t levels_above(uint32_t L, const uint32_t P[7], uint32_t valid) {
    uint32_t gt = 0u, eq = valid;
#pragma unroll
    for (int t = 6; t >= 0; --t) {
        if ((L >> t) & 1u) {
            eq &= P[t];
        } else {
            gt |= eq & P[t];
            eq &= ~P[t];
        }
    }
    return gt;
}

__device__ __forceinline__ uint32_t level_at(uint32_t k, const uint32_t P[7]) {
    uint32_t L = 0u;
#pragma unroll
    for (int t = 0; t < 7; ++t) L |= ((P[t] >> k) & 1u) << t;
    return L;
}

// The lane of the highest boundary in the non-empty mask m (unique: two of
// one level have a higher one between them).
__device__ __forceinline__ uint32_t top_level(uint32_t m, const uint32_t P[7]) {
#pragma unroll
    for (int t = 6; t >= 0; --t) {
        const uint32_t c = m & P[t];
        if (c) m = c;
    }
    return (uint32_t)__ffs(m) - 1u;
}

// min / max of one axis over items a..b (a <= b, b - a < 31) from the table.
__device__ __forceinline__ float2 axis_range(const WarpScratch& W, uint32_t a, uint32_t b) {
    const uint32_t t = 31u - (uint32_t)__clz(b - a + 1u);
    const float2 u = W.st[t][a], v = W.st[t][b + 1u - (1u << t)];
    return make_float2(fminf(u.x, v.x), fmaxf(u.y, v.y));
}

// Joins the items of lanes 0..cnt-1 of the warp (all 32 lanes call it):
// every node whose range lies inside these items is written out, and the
// runs left over (maximal subtrees whose parent lies outside) stay, each in
// the lane of its first item (true for those lanes, `it` holding the run); a
// run that reaches [0, n-1] writes the header instead.  `edge` is the
// boundary after the last item.  With d[j] the boundary before item j, the
// node split at boundary j spans from the nearest higher boundary on its
// left to the one on its right, and its parent is split at the lower of
// those two.  All of it comes from bit planes of the boundary levels, with
// no rounds; the children's boxes come from sparse tables of the item boxes.
// fminf / fmaxf order -0 below +0 and skip NaN whatever the operand order,
// so any grouping of a range gives the bits of the bottom-up merge.  TRIS: the
// items are consecutive triangles, lane l's it.l = it.l of lane 0 + l.
template <bool TRIS>
__device__ __forceinline__ bool warp_join(WarpItem& it, uint32_t cnt, uint64_t edge, uint32_t n,
                                          int min_leaf, float4* __restrict__ nodes,
                                          float4* tris, WarpScratch& W,
                                          BvhHeader* __restrict__ hdr) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned FULL = 0xffffffffu;
    if (cnt == 0u) return false;
    const bool item = lane < cnt;
    __syncwarp();   // the lanes have read their items out of this space
    if (item) {
        W.ikl[lane] = it.kl;
        if (!TRIS) {
            W.il[lane] = it.l;
            W.ir[lane] = it.r;
            W.ikr[lane] = it.kr;
            W.iref[lane] = it.ref;
            W.icnt[lane] = it.cnt;
        }
    }
    const uint32_t first = TRIS ? it.l - lane : 0u;   // TRIS: item a is triangle first + a
    auto left_end = [&](uint32_t a) { return TRIS ? first + a : W.il[a]; };
    auto right_end = [&](uint32_t a) { return TRIS ? first + a : W.ir[a]; };
    auto right_key = [&](uint32_t a) { return TRIS ? W.ikl[a] : W.ikr[a]; };
    // --- topology, from the levels of the boundaries
    // the node split at boundary j = lane (1 <= j < cnt), when it lies
    // inside: left child items A..j-1 (split at lsplit's right end), right
    // child j..B (split at rsplit's)
    bool local = false, out = false, up_left = false;   // up_left: a left child
    uint32_t A = lane, B = lane, lsplit = 0u, rsplit = 0u;
    {
        const uint32_t lev = item ? delta_level(it.db) : 0u;
        uint32_t P[7];
#pragma unroll
        for (int t = 0; t < 7; ++t) P[t] = __ballot_sync(FULL, item && ((lev >> t) & 1u));
        const uint32_t valid = cnt >= 32u ? FULL : ((1u << cnt) - 1u);
        const uint32_t edge_lev = delta_level(edge);
        if (item && lane >= 1u) {
            const uint32_t gt = levels_above(lev, P, valid);
            const uint32_t lm = gt & ((1u << lane) - 1u);
            const uint32_t rm = gt & ~((2u << lane) - 1u);
            if (lm != 0u && (rm != 0u || edge_lev > lev)) {
                local = true;
                A = 31u - (uint32_t)__clz(lm);
                B = rm ? (uint32_t)__ffs(rm) - 2u : cnt - 1u;
                const uint32_t lin = ((1u << lane) - 1u) & ~((2u << A) - 1u);   // A+1..j-1
                const uint32_t rin = ((2u << B) - 1u) & ~((2u << lane) - 1u);   // j+1..B
                lsplit = lin ? top_level(lin, P) - 1u : 0u;
                rsplit = rin ? top_level(rin, P) - 1u : 0u;
            }
        }
        const uint32_t LM = __ballot_sync(FULL, local);
        // the part of this lane whose parent may lie outside (items A..B:
        // its node if local, else its item) and whether it does
        if (item) {
            const uint32_t la = level_at(A, P);
            const uint32_t lb = B + 1u < cnt ? level_at(B + 1u, P) : edge_lev;
            up_left = lb < la;
            const uint32_t p = up_left ? B + 1u : A;   // the parent's split
            out = p == 0u || p >= cnt || !((LM >> p) & 1u);
        }
    }
    // --- boxes: the children's for a local node, the item's otherwise
    float llo[3], lhi[3], rlo[3], rhi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float vlo = k == 0 ? it.lox : (k == 1 ? it.loy : it.loz);
        const float vhi = k == 0 ? it.hix : (k == 1 ? it.hiy : it.hiz);
        __syncwarp();   // the previous axis' queries are done
        float2 u = make_float2(vlo, vhi);   // this lane's entry of the level below
        if (item) W.st[0][lane] = u;
#pragma unroll
        for (int t = 1; t < 5; ++t) {
            __syncwarp();
            const uint32_t h = 1u << (t - 1);
            if (lane + 2u * h <= cnt) {
                const float2 v = W.st[t - 1][lane + h];
                u = make_float2(fminf(u.x, v.x), fmaxf(u.y, v.y));
                W.st[t][lane] = u;
            }
        }
        __syncwarp();
        llo[k] = vlo;
        lhi[k] = vhi;
        rlo[k] = vlo;
        rhi[k] = vhi;
        if (local) {
            const float2 l = axis_range(W, A, lane - 1u), r = axis_range(W, lane, B);
            llo[k] = l.x; lhi[k] = l.y;
            rlo[k] = r.x; rhi[k] = r.y;
        }
    }
    // reference and leaf count of items a..b as one node (split at the
    // right end of item `split`) or as the item itself
    auto ref_of = [&](uint32_t a, uint32_t b, uint32_t split, int32_t& ref, int32_t& c) {
        if (a == b) {
            ref = TRIS ? (int32_t)(first + a) : W.iref[a];
            c = TRIS ? 1 : W.icnt[a];
            return;
        }
        const uint32_t L = left_end(a), count = right_end(b) - L + 1u;
        const bool interior = count >= (uint32_t)min_leaf + 3u && W.ikl[a] != right_key(b);
        ref = interior ? (int32_t)right_end(split) : (int32_t)L;
        c = interior ? 0 : (int32_t)count;
    };
    if (local) {
        const uint32_t gl = left_end(A), gr = right_end(B), self = right_end(lane - 1u);
        if (gr - gl + 1u >= (uint32_t)min_leaf + 3u && W.ikl[A] != right_key(B)) {
            // an interior node: its children fill its half of its parent's
            // record, which lies beside its range; a child that is a leaf
            // fills a half of the node's own record (an interior child fills
            // that half itself)
            const bool root = gl == 0u && gr == n - 1u;
            const uint32_t up = up_left ? gr : gl - 1u, up_slot = up_left ? 0u : 2u;
            auto put = [&](uint32_t side, uint32_t a, uint32_t b, uint32_t split, const float* lo,
                           const float* hi) {
                int32_t ref, c;
                ref_of(a, b, split, ref, c);
                const float4 s0 = make_float4(lo[0], lo[1], hi[0], hi[1]);
                const float4 s1 = make_float4(lo[2], hi[2], __int_as_float(c > 0 ? ~ref : ref),
                                              __int_as_float(c > 0 ? c : (int32_t)self));
                if (!root) {
                    float4* q = nodes + 8 * (size_t)up + 2 * (up_slot + side);
                    q[0] = s0;
                    q[1] = s1;
                }
                if (c > 0) {
                    float4* q = nodes + 8 * (size_t)self + 4 * side;
                    const float inf = __int_as_float(0x7f800000);
                    q[0] = s0;
                    q[1] = s1;
                    q[2] = make_float4(inf, inf, inf, inf);
                    q[3] = make_float4(inf, inf, s1.z, __int_as_float(EMPTY_SLOT));
                }
            };
            put(0u, A, lane - 1u, lsplit, llo, lhi);
            put(1u, lane, B, rsplit, rlo, rhi);
        } else {
            tris[3 * (size_t)self].w = 1.0f;   // a boundary inside a leaf
        }
    }
    float4 q0, q1, q2;
    if (out) {
        int32_t eref, ecnt;
        ref_of(A, B, lane - 1u, eref, ecnt);
        const float lx = local ? fminf(llo[0], rlo[0]) : llo[0],
                    ly = local ? fminf(llo[1], rlo[1]) : llo[1],
                    lz = local ? fminf(llo[2], rlo[2]) : llo[2];
        const float hx = local ? fmaxf(lhi[0], rhi[0]) : lhi[0],
                    hy = local ? fmaxf(lhi[1], rhi[1]) : lhi[1],
                    hz = local ? fmaxf(lhi[2], rhi[2]) : lhi[2];
        const uint32_t gl = left_end(A), gr = right_end(B);
        if (gl == 0u && gr == n - 1u) {   // the root
            hdr->root_ref = eref;
            hdr->root_cnt = ecnt;
            hdr->n_tris = n;
            hdr->root_lo = make_float4(lx, ly, lz, 0.f);
            hdr->root_hi = make_float4(hx, hy, hz, 0.f);
            out = false;
        }
        q0 = make_float4(__uint_as_float(gl), __uint_as_float(gr), __uint_as_float(W.ikl[A]),
                         __uint_as_float(right_key(B)));
        q1 = make_float4(lx, ly, lz, hx);
        q2 = make_float4(hy, hz, __int_as_float(eref), __int_as_float(ecnt));
    }
    // hand each run left over to the lane of its first item
    const uint32_t keep = __reduce_or_sync(FULL, out ? (1u << A) : 0u);
    __syncwarp();   // every read of the scratch is done
    if (out) {
        W.stage[0][A] = q0;
        W.stage[1][A] = q1;
        W.stage[2][A] = q2;
    }
    __syncwarp();
    const bool mine = (keep >> lane) & 1u;
    if (mine) {
        q0 = W.stage[0][lane];
        q1 = W.stage[1][lane];
        q2 = W.stage[2][lane];
        it.l = __float_as_uint(q0.x);
        it.r = __float_as_uint(q0.y);
        it.kl = __float_as_uint(q0.z);
        it.kr = __float_as_uint(q0.w);
        it.lox = q1.x; it.loy = q1.y; it.loz = q1.z; it.hix = q1.w;
        it.hiy = q2.x; it.hiz = q2.y;
        it.ref = __float_as_int(q2.z);
        it.cnt = __float_as_int(q2.w);   // it.db stays: the run starts at this lane
    }
    __syncwarp();   // the staged runs are read before the space is reused
    return mine;
}

// Shared state of an emit block of T threads over up to C items: the items,
// in order, and the warps' scratch.  With a thread per item the scratch takes
// the place of the list, whose items are all in registers by then.
template <int C, int T>
struct EmitSmem {
    ItemList<C> list;
    WarpScratch scratch[T / 32];
    uint32_t wcount[T / 32];
    uint32_t goff[EMIT_GROUP + 1];
    uint64_t edge;   // boundary after the block's last item
};
template <int C>
struct EmitSmem<C, C> {
    union {
        ItemList<C> list;
        WarpScratch scratch[C / 32];
    };
    uint32_t wcount[C / 32];
    uint64_t edge;
};

// Appends, in order, the runs still held by the warps' lanes to the `base`
// runs of S.list and returns their number.  Call with all T threads; `keep`
// marks held runs.
template <int C, int T>
__device__ __forceinline__ uint32_t gather_runs(EmitSmem<C, T>& S, const WarpItem& it, bool keep,
                                                uint32_t base = 0u) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) S.wcount[w] = __popc(bal);
    __syncthreads();   // also: every warp has read its chunk of S.list
    // each warp sums the counts itself: no second barrier behind a scan
    const uint32_t v = lane < (uint32_t)(T / 32) ? S.wcount[lane] : 0u;
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? v : 0u);
    const uint32_t m = __reduce_add_sync(0xffffffffu, v);
    if (keep) S.list.store(base + before + __popc(bal & ((1u << lane) - 1u)), it);
    __syncthreads();
    return m;
}

// One level of the emit for block `blk` of T threads (T = C at level 0).  Level
// 0 (SRC not EMIT_ITEMS): the items are triangles blk*C .. blk*C+C-1; otherwise the
// items left by blocks blk*EMIT_GROUP .. of the previous level (in_count[k]
// items at in[k * EMIT_FMAX]).  Leaves the block's own items at
// out[blk * EMIT_FMAX] and their number in out_count[blk].  The block stops
// joining once `leave` runs or fewer are left (leave <= EMIT_FMAX; 32: join
// down to one warp's runs, as the root's level must).
//
// Level 0 makes its triangles' records itself and keeps their boxes in
// registers: it performs the permutation of a build (SRC = EMIT_PERMUTE,
// permute_tri with `perm`) or a refit (EMIT_REFIT, refit_tri).  After a sort
// whose wait gave up (hdr->status) the values are not a permutation, and unsorted
// keys would give nodes that are their own descendants: the triangles then keep
// their order, and the tree is the leaf of triangle 0 alone, so that whatever
// reads it before the caller has seen RT_DEV_TIMEOUT stays in range and ends.
//
// `tris` is not __restrict__: at level 0 it is `perm.tris`, whose records the
// marks are written into.
enum EmitSource { EMIT_ITEMS, EMIT_PERMUTE, EMIT_REFIT };
template <int C, int T, EmitSource SRC = EMIT_ITEMS>
__device__ __forceinline__ void emit_level(EmitSmem<C, T>& S, uint32_t blk, uint32_t n,
                                           const uint32_t* __restrict__ skeys,
                                           const EmitItem* __restrict__ in,
                                           const uint32_t* __restrict__ in_count,
                                           uint32_t n_in, EmitItem* __restrict__ out,
                                           uint32_t* __restrict__ out_count,
                                           float4* __restrict__ nodes,
                                           float4* tris, int min_leaf,
                                           uint32_t leave, BvhHeader* __restrict__ hdr,
                                           uint32_t* __restrict__ status,
                                           const PermuteIO& perm = PermuteIO{}) {
    static_assert(C % T == 0 && T % 32 == 0 && T >= EMIT_FMAX, "block size");
    static_assert(SRC == EMIT_ITEMS || T == C, "a thread per triangle");
    const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
    WarpItem it;
    bool keep;
    uint32_t m;
    if constexpr (SRC != EMIT_ITEMS) {
        // level 0: warp w joins triangles b0 + 32w ..
        const bool failed = ld_dep(&hdr->status) != 0u;
        const uint32_t b0 = blk * (uint32_t)C, i = b0 + t;
        const uint32_t w0 = b0 + 32u * w;
        const uint32_t cnt = w0 < n ? min(32u, n - w0) : 0u;
        const bool have = i < n;
        const uint32_t k = have ? ld_dep(&skeys[i]) : 0u;
        uint32_t kprev = __shfl_up_sync(0xffffffffu, k, 1);
        if (lane == 0 && have && i > 0) kprev = ld_dep(&skeys[i - 1]);
        it.l = it.r = i;
        it.kl = it.kr = k;
        it.db = (!have || i == 0) ? ~0ull
                                  : (((uint64_t)(kprev ^ k) << 32) | (uint64_t)((i - 1) ^ i));
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (have) {
            if constexpr (SRC == EMIT_PERMUTE)
                permute_tri(i, perm, !failed, lo, hi);
            else
                refit_tri(i, perm, lo, hi);
        }
        it.lox = lo.x; it.loy = lo.y; it.loz = lo.z;
        it.hix = hi.x; it.hiy = hi.y; it.hiz = hi.z;
        it.ref = (int32_t)i;
        it.cnt = 1;
        const uint64_t edge = cnt ? delta_or_max(skeys, (int64_t)w0 + cnt - 1, n) : 0ull;
        if (n == 1 || failed) {
            if (i == 0) {
                hdr->root_ref = 0;
                hdr->root_cnt = 1;
                hdr->n_tris = n;
                hdr->root_lo = lo;
                hdr->root_hi = hi;
            }
            if (t == 0 && out_count) out_count[blk] = 0;
            return;
        }
        if (t == 0) S.edge = delta_or_max(skeys, (int64_t)min(b0 + (uint32_t)C, n) - 1, n);
        keep = warp_join<true>(it, cnt, edge, n, min_leaf, nodes, tris, S.scratch[w], hdr);
        m = gather_runs(S, it, keep);
    } else {
        // the items left by EMIT_GROUP blocks of the previous level, in order
        if (w == 0) {
            const uint32_t k = blk * EMIT_GROUP + lane;
            const uint32_t v = (lane < (uint32_t)EMIT_GROUP && k < n_in)
                                   ? min(ld_dep(&in_count[k]), (uint32_t)EMIT_FMAX) : 0u;
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += u;
            }
            if (lane < (uint32_t)EMIT_GROUP) S.goff[lane] = x - v;
            if (lane == 31) S.goff[EMIT_GROUP] = x;
        }
        __syncthreads();
        m = S.goff[EMIT_GROUP];
        for (uint32_t e = t; e < m; e += T) {
            int g = 0;
            while (g + 1 < EMIT_GROUP && S.goff[g + 1] <= e) ++g;
            read_item(in + (size_t)(blk * EMIT_GROUP + g) * EMIT_FMAX + (e - S.goff[g]), it);
            S.list.store(e, it);
        }
        __syncthreads();   // the last item may have been copied by another thread
        if (t == 0 && m) S.edge = delta_or_max(skeys, (int64_t)S.list.range[m - 1].y, n);
        __syncthreads();
    }
    // Join the gathered runs in chunks of at most 32, one chunk per warp,
    // until one warp holds them all or none can be joined inside the block.
    // A pass joins only nodes that lie inside one chunk, so passes alternate
    // between chunks aligned at multiples of 32 and chunks shifted by 16: if
    // a node inside the block is left, so is one whose two children are
    // adjacent runs, and those share a chunk in one of the two layouts.  Two
    // passes in a row without a join therefore mean that every run left has
    // its parent outside the block.
    uint32_t stalls = 0;
    for (uint32_t pass = 0;; ++pass) {
        if (m <= leave && leave > 32u) {
            // few enough to be items of the next level as they are: the
            // next level joins them (a block's passes get longer and emptier
            // as its runs thin out)
            for (uint32_t e = t; e < m; e += (uint32_t)T) {
                S.list.load(e, it);
                write_item(&out[(size_t)blk * EMIT_FMAX + e], it);
            }
            if (t == 0 && out_count) out_count[blk] = m;
            return;
        }
        if (m <= 32u) {
            if (w == 0) {
                const uint32_t cnt = m;
                if (lane < cnt) S.list.load(lane, it);
                keep = warp_join<false>(it, cnt, S.edge, n, min_leaf, nodes, tris, S.scratch[0], hdr);
                const unsigned bal = __ballot_sync(0xffffffffu, keep);
                if (keep) write_item(&out[(size_t)blk * EMIT_FMAX + __popc(bal & ((1u << lane) - 1u))], it);
                if (lane == 0 && out_count) out_count[blk] = __popc(bal);
            }
            return;
        }
        if (stalls >= 2u || pass >= 2u * (uint32_t)C + 4u) {
            if (stalls < 2u && t == 0) atomicOr(status, RT_DEV_BADINDEX);
            // every run left has its parent outside the block: all of them,
            // in order, are items of the next level
            const uint32_t nf = min(m, (uint32_t)EMIT_FMAX);
            for (uint32_t e = t; e < nf; e += (uint32_t)T) {
                S.list.load(e, it);
                write_item(&out[(size_t)blk * EMIT_FMAX + e], it);
            }
            if (t == 0) {
                if (m > (uint32_t)EMIT_FMAX) atomicOr(status, RT_DEV_OVERFLOW);
                if (out_count) out_count[blk] = nf;
            }
            return;
        }
        // chunk c is [0, off) for c == 0, else [off + 32(c-1), off + 32c); the
        // block's warps take T / 32 chunks per round, and what a round leaves
        // goes to the front of the list, over chunks that are done
        const uint32_t off = ((pass & 1u) && m + 16u <= (uint32_t)C) ? 16u : 32u;
        uint32_t m_new = 0u;
        for (uint32_t r0 = 0u; r0 == 0u || off + 32u * (r0 - 1u) < m; r0 += (uint32_t)(T / 32)) {
            const uint32_t c = r0 + w;
            const uint32_t c0 = c == 0 ? 0u : off + 32u * (c - 1u);
            const uint32_t c1 = min(m, off + 32u * c);
            const uint32_t cnt = c0 < m ? c1 - c0 : 0u;
            if (lane < cnt) S.list.load(c0 + lane, it);
            const uint64_t edge = c1 < m ? S.list.db[c1] : S.edge;
            if (C == T) __syncthreads();   // the chunks are read: their space is the warps' scratch
            keep = warp_join<false>(it, cnt, edge, n, min_leaf, nodes, tris, S.scratch[w], hdr);
            m_new += gather_runs(S, it, keep, m_new);
            if (C == T) break;
        }
        stalls = m_new == m ? stalls + 1u : 0u;
        m = m_new;
    }
}


}  // namespace rt
