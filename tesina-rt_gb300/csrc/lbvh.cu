// lbvh.cu — LBVH construction of one scene for sm_103a.
//
// Stages (the reference's BVHBuilder::build_lbvh, src/rt/bvh-builder.cpp:201-741):
//   k_bounds        per-triangle AABB (build_primitive_bbox, bvh-builder.cl:100-130)
//                   reduced to the scene AABB (max_local_bbox, :318-391) with
//                   order-free integer min/max atomics;
//   k_morton_hist   morton_encode (:181-252) fused with the digit histograms of
//                   every radix pass;
//   k_onesweep      stable LSD radix pass, 8-bit digits, warp-level
//                   ballot ranking and decoupled look-back with a
//                   bounded spin (replaces the bitonic network of
//                   bvh-builder-sort.cl and bvh-builder.cpp:361-454);
//   k_emit_level0   rearrange_indices / rearrange_map (:49-72) and the
//                   triangle records used by traversal, fused with level 0 of
//                   the emit, which joins the triangles with their AABBs
//                   still in registers; a refit's instance makes the records
//                   and AABBs from the moved vertices;
//   k_emit_level    bottom-up build of the radix tree (Apetrei's
//                   agglomerative formulation of Karras' tree), collapsed to
//                   the reference's leaf rule (find_middle, :484-552), with
//                   every AABB (build_leaf_bbox / build_node_bbox, :262-311)
//                   computed on the way up; a few launches whose warps join
//                   runs of 32 items (level 0 over 512 triangles per block,
//                   then over what 8 blocks left).
//   k_permute       the permutation alone (under a tree built on the host).
// The per-element work lives in lbvh_dev.cuh, shared with the many-scene
// persistent build of batch.cu.
#include <cuda_runtime.h>
#include <stdint.h>
#include <mutex>
#include <vector>

#include "lbvh.cuh"
#include "lbvh_dev.cuh"
#include "rt_internal.cuh"

// Radix passes of 8-bit digits (10-bit ones were slower: a tile's fixed work
// grows with the digit count).
constexpr int kBuildBits = 8;
constexpr int kBuildRadix = 1 << kBuildBits;
constexpr int kMaxBuildPasses = 4;

namespace rt {

// Programmatic dependent launch.  The build's kernels after the first are
// launched while their predecessor still runs (launch_dep); each waits at
// its start for the predecessor grid to finish and its writes to be visible
// (griddepcontrol.wait, which returns at once for a kernel launched without
// the dependency), then lets its own successor launch.  It hides the
// launches' latency: the mid-scale build took 0.2752-0.2772 ms against
// 0.2802 ms without it, the 17.7 M-triangle build 2.584-2.589 against
// 2.604-2.605 ms (three alternating runs each, one box).
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... KArgs, typename... Args>
static cudaError_t launch_dep(void (*kern)(KArgs...), unsigned grid, unsigned block, size_t smem,
                              cudaStream_t s, bool dependent, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

__global__ void __launch_bounds__(256) k_bounds(const float4* __restrict__ pos,
                                                const uint32_t* __restrict__ idx, uint32_t n,
                                                uint32_t* __restrict__ bounds,
                                                uint4* __restrict__ clear, uint32_t clear_n,
                                                uint32_t* __restrict__ build_status) {
    pdl_enter();
    if (blockIdx.x == 0 && threadIdx.x == 0) *build_status = 0u;
    // the later kernels' counters are cleared here, beside the gathers
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < clear_n; i += gridDim.x * blockDim.x)
        clear[i] = make_uint4(0u, 0u, 0u, 0u);
    float lo[3] = {1e37f, 1e37f, 1e37f}, hi[3] = {-1e37f, -1e37f, -1e37f};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float tl[3], th[3];
        tri_aabb(pos, idx, i, tl, th);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = fminf(lo[c], tl[c]);
            hi[c] = fmaxf(hi[c], th[c]);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], off));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], off));
        }
    __shared__ float s[8][6];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0)
        for (int c = 0; c < 3; ++c) {
            s[w][c] = lo[c];
            s[w][3 + c] = hi[c];
        }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int c = threadIdx.x;
        float a = s[0][c], b = s[0][3 + c];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            a = fminf(a, s[k][c]);
            b = fmaxf(b, s[k][3 + c]);
        }
        bounds_add(bounds, c, a, b);
    }
}

__global__ void __launch_bounds__(256) k_morton_hist(const float4* __restrict__ pos,
                                                     const uint32_t* __restrict__ idx, uint32_t n,
                                                     const uint32_t* __restrict__ bounds, int depth,
                                                     int passes, uint32_t* __restrict__ keys,
                                                     uint32_t* __restrict__ hist) {
    pdl_enter();
    __shared__ uint32_t sh[kMaxBuildPasses][kBuildRadix];
    for (int i = threadIdx.x; i < kMaxBuildPasses * kBuildRadix; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
    const MortonParams P = morton_params(bounds, depth);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float lo[3], hi[3];
        tri_aabb(pos, idx, i, lo, hi);
        const uint32_t code = morton_code(P, lo, hi);
        keys[i] = code;
        for (int p = 0; p < passes; ++p)
            atomicAdd(&sh[p][(code >> (kBuildBits * p)) & (uint32_t)(kBuildRadix - 1)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kBuildRadix; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(&hist[i], v);
    }
}

// Digit histograms of every radix pass over plain keys (the sort without the
// fused Morton stage).
__global__ void __launch_bounds__(256) k_radix_hist(const uint32_t* __restrict__ keys, uint32_t n,
                                                    int passes, uint32_t* __restrict__ hist) {
    __shared__ uint32_t sh[4][256];
    for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t code = __ldg(&keys[i]);
        for (int p = 0; p < passes; ++p) atomicAdd(&sh[p][(code >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(&hist[i], v);
    }
}

// One radix pass of 8-bit digits; dynamic shared memory of sizeof(SortSmem).
// MINB tiles resident per SM bound the registers: a pass whose tiles all fit in
// one wave at 2 per SM runs the MINB = 2 instance (7 % faster per mid-scale
// build), a longer one SORT_MINB (3, 80 registers: the third tile hides
// latency).
template <int MINB>
__global__ void __launch_bounds__(SORT_THREADS, MINB) k_onesweep(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
    uint32_t* __restrict__ vout, uint32_t n, int shift, const uint32_t* __restrict__ hist,
    uint32_t* __restrict__ lookback, uint32_t* __restrict__ tile_ctr, uint32_t* __restrict__ status,
    uint32_t* __restrict__ failed) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char sort_smem[];
    auto& S = *reinterpret_cast<SortSmem*>(sort_smem);
    if (threadIdx.x == 0) S.tile = atomicAdd(tile_ctr, 1u);   // tiles in launch order
    __syncthreads();
    onesweep_tile<>(S, S.tile, kin, vin, kout, vout, n, shift, hist, lookback, status, failed);
}

constexpr int kOneWaveMinB = 2;
// The instance for a pass of `tiles` tiles on `sms` SMs.
static auto onesweep_kernel(size_t tiles, int sms) {
    return tiles <= (size_t)kOneWaveMinB * (size_t)sms ? k_onesweep<kOneWaveMinB>
                                                       : k_onesweep<SORT_MINB>;
}

// Self-test of the look-back timeout: one block sorts tile 1 of a pass
// whose tile 0 is never launched, so its look-back word stays unpublished;
// with a spin limit of 1,024 polls the wait gives up at once.
constexpr uint32_t kProbeSpinLimit = 1024;
__global__ void __launch_bounds__(SORT_THREADS, 1) k_onesweep_wait_probe(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
    uint32_t* __restrict__ vout, uint32_t n, const uint32_t* __restrict__ hist,
    uint32_t* __restrict__ lookback, uint32_t* __restrict__ status, uint32_t* __restrict__ failed) {
    __shared__ SortSmem S;
    onesweep_tile<SORT_ITEMS, kProbeSpinLimit>(S, 1, kin, vin, kout, vout, n, 0, hist, lookback,
                                               status, failed);
}

// The permutation of a tree built on the host, whose leaf marks (1: the next
// triangle is in the same leaf) come from there too.
__global__ void __launch_bounds__(256) k_permute(uint32_t n, PermuteIO P,
                                                  const uint8_t* __restrict__ more) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 lo, hi;
        permute_tri(i, P, true, lo, hi);
        if (more[i]) P.tris[3 * (size_t)i].w = 1.0f;
    }
}

// One level of the emit above level 0 (emit_level), one block of T threads per
// EMIT_GROUP blocks of the level below.
template <int T>
__global__ void __launch_bounds__(T, T == EMIT_T_WIDE ? 2 : 1) k_emit_level(
    uint32_t n, const uint32_t* __restrict__ skeys, const EmitItem* __restrict__ in,
    const uint32_t* __restrict__ in_count, uint32_t n_in, EmitItem* __restrict__ out,
    uint32_t* __restrict__ out_count, float4* __restrict__ nodes, float4* __restrict__ tris,
    int min_leaf, uint32_t leave, BvhHeader* __restrict__ hdr, uint32_t* __restrict__ status) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char emit_smem[];
    auto& S = *reinterpret_cast<EmitSmem<EMIT_C1, T>*>(emit_smem);
    emit_level<EMIT_C1, T>(S, blockIdx.x, n, skeys, in, in_count, n_in, out, out_count, nodes, tris,
                        min_leaf, leave, hdr, status);
}

// Level 0: each block first makes its own triangles' records (permuting
// index buffer, material map and upload ids in a build) and joins them with
// their boxes still in registers, so no leaf AABB goes through memory.
template <EmitSource SRC>
__global__ void __launch_bounds__(EMIT_C0, EMIT_MINB0) k_emit_level0(
    uint32_t n, const uint32_t* __restrict__ skeys, PermuteIO P, EmitItem* __restrict__ out,
    uint32_t* __restrict__ out_count, float4* __restrict__ nodes, int min_leaf, uint32_t leave,
    BvhHeader* __restrict__ hdr, uint32_t* __restrict__ status) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char emit_smem[];
    auto& S = *reinterpret_cast<EmitSmem<EMIT_C0, EMIT_C0>*>(emit_smem);
    emit_level<EMIT_C0, EMIT_C0, SRC>(S, blockIdx.x, n, skeys, nullptr, nullptr, 0, out, out_count, nodes,
                             P.tris, min_leaf, leave, hdr, status, P);
}

static size_t sort_scratch_bytes(uint32_t n, int passes) {
    const size_t tiles = ((size_t)n + SORT_TILE - 1) / SORT_TILE;
    return (sizeof(uint32_t) * (8 + (size_t)kMaxBuildPasses * kBuildRadix + 4 +
                                (size_t)passes * tiles * kBuildRadix) + 255) & ~(size_t)255;
}

static size_t emit_scratch_bytes(uint32_t n) { return emit_buffers_bytes(n); }

// The emit's levels: level 0 over triangles, then levels over the items left
// by EMIT_GROUP blocks each until a single block reaches the root.  Item
// buffers alternate: A holds level 0, 2, ... and B level 1, 3, ....  Level 0
// performs the permutation `perm` (SRC = EMIT_PERMUTE) or the refit of the
// triangles in their order.
// The shared-memory opt-ins of the kernels with dynamic shared memory (a
// property of the kernel on each device), once per device.
static cudaError_t setup_kernels() {
    static std::mutex mu;
    static uint64_t done = 0;   // devices 0..63 set up
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 64 && ((done >> dev) & 1)) return cudaSuccess;
    auto opt_in = [&](const void* f, size_t bytes) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    opt_in((const void*)k_emit_level0<EMIT_PERMUTE>, sizeof(EmitSmem<EMIT_C0, EMIT_C0>));
    opt_in((const void*)k_emit_level0<EMIT_REFIT>, sizeof(EmitSmem<EMIT_C0, EMIT_C0>));
    opt_in((const void*)k_emit_level<EMIT_T_WIDE>, sizeof(EmitSmem<EMIT_C1, EMIT_T_WIDE>));
    opt_in((const void*)k_emit_level<EMIT_T_NARROW>, sizeof(EmitSmem<EMIT_C1, EMIT_T_NARROW>));
    opt_in((const void*)k_onesweep<kOneWaveMinB>, sizeof(SortSmem));
    opt_in((const void*)k_onesweep<SORT_MINB>, sizeof(SortSmem));
    if (e != cudaSuccess) return e;
    if (dev < 64) done |= 1ull << dev;
    return cudaSuccess;
}

template <EmitSource SRC>
static cudaError_t launch_emit(const LbvhArgs& a, uint8_t* emit_scratch, const PermuteIO& perm,
                               cudaStream_t s) {
    const uint32_t n = a.n;
    if (cudaError_t e0 = setup_kernels()) return e0;
    const uint32_t nb0 = emit_blocks0(n);
    const EmitBuffers B = emit_buffers(n, emit_scratch);
    // a refit starts here, after whatever moved the vertices: an ordinary launch
    cudaError_t e = launch_dep(k_emit_level0<SRC>, nb0, EMIT_C0, sizeof(EmitSmem<EMIT_C0, EMIT_C0>),
                               s, SRC == EMIT_PERMUTE, n, (const uint32_t*)a.keys_sorted, perm,
                               B.items[0], B.counts[0], a.nodes, a.min_leaf, emit_leave(0, nb0),
                               a.hdr, a.status);
    if (e) return e;
    uint32_t n_in = nb0;
    int src = 0;
    while (n_in > 1) {
        const uint32_t g = emit_next_level(n_in);
        const bool wide = g > (uint32_t)a.num_sms;
        e = launch_dep(wide ? k_emit_level<EMIT_T_WIDE> : k_emit_level<EMIT_T_NARROW>, g,
                       wide ? EMIT_T_WIDE : EMIT_T_NARROW,
                       wide ? sizeof(EmitSmem<EMIT_C1, EMIT_T_WIDE>)
                            : sizeof(EmitSmem<EMIT_C1, EMIT_T_NARROW>),
                       s, true, n, (const uint32_t*)a.keys_sorted, (const EmitItem*)B.items[src],
                       (const uint32_t*)B.counts[src], n_in, B.items[src ^ 1], B.counts[src ^ 1],
                       a.nodes, a.tris, a.min_leaf, emit_leave(1, g), a.hdr, a.status);
        if (e) return e;
        n_in = g;
        src ^= 1;
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------

static int grid_for(uint32_t n, int threads, int max_blocks) {
    int64_t b = ((int64_t)n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > max_blocks) b = max_blocks;
    return (int)b;
}

size_t lbvh_scratch_bytes(uint32_t n, int passes) {
    return sort_scratch_bytes(n, passes) + emit_scratch_bytes(n);
}

size_t lbvh_emit_offset(uint32_t n) { return sort_scratch_bytes(n, kMaxBuildPasses); }

cudaError_t lbvh_build(const LbvhArgs& a, cudaStream_t s) {
    const uint32_t n = a.n;
    const int passes = (a.depth + kBuildBits - 1) / kBuildBits;
    const size_t tiles = ((size_t)n + SORT_TILE - 1) / SORT_TILE;
    // scratch: bounds[8] | hist[passes max * radix] | tile_ctr[4] |
    // lookback[passes * tiles * radix]
    uint32_t* bounds = a.scratch;
    uint32_t* hist = bounds + 8;
    uint32_t* tile_ctr = hist + kMaxBuildPasses * kBuildRadix;
    uint32_t* lookback = tile_ctr + 4;
    cudaError_t e = setup_kernels();
    if (e) return e;
    e = cudaMemsetAsync(bounds, 0, 8 * sizeof(uint32_t), s);
    if (e) return e;
    static_assert((kMaxBuildPasses * kBuildRadix + 4) % 4 == 0 && kBuildRadix % 4 == 0, "whole uint4");
    const size_t clear = (kMaxBuildPasses * kBuildRadix + 4 + (size_t)passes * tiles * kBuildRadix) / 4;
    const int sms = a.num_sms;
    k_bounds<<<grid_for(n, 256, sms * 8), 256, 0, s>>>(a.pos, a.idx_in, n, bounds,
                                                       reinterpret_cast<uint4*>(hist), (uint32_t)clear,
                                                       &a.hdr->status);
    e = launch_dep(k_morton_hist, grid_for(n, 256, sms * 8), 256, 0, s, true, a.pos, a.idx_in, n,
                   bounds, a.depth, passes, a.keys_unsorted, hist);
    if (e) return e;
    const uint32_t* kin = a.keys_unsorted;
    const uint32_t* vin = nullptr;   // the first pass makes the values 0..n-1 itself
    uint32_t* kbuf[2] = {a.keys1, a.keys_sorted};
    uint32_t* vbuf[2] = {a.vals1, a.vals_sorted};
    for (int p = 0; p < passes; ++p) {
        // the last pass always lands in keys_sorted / vals_sorted
        const int dst = ((passes - 1 - p) & 1) ? 0 : 1;
        e = launch_dep(onesweep_kernel(tiles, sms), (unsigned)tiles, SORT_THREADS,
                       sizeof(SortSmem), s, true, kin, vin, kbuf[dst], vbuf[dst], n,
                       kBuildBits * p, (const uint32_t*)(hist + kBuildRadix * p),
                       lookback + (size_t)p * tiles * kBuildRadix, tile_ctr + p, a.status,
                       &a.hdr->status);
        if (e) return e;
        kin = kbuf[dst];
        vin = vbuf[dst];
    }
    const PermuteIO P{a.vals_sorted, a.idx_in,  a.map_in,   a.orig_in, a.pos,
                      a.idx_out,     a.map_out, a.orig_out, a.tris};
    return launch_emit<EMIT_PERMUTE>(a, reinterpret_cast<uint8_t*>(a.scratch) + lbvh_emit_offset(n),
                                     P, s);
}

size_t radix_scratch_words(uint32_t n, int passes) {
    const size_t tiles = ((size_t)n + SORT_TILE - 1) / SORT_TILE;
    return 4 * 256 + 4 + (size_t)passes * tiles * 256;
}

int radix_tile_size() { return SORT_TILE; }

// The probe's scene of two tiles of triangles: what a build of it takes, and
// the words of the sort probe before it (keys | vals | hist[256] | lookback[2 * 256]).
constexpr uint32_t kProbeTris = 2 * SORT_TILE;
constexpr size_t kProbeSortWords = 2 * (size_t)kProbeTris + 3 * 256;
static size_t probe_bytes() {
    const size_t n = kProbeTris, words = kProbeSortWords + 2 * n + 10 * n;
    return 4 * words + 16 * (3 * (n + 3) + 8 * n + 1) + emit_scratch_bytes(kProbeTris) +
           sizeof(BvhHeader) + 256;
}

size_t wait_probe_words() { return (probe_bytes() + 3) / 4; }

cudaError_t wait_probe(uint32_t* buf, int num_sms, uint32_t* status, bool* kept, cudaStream_t s) {
    const uint32_t n = kProbeTris;
    cudaError_t e = cudaMemsetAsync(buf, 0, sizeof(uint32_t) * wait_probe_words(), s);
    if (e) return e;
    // 16-byte types first; all of it zero: every index is vertex 0, every
    // material 0
    LbvhArgs a{};
    a.n = n;
    a.depth = 30;
    a.min_leaf = 1;
    a.num_sms = num_sms;
    a.status = status;
    a.nodes = reinterpret_cast<float4*>(buf);   // 128-byte records
    a.tris = a.nodes + 8 * (size_t)n;
    float4* pos = a.tris + 3 * ((size_t)n + 3);
    a.pos = pos;
    a.hdr = reinterpret_cast<BvhHeader*>(pos + 1);
    uint8_t* emit = reinterpret_cast<uint8_t*>(a.hdr + 1);
    uint32_t* w = reinterpret_cast<uint32_t*>(emit + emit_scratch_bytes(n));
    auto take = [&](size_t words) {
        uint32_t* p = w;
        w += words;
        return p;
    };
    uint32_t* keys = take(n);
    uint32_t* vals = take(n);
    uint32_t* hist = take(256);
    uint32_t* lookback = take(2 * 256);
    a.keys_sorted = take(n);
    a.vals_sorted = take(n);
    uint32_t* idx = take(3 * (size_t)n);
    uint32_t* map = take(n);
    uint32_t* orig = take(n);
    a.idx_in = idx;
    a.map_in = map;
    a.orig_in = orig;
    a.idx_out = take(3 * (size_t)n);
    a.map_out = take(n);
    a.orig_out = take(n);
    // the sorted arrays' memory held something else before
    if ((e = cudaMemsetAsync(a.keys_sorted, 0xa5, 8 * (size_t)n, s))) return e;
    std::vector<uint32_t> ids(n);
    for (uint32_t i = 0; i < n; ++i) ids[i] = i ^ 5u;
    if ((e = cudaMemcpyAsync(orig, ids.data(), 4 * (size_t)n, cudaMemcpyHostToDevice, s))) return e;
    k_radix_hist<<<1, 256, 0, s>>>(keys, n, 1, hist);
    k_onesweep_wait_probe<<<1, SORT_THREADS, 0, s>>>(keys, vals, a.keys_sorted, a.vals_sorted, n,
                                                     hist, lookback, status, &a.hdr->status);
    const PermuteIO P{a.vals_sorted, a.idx_in,  a.map_in,   a.orig_in, a.pos,
                      a.idx_out,     a.map_out, a.orig_out, a.tris};
    if ((e = launch_emit<EMIT_PERMUTE>(a, emit, P, s))) return e;
    std::vector<uint32_t> got(n);
    BvhHeader h;
    if ((e = cudaMemcpyAsync(got.data(), a.orig_out, 4 * (size_t)n, cudaMemcpyDeviceToHost, s)) ||
        (e = cudaMemcpyAsync(&h, a.hdr, sizeof h, cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
        return e;
    *kept = got == ids && h.status == RT_DEV_TIMEOUT && h.root_ref == 0 && h.root_cnt == 1;
    return cudaGetLastError();
}

cudaError_t radix_sort_pairs(const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                             uint32_t* vout, uint32_t* ktmp, uint32_t* vtmp, uint32_t n,
                             int key_bits, uint32_t* scratch, uint32_t* status, int num_sms,
                             cudaStream_t s) {
    const int passes = (key_bits + 7) / 8;
    const size_t tiles = ((size_t)n + SORT_TILE - 1) / SORT_TILE;
    uint32_t* hist = scratch;
    uint32_t* tile_ctr = hist + 4 * 256;
    uint32_t* lookback = tile_ctr + 4;
    cudaError_t e = setup_kernels();
    if (e) return e;
    e = cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * radix_scratch_words(n, passes), s);
    if (e) return e;
    if (n == 0) return cudaSuccess;
    k_radix_hist<<<grid_for(n, 256, num_sms * 8), 256, 0, s>>>(kin, n, passes, hist);
    const uint32_t* ki = kin;
    const uint32_t* vi = vin;
    for (int p = 0; p < passes; ++p) {
        const bool to_out = ((passes - 1 - p) & 1) == 0;
        uint32_t* ko = to_out ? kout : ktmp;
        uint32_t* vo = to_out ? vout : vtmp;
        onesweep_kernel(tiles, num_sms)<<<(unsigned)tiles, SORT_THREADS, sizeof(SortSmem), s>>>(
            ki, vi, ko, vo, n, 8 * p, hist + 256 * p, lookback + (size_t)p * tiles * 256,
            tile_ctr + p, status, nullptr);
        ki = ko;
        vi = vo;
    }
    return cudaGetLastError();
}

cudaError_t lbvh_permute(const LbvhArgs& a, const uint32_t* order, const uint8_t* more,
                         cudaStream_t s) {
    const PermuteIO P{order,     a.idx_in,  a.map_in,   a.orig_in, a.pos,
                      a.idx_out, a.map_out, a.orig_out, a.tris};
    k_permute<<<grid_for(a.n, 256, a.num_sms * 16), 256, 0, s>>>(a.n, P, more);
    return cudaGetLastError();
}

cudaError_t lbvh_refit(const LbvhArgs& a, cudaStream_t s) {
    // the emit is deterministic in the sorted keys, so rerunning it on the
    // same keys reproduces the same topology with the new boxes
    const PermuteIO P{nullptr,   nullptr, nullptr, nullptr, a.pos,
                      a.idx_out, nullptr, nullptr, a.tris};
    return launch_emit<EMIT_REFIT>(a, reinterpret_cast<uint8_t*>(a.scratch) + lbvh_emit_offset(a.n),
                                   P, s);
}

}  // namespace rt
