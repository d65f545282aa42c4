// rt_internal.cuh — device-side data layout and exact-arithmetic helpers shared
// by the LBVH builder and the tracer.  Every translation unit is compiled with
// --fmad=false: single-precision arithmetic is evaluated in the reference
// kernels' operation order without contraction, so results are bit-identical
// to the IEEE restatement of the reference math.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rt_cuda.h"

namespace rt {

// --------------------------------------------------------------------------
// BVH layout in HBM
// --------------------------------------------------------------------------
// Every interior node of the binary tree has a record of its four
// grandchildren (128 B = 8 x float4), indexed by the split position of the
// radix tree node (the last triangle of its left part): slots 0 and 1 are the
// children of its left child, 2 and 3 those of its right child, 32 B each:
//   lo.x lo.y hi.x hi.y lo.z hi.z code aux
//   inner grandchild:  code = its record,            aux = the child's record
//   leaf grandchild:   code = ~(first triangle),     aux = its triangle count
// A child that is a leaf itself takes the first slot of its pair; the second
// is then empty: a box at +infinity (no ray with a finite slab hits it), the
// leaf's code again and aux = -1.  A traversal enters two binary levels by
// reading one record: it waits for memory half as often as one that reads a
// 64 B pair of children per level, for the same bytes per two levels.  The
// corners are laid out so that one 256-bit load gives the register pairs of
// the two-lane slab arithmetic (trace_dev.cuh).
struct BvhHeader {
    int32_t root_ref;       // interior node index, or first triangle of a root leaf
    int32_t root_cnt;       // 0: interior root; > 0: the whole tree is one leaf
    uint32_t n_tris;
    uint32_t status;        // RT_DEV_TIMEOUT: a wait of the build's sort gave up (no tree)
    float4 root_lo;
    float4 root_hi;
};

// Slot of a node record.
struct Slot {
    float lox, loy, hix, hiy, loz, hiz;
    int32_t code, aux;
};
constexpr int32_t EMPTY_SLOT = -1;   // aux of the slot beside a leaf child

// Whether the child whose second slot is b is a leaf, and else the child's
// record from its first slot a: a's aux, or, a being a leaf, the triangle
// where the child splits, a's last.
__host__ __device__ __forceinline__ bool slot_pair_is_leaf(const Slot& b) { return b.aux == EMPTY_SLOT; }
__host__ __device__ __forceinline__ int32_t slot_pair_node(const Slot& a) {
    return a.code >= 0 ? a.aux : ~a.code + a.aux - 1;
}

// Triangle records in sorted order, 48 B: v0, e1 = v1 - v0, e2 = v2 - v0
// (the same float subtractions as leaf_hit, trace-bvh.cl:297-298).  v0.w is
// 1 where the next triangle belongs to the same leaf, else 0: a leaf is found
// from its first triangle alone.  Three records past the last are allocated.
struct TriRec {
    float4 v0, e1, e2;
};

// Render kernel variants a context keeps per-variant state for.
constexpr int kMaxRenderVariants = 32;
// The pooled kernel of large frames, the one with four lanes per pixel, and the
// choice between them by the size of the frame, which is the default.
constexpr int kPoolVariant = 9, kQuadVariant = 15, kAutoVariant = 16;

// Views passed to kernels.
struct SceneView {
    const float4* __restrict__ nodes;     // 8 float4 per record
    const float4* __restrict__ tris;      // 3 float4 per triangle
    const uint32_t* __restrict__ idx;     // sorted index buffer (3 per tri)
    const float4* __restrict__ nrm;       // vertex normals
    const uint32_t* __restrict__ map;     // sorted material map
    const rt_material* __restrict__ mats;
    const BvhHeader* __restrict__ hdr;
};

// --------------------------------------------------------------------------
// exact float3 helpers (operation order of the OpenCL built-ins as restated)
// --------------------------------------------------------------------------
struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk3(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 ld3(const float4& v) { return f3{v.x, v.y, v.z}; }
__device__ __forceinline__ f3 add(f3 a, f3 b) { return mk3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ f3 sub(f3 a, f3 b) { return mk3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ f3 mul(f3 a, f3 b) { return mk3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ f3 muls(f3 a, float s) { return mk3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ f3 neg(f3 a) { return mk3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
    return mk3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
// normalize(v) = v * (1 / sqrt(dot(v, v))), zero vector unchanged
// (correctly rounded sqrt and division: -prec-sqrt / -prec-div defaults).
__device__ __forceinline__ f3 normalize(f3 v) {
    float d = dot(v, v);
    if (d == 0.0f) return v;
    float inv = 1.0f / sqrtf(d);
    return muls(v, inv);
}
__device__ __forceinline__ float clamp01(float x) { return fminf(fmaxf(x, 0.0f), 1.0f); }
// OpenCL max / min ("y if x < y, else x"), used by the shadow slab test.
__device__ __forceinline__ float cl_max(float x, float y) { return (x < y) ? y : x; }
__device__ __forceinline__ float cl_min(float x, float y) { return (y < x) ? y : x; }

// Ray state during traversal.  Axes whose |1/d| <= 1e-6 are excluded from the
// slab test by the reference (trace-bvh.cl:262-270); storing NaN in those
// lanes gives the same result without branches, because fmin/fmax (and the
// OpenCL max/min as used) return the non-NaN operand.
struct TRay {
    f3 o, d, inv;   // inv: masked inverse direction
    float tmin;
};

__device__ __forceinline__ float mask_inv(float inv) {
    return fabsf(inv) > 1e-6f ? inv : __int_as_float(0x7fc00000);
}

__device__ __forceinline__ TRay make_tray(f3 o, f3 d, f3 inv, float tmin) {
    TRay r;
    r.o = o;
    r.d = d;
    r.inv = mk3(mask_inv(inv.x), mask_inv(inv.y), mask_inv(inv.z));
    r.tmin = tmin;
    return r;
}

// Three-operand min / max (sm_100+): exact selections with the same NaN
// rule as fminf / fmaxf (a NaN operand is dropped), so chaining them gives the
// same value as the reference's two-operand sequence.
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Slab test of bbox_hit (trace-bvh.cl:247-273).  Returns the entry distance A
// = max(tMin, per-axis near) and whether A <= min(tMax, per-axis far).  The
// per-axis selections are exact, so their grouping does not change A.
__device__ __forceinline__ bool slab(const TRay& r, float tmax, float lox, float loy, float loz,
                                     float hix, float hiy, float hiz, float& A) {
    float ltx = (lox - r.o.x) * r.inv.x, htx = (hix - r.o.x) * r.inv.x;
    float lty = (loy - r.o.y) * r.inv.y, hty = (hiy - r.o.y) * r.inv.y;
    float ltz = (loz - r.o.z) * r.inv.z, htz = (hiz - r.o.z) * r.inv.z;
    const float tmin = fmaxf(max3f(r.tmin, fminf(ltx, htx), fminf(lty, hty)), fminf(ltz, htz));
    tmax = fminf(min3f(tmax, fmaxf(ltx, htx), fmaxf(lty, hty)), fmaxf(ltz, htz));
    A = tmin;
    return tmin <= tmax;
}

// Slab test of the shadow kernel (shadow-trace-bvh.cl:160-186, OpenCL max/min).
__device__ __forceinline__ bool slab_shadow(const TRay& r, float tmax, float lox, float loy,
                                            float loz, float hix, float hiy, float hiz) {
    float ltx = (lox - r.o.x) * r.inv.x, htx = (hix - r.o.x) * r.inv.x;
    float lty = (loy - r.o.y) * r.inv.y, hty = (hiy - r.o.y) * r.inv.y;
    float ltz = (loz - r.o.z) * r.inv.z, htz = (hiz - r.o.z) * r.inv.z;
    float tmin = r.tmin;
    tmin = cl_max(tmin, cl_min(ltx, htx));
    tmax = cl_min(tmax, cl_max(ltx, htx));
    tmin = cl_max(tmin, cl_min(lty, hty));
    tmax = cl_min(tmax, cl_max(lty, hty));
    tmin = cl_max(tmin, cl_min(ltz, htz));
    tmax = cl_min(tmax, cl_max(ltz, htz));
    return tmin <= tmax;
}

// Slot k of record p, by one 256-bit load.
__device__ __forceinline__ Slot load_slot(const float4* __restrict__ nodes, int32_t p, int k) {
    Slot s;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(s.lox), "=f"(s.loy), "=f"(s.hix), "=f"(s.hiy), "=f"(s.loz), "=f"(s.hiz),
          "=r"(s.code), "=r"(s.aux)
        : "l"(nodes + 8 * (size_t)p + 2 * k));
    return s;
}

__device__ __forceinline__ void swap_if(bool c, int32_t& a, int32_t& b, float& ta, float& tb) {
    const int32_t x = c ? b : a, y = c ? a : b;
    const float u = c ? tb : ta, v = c ? ta : tb;
    a = x;
    b = y;
    ta = u;
    tb = v;
}

__device__ __forceinline__ TriRec load_tri(const float4* __restrict__ tris, int32_t i) {
    const float4* q = tris + 3 * (size_t)i;
    return TriRec{__ldg(q), __ldg(q + 1), __ldg(q + 2)};
}

// Möller–Trumbore of leaf_hit (trace-bvh.cl:275-328).  Its rejections come
// together at the end: the values computed past a rejection are not used, and
// the few extra operations cost less than four branches that a warp rarely
// takes together.
__device__ __forceinline__ bool mt(const TriRec& T, f3 o, f3 d, float& t, float& u, float& v) {
    f3 v0 = ld3(T.v0), e1 = ld3(T.e1), e2 = ld3(T.e2);
    f3 h = cross(d, e2);
    float aa = dot(e1, h);
    float f = 1.0f / aa;
    f3 s = sub(o, v0);
    u = f * dot(s, h);
    f3 q = cross(s, e1);
    v = f * dot(d, q);
    t = f * dot(e2, q);
    return !(aa > -1e-26f && aa < 1e-26f) & !(u < 0.0f) & !(u > 1.0f) & !(v < 0.0f) & !(u + v > 1.0f);
}

}  // namespace rt
