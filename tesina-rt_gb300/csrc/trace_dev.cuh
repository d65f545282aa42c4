// trace_dev.cuh — device-side traversal, shading and ray generation shared by
// the one-scene kernels (trace.cu) and the many-scene render (batch.cu).
//
// Device functions restate, in the reference's operation order:
//   closest_hit   trace_ray / leaf_hit / bbox_hit (src/kernel/trace-bvh.cl:247-417)
//   any_hit       trace_shadow_ray / leaf_hit_any (src/kernel/shadow-trace-bvh.cl:160-315)
//   complete_hit  complete_trace_info (trace-bvh.cl:190-245)
//   shade_hit     shade_sample (src/kernel/ray-shader.cl:116-333), untextured
//   reflect_ray   generate_secondary_rays_disc reflection branch
//                 (src/kernel/secondary-ray-generator.cl:258-270)
//   primary_dir   generate_primary_rays (src/kernel/primary-ray-generator.cl:27-103)
//
// Traversal.  The reference walks a binary tree depth first, near child first
// where near = left iff dot(dir, right.lo - left.lo) > 0
// (trace-bvh.cl:391-409), tests a node's box when it reaches it and lets a
// later hit of equal t win.  The kernels walk two of its levels per step over
// four-wide records (rt_internal.cuh) and visit the same leaves in the same
// order.  A child's box lies inside its parent's, and the slab test is
// monotone in the box (IEEE subtraction and multiplication by one factor,
// minima and maxima), so a box that passes has ancestors that all passed, at
// this tMax or an earlier, larger one: which leaves the reference reaches is
// decided by the leaves' own boxes at their turn.  Inner boxes in between may
// be skipped; the order of the four grandchildren comes from the three sign
// tests of the two levels, on lower corners that the minima give exactly.  A
// pushed entry keeps its entry distance A and is dropped if A > tMax when
// popped (tMax only shrinks, the far distances do not change).  Monotonicity
// needs slabs without 0 * inf, and an empty slot's box at infinity must be out of
// reach.  Rays for which that is not sure (careful_ray) have searches of their
// own.  With an infinite inverse component, a ray parallel to an axis, a box that
// passes has a parent that passes unless the box is flat in that axis and lies in
// the ray's plane: the axis' slab is else no bound or empty, the parent's no bound
// where the box's is, and A comes from the other axes.  Such rays take the same
// steps until they meet a box of that kind (WIDE); from there on, and rays from
// infinite or NaN origins and the like always, the two binary levels are taken one
// at a time (BINARY).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rt_internal.cuh"

namespace rt {

struct Hit {
    int32_t id;
    float t, u, v;
};

// Leaf of a scene whose root is a leaf: `cnt` triangles.
__device__ __forceinline__ void leaf_closest(const SceneView& S, const TRay& r, int32_t start,
                                             int32_t cnt, Hit& best) {
    for (int32_t i = start; i < start + cnt; ++i) {
        float t, u, v;
        if (!mt(load_tri(S.tris, i), r.o, r.d, t, u, v)) continue;
        if (t <= best.t && t >= r.tmin) best = Hit{i, t, u, v};
    }
}

__device__ __forceinline__ bool leaf_any(const SceneView& S, const TRay& r, int32_t start,
                                         int32_t cnt, float tmax) {
    for (int32_t i = start; i < start + cnt; ++i) {
        float t, u, v;
        if (!mt(load_tri(S.tris, i), r.o, r.d, t, u, v)) continue;
        if (t < tmax && t > r.tmin) return true;
    }
    return false;
}

// Leaf of an inner node: from its first triangle to the first record whose
// `more` mark is clear.  PAIR: two records are read at a time, so that most
// leaves (at most three triangles with the usual minimum) wait for memory
// once; the second may lie one past the scene's last record, which is
// allocated.  Worth its registers where the kernel has them to spare: the
// stage kernels (6 % of a 1000 x 701 pipeline of 10k triangles) and the glass
// pool (2 %); the instanced render loses 8 % to spills.
template <bool PAIR>
__device__ __forceinline__ void leaf_closest(const SceneView& S, const TRay& r, int32_t i,
                                             Hit& best) {
    auto test = [&](const TriRec& T, int32_t id, bool valid) {
        float t, u, v;
        bool h = mt(T, r.o, r.d, t, u, v);   // before t is read: & does not order its operands
        h = h & (t <= best.t) & (t >= r.tmin) & valid;
        best.id = h ? id : best.id;
        best.t = h ? t : best.t;
        best.u = h ? u : best.u;
        best.v = h ? v : best.v;
    };
    bool more;
    do {
        const TriRec A = load_tri(S.tris, i);
        more = A.v0.w != 0.0f;
        if (PAIR) {
            const TriRec B = load_tri(S.tris, i + 1);
            test(A, i, true);
            test(B, i + 1, more);
            more = more & (B.v0.w != 0.0f);
            i += 2;
        } else {
            test(A, i, true);
            ++i;
        }
    } while (more);
}

template <bool PAIR>
__device__ __forceinline__ bool leaf_any(const SceneView& S, const TRay& r, int32_t i, float tmax) {
    auto test = [&](const TriRec& T) {
        float t, u, v;
        const bool h = mt(T, r.o, r.d, t, u, v);
        return h & (t < tmax) & (t > r.tmin);
    };
    bool more, hit;
    do {
        const TriRec A = load_tri(S.tris, i);
        more = A.v0.w != 0.0f;
        if (PAIR) {
            const TriRec B = load_tri(S.tris, i + 1);
            hit = test(A);
            hit = hit | (test(B) & more);
            more = more & (B.v0.w != 0.0f);
            i += 2;
        } else {
            hit = test(A);
            ++i;
        }
    } while (more & !hit);
    return hit;
}

// A ray's slab constants as register pairs for the two-lane f32 adds and
// multiplies (exact in each lane: lo + (-o) is lo - o).
struct SlabRay {
    float2 no_xy, no_zz, iv_xy, iv_zz;
    float tmin;
};
__device__ __forceinline__ SlabRay slab_ray(const TRay& r) {
    return SlabRay{make_float2(-r.o.x, -r.o.y), make_float2(-r.o.z, -r.o.z),
                   make_float2(r.inv.x, r.inv.y), make_float2(r.inv.z, r.inv.z), r.tmin};
}
// dot(d, b - a) > 0 for the lower corners a and b of two boxes, in dot()'s
// order (b - a as the two-lane b + a * -1, which rounds the same).
__device__ __forceinline__ bool near_first(f3 d, float ax, float ay, float az, float bx, float by,
                                           float bz) {
    float px, py;
    asm("{\n\t.reg .b64 a, b, c, m;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tmov.b64 m, {%8, %8};\n\t"
        "fma.rn.f32x2 a, a, m, b;\n\tmul.rn.f32x2 a, a, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(px), "=f"(py) : "f"(ax), "f"(ay), "f"(bx), "f"(by), "f"(d.x), "f"(d.y), "f"(-1.0f));
    return (px + py) + d.z * (bz - az) > 0.0f;
}
__device__ __forceinline__ float2 add_mul2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "add.rn.f32x2 a, a, b;\n\tmul.rn.f32x2 a, a, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

// The slab test of a slot, with the entry and exit distances (`slab`; also
// slab_shadow's result wherever no slab is NaN by 0 * inf: the two differ in
// their NaN rules only).
__device__ __forceinline__ bool slab_slot(const SlabRay& r, float tmax, const Slot& s, float& A,
                                          float& B) {
    const float2 l = add_mul2(make_float2(s.lox, s.loy), r.no_xy, r.iv_xy);
    const float2 h = add_mul2(make_float2(s.hix, s.hiy), r.no_xy, r.iv_xy);
    const float2 z = add_mul2(make_float2(s.loz, s.hiz), r.no_zz, r.iv_zz);
    A = fmaxf(max3f(r.tmin, fminf(l.x, h.x), fminf(l.y, h.y)), fminf(z.x, z.y));
    B = fminf(min3f(tmax, fmaxf(l.x, h.x), fmaxf(l.y, h.y)), fmaxf(z.x, z.y));
    return A <= B;
}

enum SearchKind { PLAIN, WIDE, BINARY };

// slab_slot for rays parallel to an axis: an empty slot is no hit (tMax may be
// infinite), and a hit sets `flat` if both slabs of an axis are NaN.  SHADOW:
// slab_shadow's rule, by which 0 * inf at the lower corner takes the axis out.
template <bool SHADOW>
__device__ __forceinline__ bool slab_wide(const SlabRay& r, float tmax, const Slot& s, float& A,
                                          float& B, bool& flat) {
    const float2 l = add_mul2(make_float2(s.lox, s.loy), r.no_xy, r.iv_xy);
    const float2 h = add_mul2(make_float2(s.hix, s.hiy), r.no_xy, r.iv_xy);
    const float2 z = add_mul2(make_float2(s.loz, s.hiz), r.no_zz, r.iv_zz);
    const float nx = fminf(l.x, h.x), ny = fminf(l.y, h.y), nz = fminf(z.x, z.y);
    float fx = fmaxf(l.x, h.x), fy = fmaxf(l.y, h.y), fz = fmaxf(z.x, z.y);
    float mx = nx, my = ny, mz = nz;
    if (SHADOW) {
        mx = l.x == l.x ? mx : l.x;
        fx = l.x == l.x ? fx : l.x;
        my = l.y == l.y ? my : l.y;
        fy = l.y == l.y ? fy : l.y;
        mz = z.x == z.x ? mz : z.x;
        fz = z.x == z.x ? fz : z.x;
    }
    A = fmaxf(max3f(r.tmin, mx, my), mz);
    B = fminf(min3f(tmax, fx, fy), fz);
    const bool hit = (A <= B) & (s.aux != EMPTY_SLOT);
    flat |= hit & ((nx != nx) | (ny != ny) | (nz != nz));
    return hit;
}

// Rays whose slab tests need not be monotone (see the top of the file); those of
// them for which a flat box is not the only reason; and rays whose bounds may take
// in an empty slot's box.
__device__ __forceinline__ bool finite_origin(const TRay& r) {
    const float INF = __int_as_float(0x7f800000);
    return fabsf(r.o.x) < INF && fabsf(r.o.y) < INF && fabsf(r.o.z) < INF;
}
__device__ __forceinline__ bool careful_ray(const TRay& r) {
    const float INF = __int_as_float(0x7f800000);
    const bool inf = fabsf(r.inv.x) == INF || fabsf(r.inv.y) == INF || fabsf(r.inv.z) == INF;
    const bool axis = r.inv.x == r.inv.x || r.inv.y == r.inv.y || r.inv.z == r.inv.z;
    return inf || !axis || !finite_origin(r);
}
__device__ __forceinline__ bool binary_ray(const TRay& r) {
    return !finite_origin(r) || !(r.tmin > -__int_as_float(0x7f800000));
}
__device__ __forceinline__ bool unbounded_ray(const TRay& r, float tmax) {
    const float INF = __int_as_float(0x7f800000);
    return !(tmax < INF) || !(r.tmin > -INF);
}

// The two binary children of a record in place of its four grandchildren:
// slot 0 and 2 become the left and right child, 1 and 3 are to be ignored.
__device__ __forceinline__ void binary_step(Slot& a, const Slot& b) {
    if (slot_pair_is_leaf(b)) return;   // the child is a leaf, in slot a alone
    const int32_t self = slot_pair_node(a);
    a.lox = fminf(a.lox, b.lox); a.loy = fminf(a.loy, b.loy); a.loz = fminf(a.loz, b.loz);
    a.hix = fmaxf(a.hix, b.hix); a.hiy = fmaxf(a.hiy, b.hiy); a.hiz = fmaxf(a.hiz, b.hiz);
    a.code = self;
}

// Stack entries: a path of 32 binary levels (the deepest tree: 32 key bits)
// is 16 steps, each of which leaves at most three entries behind.  A step that
// might push past the last entry writes over the top ones instead and raises
// RT_DEV_OVERFLOW when the search ends.
constexpr int STACK = 48;
constexpr int32_t NO_NODE = (int32_t)0x80000000;   // below every leaf code

// What bounds it: each step waits for one record (L1 / L2 latency) and the
// lanes of a warp take different numbers of steps; the mid-scale frame issues in
// 65 % of the cycles with 15 of 32 lanes.  Frames over binary records, one level and
// 64 B per step, took 1.6 to 2 times as long.
//
// Leaves, met directly or popped, are tested in one place, by the lanes that
// have one together: a lane that reaches a leaf waits until the lanes with a
// leaf are a third of those still searching (leaf_turn).  At once, a leaf step
// had 5.2-6.8 lanes where a node step had 17-18: 7-9 % of large frames, 18 % of
// the stage pipeline (a fixed 4 to 16 lanes gains less; setting a leaf aside and
// walking on loses 2-5 %; small frames lose 4 % and run by four lanes).  STAY: lanes
// whose search has ended stay for the votes, which keeps the warp together; 9 %
// faster in the stage kernels, 13 % in the one-path-per-lane kernels, faster too in
// the instanced render, slower in the pooled ones; there the leaves wait until they
// are half of the lanes (a third: instances 1.855 -> 1.849 ms, stage pipeline 517 ->
// 515 us).
template <bool STAY>
__device__ __forceinline__ bool leaf_turn(unsigned group, int32_t next, bool& ended) {
    if (STAY) {
        const unsigned lm = __ballot_sync(group, next < 0 && next != NO_NODE);
        const unsigned nm = __ballot_sync(group, next >= 0);
        ended = (lm | nm) == 0u;
        return __popc(lm) >= __popc(nm) && next < 0 && next != NO_NODE;
    }
    ended = next == NO_NODE;
    if (ended) return false;
    const unsigned am = __activemask(), lm = __ballot_sync(am, next < 0);
    return 3 * __popc(lm) >= __popc(am) && next < 0;
}

//
// The steps branch as little as they can: a step is a chain of dependent
// instructions, and each branch in it costs more than the selects that take
// its place.  The rejections of mt(), a leaf's hit, an any-hit visit and the
// pushes' conditions are selects, and the kind is a template argument, so that
// ordinary rays' code has none of its tests: together 9-21 % of a frame.  (Pushes
// that store always and move `sp` by the condition lose 4 %.)
// WIDE: `flat` tells that the search was given up at a flat box.
template <bool STAY, bool PAIR, SearchKind KIND>
__device__ __forceinline__ Hit closest_search(const SceneView& S, const BvhHeader& H, const TRay& r,
                                              float tmax, uint32_t* status, bool& flat) {
    Hit best{-1, tmax, 0.f, 0.f};
    int2 st[STACK];   // code, entry distance
    int sp = 0;
    bool over = false;
    const SlabRay w = slab_ray(r);
    const float MISS = __int_as_float(0x7fc00000);   // NaN: an entry distance never is
    const unsigned group = STAY ? __activemask() : 0u;
    int32_t next = H.root_ref;
    auto pop = [&]() {
        next = NO_NODE;
        while (sp > 0) {
            const int2 e = st[--sp];
            if (__int_as_float(e.y) <= best.t) {
                next = e.x;
                break;
            }
        }
    };
    auto node = [&](int32_t cur) {
        Slot s0 = load_slot(S.nodes, cur, 0), s1 = load_slot(S.nodes, cur, 1),
             s2 = load_slot(S.nodes, cur, 2), s3 = load_slot(S.nodes, cur, 3);
        // the reference's three near-first tests (an empty slot's corner is +inf)
        const bool l_first =
            near_first(r.d, fminf(s0.lox, s1.lox), fminf(s0.loy, s1.loy), fminf(s0.loz, s1.loz),
                       fminf(s2.lox, s3.lox), fminf(s2.loy, s3.loy), fminf(s2.loz, s3.loz));
        const bool ll_first = near_first(r.d, s0.lox, s0.loy, s0.loz, s1.lox, s1.loy, s1.loz);
        const bool rl_first = near_first(r.d, s2.lox, s2.loy, s2.loz, s3.lox, s3.loy, s3.loz);
        if (KIND == BINARY) {
            binary_step(s0, s1);
            binary_step(s2, s3);
        }
        float a0, a1, a2, a3, far;
        auto test = [&](const Slot& s, float& a) {
            return KIND == WIDE ? slab_wide<false>(w, best.t, s, a, far, flat) : slab_slot(w, best.t, s, a, far);
        };
        if (!test(s0, a0)) a0 = MISS;
        if (!test(s1, a1) || KIND == BINARY) a1 = MISS;
        if (!test(s2, a2)) a2 = MISS;
        if (!test(s3, a3) || KIND == BINARY) a3 = MISS;
        int32_t c0 = s0.code, c1 = s1.code, c2 = s2.code, c3 = s3.code;
        // BINARY: slot 0 before slot 1 whatever the (meaningless) inner test says
        swap_if(!ll_first, c0, c1, a0, a1);
        swap_if(!rl_first, c2, c3, a2, a3);
        swap_if(!l_first, c0, c2, a0, a2);
        swap_if(!l_first, c1, c3, a1, a3);
        // the nearest hit goes on, the others are pushed, far to near
        over |= sp > STACK - 3;
        sp = min(sp, STACK - 3);
        const bool h0 = a0 == a0, h1 = a1 == a1, h2 = a2 == a2, h3 = a3 == a3;
        if (h3 & (h0 | h1 | h2)) st[sp++] = make_int2(c3, __float_as_int(a3));
        if (h2 & (h0 | h1)) st[sp++] = make_int2(c2, __float_as_int(a2));
        if (h1 & h0) st[sp++] = make_int2(c1, __float_as_int(a1));
        next = h0 ? c0 : h1 ? c1 : h2 ? c2 : h3 ? c3 : NO_NODE;
        if (next == NO_NODE) pop();
        if (KIND == WIDE && flat) next = NO_NODE;
    };
    for (;;) {
        if (next >= 0) node(next);
        bool ended;
        const bool leaf = leaf_turn<STAY>(group, next, ended);
        if (ended) {
            if (over) atomicOr(status, RT_DEV_OVERFLOW);
            return best;
        }
        if (leaf) {
            leaf_closest<PAIR>(S, r, ~next, best);
            pop();
        }
    }
}

// PARALLEL (closest_hit): for the callers' own rays, which may have any bounds and
// all be parallel to an axis; camera rays and reflections seldom are, and their
// bounds are given.  PARALLEL (any_hit): the shadow rays of a directional light may be
// too.  By levels and WIDE, ordinary rays beside them: trace of 4 M rays over 10k
// triangles 2140 -> 1552 us (1493), shadows of 4 M hits 445 -> 310 (285), 3840 x
// 2160 of a 20k-triangle field under a light straight above 1298 -> 1088 (1007).  A
// third search costs other rays 0.6-1.6 % in the glass, instanced, batched and
// one-path-per-lane kernels: such rays go by levels there.
template <bool STAY, bool PAIR, bool PARALLEL = false>
static __device__ Hit closest_hit(const SceneView& S, const BvhHeader& H, const TRay& r, float tmax,
                                  uint32_t* status) {
    Hit best{-1, tmax, 0.f, 0.f};
    float A;
    if (!slab(r, best.t, H.root_lo.x, H.root_lo.y, H.root_lo.z, H.root_hi.x, H.root_hi.y,
              H.root_hi.z, A))
        return best;
    if (H.root_cnt > 0) {
        leaf_closest(S, r, H.root_ref, H.root_cnt, best);
        return best;
    }
    bool flat = false;
    if (careful_ray(r) || (PARALLEL ? unbounded_ray(r, tmax) : !(tmax < __int_as_float(0x7f800000)))) {
        if (PARALLEL && !binary_ray(r)) {
            best = closest_search<false, false, WIDE>(S, H, r, tmax, status, flat);
            if (!flat) return best;
        }
        return closest_search<false, false, BINARY>(S, H, r, tmax, status, flat);
    }
    return closest_search<STAY, PAIR, PLAIN>(S, H, r, tmax, status, flat);
}

// Whether anything blocks the ray.  tMax does not shrink, so the order of
// the visits does not matter to the answer; of the children that the ray meets
// it enters the one it crosses for longest, the likeliest to hold a blocker: 1-3 %
// of a frame against the last child first, 20 % against the nearest first.
template <bool STAY, bool PAIR, SearchKind KIND>
__device__ __forceinline__ bool any_search(const SceneView& S, const BvhHeader& H, const TRay& r,
                                           float tmax, uint32_t* status, bool& flat) {
    int32_t st[STACK];
    int sp = 0;
    bool over = false;
    const SlabRay w = slab_ray(r);
    const unsigned group = STAY ? __activemask() : 0u;
    int32_t next = H.root_ref;
    bool found = false;
    auto node = [&](int32_t cur) {
        next = NO_NODE;
        auto take = [&](bool hit, int32_t c) {
            if (hit) {
                if (next != NO_NODE) st[sp++] = next;
                next = c;
            }
        };
        over |= sp > STACK - 3;
        sp = min(sp, STACK - 3);
        if (KIND == BINARY) {   // the shadow kernel's own NaN rules
#pragma unroll 1
            for (int k = 0; k < 4; k += 2) {
                Slot a = load_slot(S.nodes, cur, k);
                binary_step(a, load_slot(S.nodes, cur, k + 1));
                take(slab_shadow(r, tmax, a.lox, a.loy, a.loz, a.hix, a.hiy, a.hiz), a.code);
            }
        } else {
            const Slot s0 = load_slot(S.nodes, cur, 0), s1 = load_slot(S.nodes, cur, 1),
                       s2 = load_slot(S.nodes, cur, 2), s3 = load_slot(S.nodes, cur, 3);
            float longest = -1.f;   // of the children met so far: a hit's is >= 0
            auto visit = [&](const Slot& s) {
                float A, B;
                const bool hit = KIND == WIDE ? slab_wide<true>(w, tmax, s, A, B, flat)
                                              : slab_slot(w, tmax, s, A, B);
                const float len = B - A;
                const bool first = hit & (len > longest), push = hit & (longest >= 0.f);
                const int32_t other = first ? next : s.code;
                if (push) st[sp++] = other;
                next = first ? s.code : next;
                longest = first ? len : longest;
            };
            visit(s0);
            visit(s1);
            visit(s2);
            visit(s3);
        }
        if (next == NO_NODE && sp > 0) next = st[--sp];
        if (KIND == WIDE && flat) next = NO_NODE;
    };
    for (;;) {
        if (next >= 0) node(next);
        bool ended;
        const bool leaf = leaf_turn<STAY>(group, next, ended);
        if (ended) {
            if (over) atomicOr(status, RT_DEV_OVERFLOW);
            return found;
        }
        if (leaf) {
            found = leaf_any<PAIR>(S, r, ~next, tmax);
            next = !found && sp > 0 ? st[--sp] : NO_NODE;
        }
    }
}

template <bool STAY, bool PAIR, bool PARALLEL = false>
static __device__ bool any_hit(const SceneView& S, const BvhHeader& H, const TRay& r, float tmax,
                               uint32_t* status) {
    if (!slab_shadow(r, tmax, H.root_lo.x, H.root_lo.y, H.root_lo.z, H.root_hi.x, H.root_hi.y,
                     H.root_hi.z))
        return false;
    if (H.root_cnt > 0) return leaf_any(S, r, H.root_ref, H.root_cnt, tmax);
    bool flat = false;
    if (careful_ray(r)) {
        if (PARALLEL && !binary_ray(r)) {
            const bool found = any_search<false, false, WIDE>(S, H, r, tmax, status, flat);
            if (!flat) return found;
        }
        return any_search<false, false, BINARY>(S, H, r, tmax, status, flat);
    }
    return any_search<STAY, PAIR, PLAIN>(S, H, r, tmax, status, flat);
}

// Hit record of complete_trace_info.
struct HitInfo {
    f3 n, hp;
    uint8_t inverse_n;
};

__device__ __forceinline__ HitInfo complete_hit(const SceneView& S, f3 o, f3 d, const Hit& h) {
    HitInfo hi;
    hi.hp = add(o, muls(d, h.t));
    const uint32_t a = __ldg(&S.idx[3 * (size_t)h.id]), b = __ldg(&S.idx[3 * (size_t)h.id + 1]),
                   c = __ldg(&S.idx[3 * (size_t)h.id + 2]);
    const f3 n0 = normalize(ld3(__ldg(&S.nrm[a])));
    const f3 n1 = normalize(ld3(__ldg(&S.nrm[b])));
    const f3 n2 = normalize(ld3(__ldg(&S.nrm[c])));
    const float w = 1.0f - (h.u + h.v);
    f3 n = normalize(add(add(muls(n0, w), muls(n2, h.v)), muls(n1, h.u)));
    if (dot(n, d) > 0.0f) {
        hi.inverse_n = 1;
        n = neg(n);
    } else {
        hi.inverse_n = 0;
    }
    hi.n = n;
    return hi;
}

// Direction of the shadow ray of shadow_trace_single to a light (shadow-trace-
// bvh.cl:375-418); point lights as spot lights without a cone.  False: the
// light does not reach hp, whatever lies in between.
__device__ __forceinline__ bool shadow_dir(const rt_light& L, f3 hp, f3& dir) {
    if (L.type == RT_DIR_L) {
        dir = neg(mk3(L.dir[0], L.dir[1], L.dir[2]));
    } else if (L.type == RT_SPOT_L) {
        dir = normalize(sub(mk3(L.pos[0], L.pos[1], L.pos[2]), hp));
        if (dot(neg(dir), mk3(L.dir[0], L.dir[1], L.dir[2])) < L.angle) return false;
    } else if (L.type == RT_POINT_L) {
        dir = normalize(sub(mk3(L.pos[0], L.pos[1], L.pos[2]), hp));
    } else {
        return false;
    }
    return true;
}

template <bool STAY = false, bool PAIR = false, bool PARALLEL = false>
__device__ __forceinline__ bool occluded(const SceneView& S, const BvhHeader& H, const rt_light& L,
                                         f3 hp, uint32_t* status) {
    f3 dir;
    if (!shadow_dir(L, hp, dir)) return true;
    const f3 inv = mk3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
    const TRay r = make_tray(hp, dir, inv, 0.01f);
    return any_hit<STAY, PAIR, PARALLEL>(S, H, r, 1e37f, status);
}

// Light direction (from the light toward the hit) and colour at a hit, as
// shade_sample computes them (ray-shader.cl:116-333; point lights without a
// cone).
__device__ __forceinline__ void light_at(const rt_light& L, f3 hp, f3& Ld, f3& rgb) {
    rgb = mk3(L.color[0], L.color[1], L.color[2]);
    float LD;
    if (L.type == RT_DIR_L) {
        Ld = mk3(L.dir[0], L.dir[1], L.dir[2]);
        LD = 1.0f;
    } else if (L.type == RT_SPOT_L) {
        Ld = normalize(sub(hp, mk3(L.pos[0], L.pos[1], L.pos[2])));
        LD = dot(Ld, mk3(L.dir[0], L.dir[1], L.dir[2])) - L.angle;
        LD /= 1.0f - L.angle;
        LD = clamp01(LD);
    } else {
        Ld = normalize(sub(hp, mk3(L.pos[0], L.pos[1], L.pos[2])));
        LD = 1.0f;
    }
    rgb = muls(rgb, LD);
}

// The two terms shade_sample adds for light L when its shadow ray is not
// blocked (ray-shader.cl:312-330): diffuse rgb * diffuse * cosL and specular
// rgb * spec, with cosL = clamp(dot(n, -Ld))^2 and spec = clamp(dot(r,
// -Ld))^8 * cosL * shininess, r the incoming direction d reflected about n.
__device__ __forceinline__ void light_terms(const rt_light& L, const rt_material& mat, f3 hp, f3 n,
                                            f3 d, f3& dterm, f3& sterm) {
    f3 Ld, rgb;
    light_at(L, hp, Ld, rgb);
    const f3 diffuse = mk3(mat.diffuse[0], mat.diffuse[1], mat.diffuse[2]);
    const float dn = dot(d, n);
    const f3 rr = sub(d, muls(muls(n, 2.0f), dn));
    float cosL = clamp01(dot(n, neg(Ld)));
    cosL = cosL * cosL;
    float spec = clamp01(dot(rr, neg(Ld)));
    spec = spec * spec;
    spec = spec * spec;
    spec = spec * spec;
    spec *= cosL * mat.shininess;
    dterm = muls(mul(rgb, diffuse), cosL);
    sterm = muls(rgb, spec);
}

// True when light L adds nothing to the hit's colour whether or not its
// shadow ray is blocked: both terms of light_terms are zero (a light behind
// the surface, cosL = 0; a surface with no diffuse colour and no shininess,
// as the mirrors here; a black light).  Adding a zero term changes the sum
// at most in the sign of a zero, which floor(f * 1e6) to an integer
// removes, so skipping the shadow ray gives the same image; a NaN or
// infinite term is never skipped.  Only the fused renders skip; the
// stage-wise shadow pass reports every ray's result.
__device__ __forceinline__ bool light_vanishes(const rt_light& L, const rt_material& mat, f3 hp,
                                               f3 n, f3 d) {
    f3 dt, st;
    light_terms(L, mat, hp, n, d, dt, st);
    return dt.x == 0.0f && dt.y == 0.0f && dt.z == 0.0f && st.x == 0.0f && st.y == 0.0f &&
           st.z == 0.0f;
}

// The shadow tasks of a warp's nh hits (nh <= 32) and nl lights (nl <=
// RT_MAX_LIGHTS), in light-major order so that neighbouring lanes trace
// toward one light from neighbouring hits.  need(k, l) settles a task
// without a ray when it returns false (light_vanishes); the tasks that need
// a ray are listed densely in `list` (hit | light << 5, 32 * RT_MAX_LIGHTS
// bytes of the warp's shared memory) and trace(k, l) runs them 32 at a
// time, so a round of the warp traces 32 rays whatever was settled (against
// each lane taking the tasks of its own index: 1.5 % faster on the
// mid-scale frame, 4 % on the stress pose, equal on the small soup).  All 32
// lanes call it.
static_assert(RT_MAX_LIGHTS <= 8, "task list entries hold the light in 3 bits");
template <class Need, class Trace>
__device__ __forceinline__ void shadow_tasks(int nh, int nl, uint8_t* list, Need need, Trace trace) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int ntask = nh * nl;
    int nt = 0;
    for (int t0 = 0; t0 < ntask; t0 += 32) {
        const int t = t0 + lane;
        bool nd = false;
        int k = 0, l = 0;
        if (t < ntask) {
            l = t / nh;
            k = t - l * nh;
            nd = need(k, l);
        }
        const unsigned bm = __ballot_sync(0xffffffffu, nd);
        if (nd) list[nt + __popc(bm & lt)] = (uint8_t)(k | (l << 5));
        nt += __popc(bm);
    }
    __syncwarp();
    for (int i = lane; i < nt; i += 32) {
        const int e = list[i];
        trace(e & 31, e >> 5);
    }
}

// Local Whitted term of shade_sample, as the fixed-point increments that
// to_color_int + image[pixel] += produce (ray-shader.cl:101-109, 312-330).
__device__ __forceinline__ uint3 shade_hit(const rt_lights& Ls, const rt_material& mat, f3 hp, f3 n,
                                           f3 d, float contribution, uint32_t shadow_mask) {
    const f3 diffuse = mk3(mat.diffuse[0], mat.diffuse[1], mat.diffuse[2]);
    f3 val = mul(mk3(Ls.ambient[0], Ls.ambient[1], Ls.ambient[2]), diffuse);
    for (int l = 0; l < Ls.count; ++l) {
        if (!((shadow_mask >> l) & 1u)) {
            f3 dt, st;
            light_terms(Ls.light[l], mat, hp, n, d, dt, st);
            val = add(val, dt);
            val = add(val, st);
        }
    }
    val = muls(val, 1.0f - mat.reflectiveness);
    f3 f = muls(val, contribution);
    f = mk3(clamp01(f.x), clamp01(f.y), clamp01(f.z));
    return make_uint3((uint32_t)floorf(f.x * 1e6f), (uint32_t)floorf(f.y * 1e6f),
                      (uint32_t)floorf(f.z * 1e6f));
}

// Reflection ray (secondary-ray-generator.cl:258-270).
__device__ __forceinline__ void reflect_ray(f3 d_in, f3 n_in, f3& dir) {
    f3 d = neg(normalize(d_in));
    const f3 n = normalize(n_in);
    d = neg(d);
    dir = normalize(sub(d, muls(muls(n, 2.0f), dot(d, n))));
}

// pow(x, 5) of the Schlick term: the product in double precision, rounded to
// float once (the oracle evaluates it the same way; OpenCL allows pow 16 ulp).
__device__ __forceinline__ float pow5(float x) {
    const double p = (double)x;
    return (float)((((p * p) * p) * p) * p);
}

// Refraction branch of generate_secondary_rays_disc
// (secondary-ray-generator.cl:220-256): whether the refracted ray exists
// (k > 0), Schlick's factor R and the refracted direction.
__device__ __forceinline__ bool refract_ray(f3 d_in, f3 n_in, bool inverse_n, float ior, float& R,
                                            f3& dir) {
    const f3 d = neg(normalize(d_in));
    const f3 n = normalize(n_in);
    const float etai = inverse_n ? ior : 1.0f, etat = inverse_n ? 1.0f : ior;
    const float cosi = dot(d, n);
    const float rel_eta = etai / etat;
    const float w = rel_eta * cosi;
    float k = 1.0f + (w - rel_eta) * (w + rel_eta);
    if (!(k > 0.0f)) return false;
    float R0 = (etat - 1.0f) / (etat + 1.0f);
    R0 *= R0;
    R = R0 + (1.0f - R0) * pow5(1.0f - cosi);
    k = sqrtf(k);
    dir = normalize(sub(muls(n, w - k), muls(d, etai)));
    return true;
}

// Pixel of global id gid in the quad_size block order of generate_primary_rays.
__device__ __forceinline__ void pixel_of(int gid, int w, int h, int q, int& x, int& y) {
    const int pixels = w * h;
    const int i = gid % pixels;
    const int ba = q * q, xb = w / q, yb = h / q;
    const int block_rays = xb * yb * ba;
    const int right_rays = (w - xb * q) * h;
    if (i < block_rays) {
        const int block = i / ba, bp = i % ba;
        x = (block % xb) * q + bp % q;
        y = (block / xb) * q + bp / q;
    } else if (i < block_rays + right_rays) {
        const int sx = xb * q, slab_w = w - sx, ri = i - block_rays;
        x = sx + ri % slab_w;
        y = ri / slab_w;
    } else {
        const int sy = yb * q, slab_h = h - sy, ti = i - (block_rays + right_rays);
        x = ti / slab_h;
        y = sy + ti % slab_h;
    }
}

// Work order of the fused kernel: inside each full 32x32 block, the 32 pixels
// a warp takes form an 8x4 tile instead of one 32-pixel row (rays closer
// together).  Only the assignment of pixels to lanes changes; every pixel is
// still rendered exactly once.
__device__ __forceinline__ int warp_tile_order(int gid, int w, int h) {
    const int xb = w / 32, yb = h / 32;
    const int block_rays = xb * yb * 1024;
    if (gid >= block_rays) return gid;
    const int block = gid >> 10, bp = gid & 1023;
    const int t = bp >> 5, r = bp & 31;
    const int px = (t & 3) * 8 + (r & 7), py = (t >> 2) * 4 + (r >> 3);
    return (block << 10) + py * 32 + px;
}

__device__ __forceinline__ f3 primary_dir(const rt_camera& cam, int x, int y, int w, int h,
                                          float ox, float oy) {
    const float xn = (0.5f + (float)x + ox) / (float)w;
    const float yn = (0.5f + (float)y + oy) / (float)h;
    const float a = xn * 2.0f - 1.0f, b = yn * 2.0f - 1.0f;
    f3 d = add(add(mk3(cam.dir[0], cam.dir[1], cam.dir[2]),
                   muls(mk3(cam.right[0], cam.right[1], cam.right[2]), a)),
               muls(mk3(cam.up[0], cam.up[1], cam.up[2]), b));
    return normalize(d);
}

__device__ __forceinline__ uint8_t to_unorm8(uint32_t v, float inv1e6) {
    const float f = (float)v * inv1e6;
    return (uint8_t)__float2uint_rn(clamp01(f) * 255.0f);
}

__device__ __forceinline__ uchar4 rgba8_of(uint3 sum, float inv1e6) {
    return make_uchar4(to_unorm8(sum.x, inv1e6), to_unorm8(sum.y, inv1e6),
                       to_unorm8(sum.z, inv1e6), 255);
}


// Result of one pixel's Whitted path.
struct PixelResult {
    uint32_t r, g, b;
    uint32_t secondary, shadow, hits;
};

// The whole path of one pixel (Renderer::render_to_framebuffer's tile and
// bounce loops restricted to the pixel): primary ray, closest hit, one
// shadow ray per light, local shading, reflection ray while the material
// reflects and the bounce budget lasts.  Integer accumulation of the
// fixed-point contributions makes the sum independent of evaluation order.
// Pending secondary ray of a pixel's ray tree (refraction branches it).
struct PendingRay {
    f3 o, d;
    float contribution;
    int bounce;
};
constexpr int REFR_STACK = 16;   // pending rays per lane: one per level of the tree

// One pixel's Whitted rays: the primary ray and, up to max_bounces, the
// secondary rays of generate_secondary_rays_disc (a reflected ray with
// contribution * reflectiveness * R, and with REFR a refracted one with
// contribution * reflectiveness * (1 - R), R = Schlick's factor, 1 without
// refraction), each traced, shadowed and shaded as the reference's wavefront
// does.  The sums are integers, so the depth-first order of this tree walk
// gives the wavefront's image.
template <bool REFR = false>
__device__ __forceinline__ PixelResult render_pixel(const SceneView& S, const BvhHeader& H,
                                                    const rt_lights& L, const rt_camera& cam,
                                                    int x, int y, int w, int h, int max_bounces,
                                                    uint32_t* status) {
    PixelResult res = {0, 0, 0, 0, 0, 0};
    f3 o = mk3(cam.pos[0], cam.pos[1], cam.pos[2]);
    f3 d = primary_dir(cam, x, y, w, h, 0.0f, 0.0f);
    float tmin = 0.0f, tmax = 1e36f, contribution = 1.0f;
    PendingRay stack[REFR ? REFR_STACK : 1];
    int sp = 0;
    for (int bounce = 0;;) {
        bool next = false;
        const f3 inv = mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        const TRay r = make_tray(o, d, inv, tmin);
        const Hit hit = closest_hit<true, false>(S, H, r, tmax, status);
        if (hit.id >= 0) {
            ++res.hits;
            const HitInfo hi = complete_hit(S, o, d, hit);
            const rt_material mat = S.mats[__ldg(&S.map[hit.id])];
            uint32_t mask = 0;
            for (int l = 0; l < L.count; ++l)
                if (!light_vanishes(L.light[l], mat, hi.hp, hi.n, d) &&
                    occluded<true, false>(S, H, L.light[l], hi.hp, status))
                    mask |= 1u << l;
            res.shadow += (uint32_t)L.count;
            const uint3 c = shade_hit(L, mat, hi.hp, hi.n, d, contribution, mask);
            res.r += c.x;
            res.g += c.y;
            res.b += c.z;
            if (bounce < max_bounces) {
                float R = 1.0f;
                if (REFR && mat.refractive_index > 0.0f) {
                    f3 td;
                    if (refract_ray(d, hi.n, hi.inverse_n != 0, mat.refractive_index, R, td)) {
                        if (sp < REFR_STACK) {
                            stack[sp].o = hi.hp;
                            stack[sp].d = td;
                            stack[sp].contribution = contribution * mat.reflectiveness * (1.0f - R);
                            stack[sp].bounce = bounce + 1;
                            ++sp;
                        } else {
                            atomicOr(status, RT_DEV_OVERFLOW);
                        }
                    }
                }
                if (mat.reflectiveness > 0.0f) {
                    f3 nd;
                    reflect_ray(d, hi.n, nd);
                    contribution = contribution * mat.reflectiveness * R;
                    o = hi.hp;
                    d = nd;
                    tmin = 0.0001f;
                    tmax = 1e37f;
                    ++bounce;
                    ++res.secondary;
                    next = true;
                }
            }
        }
        if (next) continue;
        if (!REFR || sp == 0) break;
        --sp;   // the next refracted ray set aside
        o = stack[sp].o;
        d = stack[sp].d;
        contribution = stack[sp].contribution;
        bounce = stack[sp].bounce;
        tmin = 0.0001f;
        tmax = 1e37f;
        ++res.secondary;
    }
    return res;
}

}  // namespace rt
