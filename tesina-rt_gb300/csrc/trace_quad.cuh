// trace_quad.cuh — one ray per four lanes, for launches with few rays.
//
// A ray's search is a chain of steps, and with too few rays to fill the SMs a
// launch takes as long as its longest chain.  Four lanes shorten the steps:
// lane q tests slot q of the record (one 128-byte line per ray) and triangle q
// of a leaf, votes and shuffles replace the serial tests, and eight rays
// instead of 32 share a warp, so that fewer of its turns are another ray's.
// The rays visit the same leaves in the same order as in trace_dev.cuh, with
// the same arithmetic.  Trace and shadow stage of a 10k-triangle soup, without
// and with: 21k secondary rays 93 + 63 -> 61 + 43 us, 2k 100 + 66 -> 46 + 39.
// A warp's leaves are tested in the turn that reaches them: to wait for more, as
// leaf_turn does, loses 1 % of a small frame.
// (Prefetching the records and triangles of the children hit loses 3 %: it is
// the instructions' latency, not the memory's.)
#pragma once
#include "trace_dev.cuh"

namespace rt {

// Stack of a ray, in shared memory: code and entry distance.
struct QuadStack {
    int2 e[STACK];
};

// The four bits of this lane's ray in a warp's ballot.
__device__ __forceinline__ unsigned quad_ballot(bool p) {
    return __ballot_sync(0xffffffffu, p) >> (threadIdx.x & 28) & 15u;
}
__device__ __forceinline__ float quad_xor(float v, int m) {
    return __shfl_xor_sync(0xffffffffu, v, m);
}

// Takes entries, the last pushed first, until one has its distance within tmax.
__device__ __forceinline__ void quad_pop(bool want, const int2* st, int& sp, float tmax,
                                         int32_t& next) {
    const int q = threadIdx.x & 3, base = threadIdx.x & 28;
    want = want && sp > 0;
    while (__any_sync(0xffffffffu, want)) {
        int2 e = make_int2(NO_NODE, 0);
        const bool have = want && q < sp;
        if (have) e = st[sp - 1 - q];
        const unsigned ok = quad_ballot(have && __int_as_float(e.y) <= tmax);
        const int k = ok ? __ffs(ok) - 1 : 0;
        const int32_t c = __shfl_sync(0xffffffffu, e.x, base + k);
        if (want) {
            if (ok) next = c;
            sp = ok ? sp - 1 - k : max(sp - 4, 0);
            want = !ok && sp > 0;
        }
    }
}

// Triangle i + q of the leaf for lane q; `valid` if the leaf has it, `full` if
// the leaf goes on after all four.
__device__ __forceinline__ bool quad_triangle(const SceneView& S, const TRay& r, bool on, int32_t i,
                                              float& t, float& u, float& v, bool& full) {
    const int q = threadIdx.x & 3;
    bool more = false, hit = false;
    if (on) {
        const TriRec T = load_tri(S.tris, i + q);
        more = T.v0.w != 0.0f;
        hit = mt(T, r.o, r.d, t, u, v);
    }
    const unsigned m = quad_ballot(more), below = (1u << q) - 1u;
    full = m == 15u;
    return hit && (m & below) == below;
}

// closest_search by the four lanes of the ray; all lanes of the warp call
// together, those without a ray with `live` false.
__device__ __forceinline__ Hit closest_quad(const SceneView& S, int32_t root, const TRay& r,
                                            float tmax, bool live, int2* st, uint32_t* status) {
    const int q = threadIdx.x & 3, base = threadIdx.x & 28;
    const SlabRay w = slab_ray(r);
    Hit best{-1, tmax, 0.f, 0.f};
    int sp = 0;
    bool over = false;
    int32_t next = live ? root : NO_NODE;
    for (;;) {
        if (__any_sync(0xffffffffu, next >= 0)) {
            const bool on = next >= 0;
            Slot s{};
            if (on) s = load_slot(S.nodes, next, q);
            // the pair's order, then the pairs' (see closest_search)
            const float ox = quad_xor(s.lox, 1), oy = quad_xor(s.loy, 1), oz = quad_xor(s.loz, 1);
            const bool odd = q & 1, hi = q & 2;
            const float ax = odd ? ox : s.lox, ay = odd ? oy : s.loy, az = odd ? oz : s.loz;
            const float bx = odd ? s.lox : ox, by = odd ? s.loy : oy, bz = odd ? s.loz : oz;
            const bool first = near_first(r.d, ax, ay, az, bx, by, bz);
            const float mx = fminf(ax, bx), my = fminf(ay, by), mz = fminf(az, bz);
            const float px = quad_xor(mx, 2), py = quad_xor(my, 2), pz = quad_xor(mz, 2);
            const bool l_first = near_first(r.d, hi ? px : mx, hi ? py : my, hi ? pz : mz,
                                            hi ? mx : px, hi ? my : py, hi ? mz : pz);
            float A, far;
            const bool hit = slab_slot(w, best.t, s, A, far) && on;
            const unsigned hm = quad_ballot(hit);
            const bool second = odd == first, second_pair = hi == l_first;
            const int mate = hm >> (q ^ 1) & 1, others = __popc(hm & (hi ? 3u : 12u));
            const int before = (second_pair ? others : 0) + (second ? mate : 0);
            const int n = __popc(hm), after = n - 1 - before;
            over |= on && sp > STACK - 3;
            sp = min(sp, STACK - 3);
            if (hit && before > 0) st[sp + after] = make_int2(s.code, __float_as_int(A));
            const unsigned nearest = quad_ballot(hit && before == 0);
            const int32_t c = __shfl_sync(0xffffffffu, s.code, base + (nearest ? __ffs(nearest) - 1 : 0));
            if (on) {
                next = nearest ? c : NO_NODE;
                sp += max(n - 1, 0);
            }
            __syncwarp();
            quad_pop(on && next == NO_NODE, st, sp, best.t, next);
        }
        if (__any_sync(0xffffffffu, next < 0 && next != NO_NODE)) {
            const bool leaf = next < 0 && next != NO_NODE;
            bool on = leaf;
            int32_t i = ~next;
            do {
                float t = 0.f, u = 0.f, v = 0.f;
                bool full;
                const bool h = quad_triangle(S, r, on, i, t, u, v, full) && t <= best.t && t >= r.tmin;
                if (__any_sync(0xffffffffu, h)) {
                    // of equal distances the later one wins
                    float m = h ? t : __int_as_float(0x7f800000);
                    m = fminf(m, quad_xor(m, 1));
                    m = fminf(m, quad_xor(m, 2));
                    const unsigned win = quad_ballot(h && t == m);
                    const int k = base + (win ? 31 - __clz(win) : 0);
                    const float wt = __shfl_sync(0xffffffffu, t, k), wu = __shfl_sync(0xffffffffu, u, k),
                                wv = __shfl_sync(0xffffffffu, v, k);
                    if (win) best = Hit{i + (k & 3), wt, wu, wv};
                }
                on = on && full;
                i += 4;
            } while (__any_sync(0xffffffffu, on));
            if (leaf) next = NO_NODE;
            quad_pop(leaf, st, sp, best.t, next);
        } else if (!__any_sync(0xffffffffu, next >= 0)) {
            if (over) atomicOr(status, RT_DEV_OVERFLOW);
            return best;
        }
    }
}

__device__ __forceinline__ bool any_quad(const SceneView& S, int32_t root, const TRay& r, float tmax,
                                         bool live, int2* st, uint32_t* status) {
    const int q = threadIdx.x & 3, base = threadIdx.x & 28;
    const SlabRay w = slab_ray(r);
    int sp = 0;
    bool over = false, found = false;
    int32_t next = live ? root : NO_NODE;
    for (;;) {
        if (__any_sync(0xffffffffu, next >= 0)) {
            const bool on = next >= 0;
            Slot s{};
            if (on) s = load_slot(S.nodes, next, q);
            float A, B;
            const bool hit = slab_slot(w, tmax, s, A, B) && on;
            const float len = hit ? B - A : -1.f;
            float m = fmaxf(len, quad_xor(len, 1));
            m = fmaxf(m, quad_xor(m, 2));
            const unsigned hm = quad_ballot(hit), lm = quad_ballot(hit && len == m);
            const int k = lm ? __ffs(lm) - 1 : 0;
            const unsigned rest = hm & ~(1u << k);
            over |= on && sp > STACK - 3;
            sp = min(sp, STACK - 3);
            if (rest >> q & 1) st[sp + __popc(rest & ((1u << q) - 1u))] = make_int2(s.code, 0);
            const int32_t c = __shfl_sync(0xffffffffu, s.code, base + k);
            if (on) {
                next = hm ? c : NO_NODE;
                sp += __popc(rest);
            }
            __syncwarp();
            if (on && next == NO_NODE && sp > 0) next = st[--sp].x;
        }
        if (__any_sync(0xffffffffu, next < 0 && next != NO_NODE)) {
            const bool leaf = next < 0 && next != NO_NODE;
            bool on = leaf;
            int32_t i = ~next;
            do {
                float t = 0.f, u, v;
                bool full;
                const bool h = quad_triangle(S, r, on, i, t, u, v, full) && t < tmax && t > r.tmin;
                if (quad_ballot(h)) {
                    found = true;
                    on = false;
                }
                on = on && full;
                i += 4;
            } while (__any_sync(0xffffffffu, on));
            if (leaf) next = !found && sp > 0 ? st[--sp].x : NO_NODE;
        } else if (!__any_sync(0xffffffffu, next >= 0)) {
            if (over) atomicOr(status, RT_DEV_OVERFLOW);
            return found;
        }
    }
}

// closest_hit and any_hit by the four lanes of the ray, with `live` as above.
// What the search by four does not take, each lane does by itself.
__device__ __forceinline__ Hit closest_hit_quad(const SceneView& S, const BvhHeader& H, const TRay& r,
                                                float tmax, bool live, int2* st, uint32_t* status) {
    Hit best{-1, tmax, 0.f, 0.f};
    float A;
    live = live && slab(r, tmax, H.root_lo.x, H.root_lo.y, H.root_lo.z, H.root_hi.x, H.root_hi.y,
                        H.root_hi.z, A);
    const bool careful = careful_ray(r) || unbounded_ray(r, tmax);
    bool flat = false;
    if (live && H.root_cnt > 0)
        leaf_closest(S, r, H.root_ref, H.root_cnt, best);
    else if (live && careful)
        best = closest_search<false, false, BINARY>(S, H, r, tmax, status, flat);
    live = live && H.root_cnt <= 0 && !careful;
    __syncwarp();
    const Hit h = closest_quad(S, H.root_ref, r, tmax, live, st, status);
    return live ? h : best;
}

__device__ __forceinline__ bool any_hit_quad(const SceneView& S, const BvhHeader& H, const TRay& r,
                                             float tmax, bool live, int2* st, uint32_t* status) {
    bool found = false;
    live = live && slab_shadow(r, tmax, H.root_lo.x, H.root_lo.y, H.root_lo.z, H.root_hi.x,
                               H.root_hi.y, H.root_hi.z);
    const bool careful = careful_ray(r);
    bool flat = false;
    if (live && H.root_cnt > 0)
        found = leaf_any(S, r, H.root_ref, H.root_cnt, tmax);
    else if (live && careful)
        found = any_search<false, false, BINARY>(S, H, r, tmax, status, flat);
    live = live && H.root_cnt <= 0 && !careful;
    __syncwarp();
    const bool f = any_quad(S, H.root_ref, r, tmax, live, st, status);
    return live ? f : found;
}

}  // namespace rt
