// rzk_traverse.cuh - BVH traversal on the packed layout (device functions).
//
// Node slot s = BFS index + 1 holds two float4: {bmin.xyz, a}, {bmax.xyz, b}.  For an
// inner node a is its left child (the right child is a + 1, so both children are one
// contiguous, 64-byte-aligned 64-byte record); for a leaf a = -1 - sorted triangle slot.
// The stack holds these `a` codes, so popping an inner node costs a single 64-byte load
// that yields both child boxes and both children's own codes.
//
// Closest hit gives the reference's answer (aggregate_bvh.cc:402-448: pop, leaf -> triangle
// test that shrinks tmax, inner -> test left box then right box with the current tmax, push the
// ones that pass, right popped first) in one of two ways: a nearer-child-first walk of the
// closest-hit tree wherever that provably finds the same triangle, else the reference's own
// visit order on the reference tree; see closest_hit below.  Any-hit
// (aggregate_bvh.cc:452-478) returns whether any reachable triangle passes; its answer
// does not depend on visit order, so leaf children are tested as soon as their box
// passes instead of being pushed.  The loops go straight on to the entry that would be popped
// next instead of pushing and popping it.  All keep the reference's 64-entry stack, which drops
// pushes when full (holding one entry fewer per level than the reference's, it fills
// later); a drop sets ERR_STACK in the scene's error word.
#pragma once

#include "rzk_internal.cuh"

namespace rzk {

// Per-thread stack: STRIDE = 1 for a private array, STRIDE = block size for a stack
// interleaved in shared memory (entry k of thread t at [k * STRIDE + t]).
template <int STRIDE>
struct Stack {
    int *base;
    int top, cap;
    __device__ __forceinline__ void init(int *b, int entries = STACK_CAP) { base = b; top = -1; cap = entries; }
    __device__ __forceinline__ bool empty() const { return top < 0; }
    __device__ __forceinline__ int pop() { return base[(top--) * STRIDE]; }
    __device__ __forceinline__ bool push(int v) {
        if (top < cap - 1) { base[(++top) * STRIDE] = v; return true; }
        return false;
    }
};

struct TraceStats {
    uint32_t inner, leaf;
    __device__ __forceinline__ void reset() { inner = 0; leaf = 0; }
};

__device__ __forceinline__ void load_tri(const GatherScene &s, int slot, float4 &a, float4 &b, float4 &c) {
    const float4 *p = s.tri_isect + 3 * slot;
    a = __ldg(p); b = __ldg(p + 1); c = __ldg(p + 2);
}

// A pair of sibling nodes: two 32-byte loads (the record is 64-byte aligned).
__device__ __forceinline__ void load_node(const float4 *p, float4 &a, float4 &b) {
    uint64_t q[4];
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(q[0]), "=l"(q[1]), "=l"(q[2]), "=l"(q[3]) : "l"(p));
    auto lo = [](uint64_t x) { return __uint_as_float((uint32_t)x); };
    auto hi = [](uint64_t x) { return __uint_as_float((uint32_t)(x >> 32)); };
    a = make_float4(lo(q[0]), hi(q[0]), lo(q[1]), hi(q[1]));
    b = make_float4(lo(q[2]), hi(q[2]), lo(q[3]), hi(q[3]));
}
__device__ __forceinline__ void load_pair(const float4 *p, float4 &l0, float4 &l1, float4 &r0, float4 &r1) {
    load_node(p, l0, l1);
    load_node(p + 2, r0, r1);
}

// TRAV: walk the any-hit tree (DevScene::trav) instead of the reference tree; the answer is
// the same (see rzk_sah.cu), only the visit order differs.  FASTBOX: the ray was made by
// make_ray, so box_hit_fast applies (1,000,003 segments on 300k triangles 571 -> 517 us, B200);
// a caller's own ray may hold any reciprocals and takes box_hit.
template <int STRIDE, bool STATS, bool TRAV = false, bool FASTBOX = true, class Scene>   // GatherScene: TRAV only
__device__ __forceinline__ bool any_hit(const Scene &s, const Ray &r, float tmin, float tmax,
                                        Stack<STRIDE> &stk, TraceStats *ts = nullptr) {
    if (s.n_nodes == 0) return false;
    const float4 *tree;
    if constexpr (TRAV) tree = s.trav;
    else tree = s.nodes;
    float4 lo = __ldg(tree + 2), hi = __ldg(tree + 3);
    if (!box_hit(lo, hi, r, tmin, tmax)) return false;
    int a = __float_as_int(lo.w);
    float4 ta, tb, tc;
    if (a < 0) {
        if (STATS) ts->leaf++;
        load_tri(s, -1 - a, ta, tb, tc);
        return tri_hit<false>(ta, tb, tc, r, tmin, tmax, nullptr, nullptr, nullptr);
    }
    // the loop continues into the child it would pop next (the right one where both are
    // entered) and pushes only the other: the visit order of pushing both, without a stack
    // store and load on each step's dependency chain
    stk.top = -1;
    int c = a;
    bool overflow = false;
    for (;;) {
        if (STATS) ts->inner++;
        const float4 *p = tree + 2 * (c + 1);
        float4 l0, l1, r0, r1;
        load_pair(p, l0, l1, r0, r1);
        float tl, tr;
        bool hl = FASTBOX ? box_hit_fast(l0, l1, r, tmin, tmax, tl) : box_hit(l0, l1, r, tmin, tmax);
        bool hr = FASTBOX ? box_hit_fast(r0, r1, r, tmin, tmax, tr) : box_hit(r0, r1, r, tmin, tmax);
        int al = __float_as_int(l0.w), ar = __float_as_int(r0.w);
        if (hl && al < 0) {
            if (STATS) ts->leaf++;
            load_tri(s, -1 - al, ta, tb, tc);
            if (tri_hit<false>(ta, tb, tc, r, tmin, tmax, nullptr, nullptr, nullptr)) return true;
        }
        if (hr && ar < 0) {
            if (STATS) ts->leaf++;
            load_tri(s, -1 - ar, ta, tb, tc);
            if (tri_hit<false>(ta, tb, tc, r, tmin, tmax, nullptr, nullptr, nullptr)) return true;
        }
        const bool gl = hl && al >= 0, gr = hr && ar >= 0;
        if (gr) {
            if (gl && !stk.push(al)) overflow = true;
            c = ar;
        } else if (gl) {
            c = al;
        } else {
            if (stk.empty()) break;
            c = stk.pop();
        }
    }
    if (overflow && s.err) atomicOr(s.err, ERR_STACK);
    return false;
}

// any_hit on the any-hit tree (TRAV, FASTBOX), one pair of nodes per step.
template <int STRIDE>
struct AnyHitWalk {
    Stack<STRIDE> stk;
    Ray r;
    float tmin, tmax;
    int c;
    bool hit, over;
    __device__ __forceinline__ void start(const DevScene &s, const Ray &ray, float t0, float t1) {
        r = ray;
        tmin = t0;
        tmax = t1;
        hit = false;
        over = s.n_nodes == 0;
        stk.top = -1;
        c = 0;
        if (over) return;
        const float4 lo = __ldg(s.trav + 2), hi = __ldg(s.trav + 3);
        over = !box_hit(lo, hi, r, tmin, tmax);
        c = __float_as_int(lo.w);
        if (!over && c < 0) {
            hit = tri(s, c);
            over = true;
        }
    }
    __device__ __forceinline__ bool tri(const DevScene &s, int code) const {
        float4 ta, tb, tc;
        load_tri(s, -1 - code, ta, tb, tc);
        return tri_hit<false>(ta, tb, tc, r, tmin, tmax, nullptr, nullptr, nullptr);
    }
    __device__ __forceinline__ bool step(const DevScene &s) {   // true when the walk is over
        if (over) return true;
        float4 l0, l1, r0, r1;
        load_pair(s.trav + 2 * (c + 1), l0, l1, r0, r1);
        float tl, tr;
        const bool hl = box_hit_fast(l0, l1, r, tmin, tmax, tl);
        const bool hr = box_hit_fast(r0, r1, r, tmin, tmax, tr);
        const int al = __float_as_int(l0.w), ar = __float_as_int(r0.w);
        if (hl && al < 0) hit = tri(s, al);
        if (!hit && hr && ar < 0) hit = tri(s, ar);
        if (hit) return true;
        const bool gl = hl && al >= 0, gr = hr && ar >= 0;
        if (gr) {
            if (gl && !stk.push(al) && s.err) atomicOr(s.err, ERR_STACK);
            c = ar;
        } else if (gl) {
            c = al;
        } else {
            if (stk.empty()) return true;
            c = stk.pop();
        }
        return false;
    }
};

struct ClosestHit {
    int slot;   // sorted triangle slot, -1: none
    float t, beta, gamma;
};

// The reference's query: its tree, its visit order, its box test, its 64-entry stack (`stack` as
// Stack::base).
template <int STRIDE>
__device__ __forceinline__ ClosestHit closest_in_order(const float4 *nodes, const float4 *tri_isect, uint32_t *err,
                                                       const Ray &r, float tmin, float tmax, int *stack) {
    ClosestHit h{-1, RAY_TMAX, 0.0f, 0.0f};
    float4 lo = __ldg(nodes + 2), hi = __ldg(nodes + 3);
    if (!box_hit(lo, hi, r, tmin, tmax)) return h;
    bool overflow = false;
    // the loop continues into the entry it would pop next (the right child where both boxes
    // pass, each tested with the tmax of that moment) and pushes only the other, so the nodes
    // are visited in the reference's order
    Stack<STRIDE> stk;
    stk.init(stack);
    int c = __float_as_int(lo.w);
    for (;;) {
        if (c < 0) {
            const float4 *p = tri_isect + 3 * (-1 - c);
            float t, b, g;
            if (tri_hit<true>(__ldg(p), __ldg(p + 1), __ldg(p + 2), r, tmin, tmax, &t, &b, &g)) {
                tmax = t;
                h.t = t; h.beta = b; h.gamma = g;
                h.slot = -1 - c;
            }
            if (stk.empty()) break;
            c = stk.pop();
            continue;
        }
        const float4 *p = nodes + 2 * (c + 1);
        const float4 l0 = __ldg(p), l1 = __ldg(p + 1), r0 = __ldg(p + 2), r1 = __ldg(p + 3);
        const bool hl = box_hit(l0, l1, r, tmin, tmax);
        const bool hr = box_hit(r0, r1, r, tmin, tmax);
        if (hr) {
            if (hl && !stk.push(__float_as_int(l0.w))) overflow = true;
            c = __float_as_int(r0.w);
        } else if (hl) {
            c = __float_as_int(l0.w);
        } else {
            if (stk.empty()) break;
            c = stk.pop();
        }
    }
    if (overflow && err) atomicOr(err, ERR_STACK);
    return h;
}

// A function of its own where it follows closest_hit's first walk, so that a kernel's registers
// are that walk's.
template <int STRIDE>
__device__ __noinline__ ClosestHit closest_reference(const float4 *nodes, const float4 *tri_isect, uint32_t *err,
                                                     Ray r, float tmin, float tmax, int *stack) {
    return closest_in_order<STRIDE>(nodes, tri_isect, err, r, tmin, tmax, stack);
}

// The closest hit of a ray made by make_ray over [tmin, tmax]: the sorted triangle slot or -1.
//
// Let S be the triangles whose own box passes the slab test over [tmin, tmax] and whose
// triangle test gives a distance t_k in it; b_k is the box's entry distance.  The reference
// accepts a triangle of S when it comes to it with max(t_k, b_k) <= its current tmax (boxes
// above it have smaller entries) and then sets tmax = t_k.  So if some w in S has
// t_k > L = max(t_w, b_w) for every other k, the reference returns w whatever its order: until
// it comes to w its tmax stays above L, so w's boxes pass and w is accepted; after that no k is.
//
// The walk below looks for w nearer child first.  Its bound is the L of the nearest triangle so
// far, and it skips only nodes that enter after the bound; the boxes of the closest-hit tree
// are inflated (rzk_sah.cu) so far that a triangle of S never has a distance below the entry of
// a box it lies in, whatever the rounding of either test.  So every triangle of S with
// t_k <= L is met (one skipped under an earlier bound lies beyond that bound's own triangle,
// which is then a witness itself), and the second distance met tells whether w stands alone.
// Where it does not (equal distances, shared edges), where the inflation does not cover the ray
// (closest_covered) or the scene has no such tree, the reference's own order decides.
// 524,288 scattered rays on 300k triangles, one per thread: 1,350 us in the reference's order, 590
// here; with the lanes refilled 433 us (B200).  Rays of the rooms here need the reference's own
// order about once in 1,000 (primary hits) to never (scattered rays).
__device__ __forceinline__ bool closest_covered(const DevScene &s, const Ray &r) {
    const V3 q = sub(r.o, ld3(s.cguard));
    return s.ctrav != nullptr && dot(q, q) <= s.cguard[3];   // no for a NaN
}

// The slab test of a sorted triangle's own box, formed from its vertices as the build forms it.
__device__ __forceinline__ bool own_box_hit(const DevScene &s, int slot, const Ray &r, float tmin, float tmax,
                                            float &enter) {
    const float *v = s.verts + 9 * (size_t)__ldg(s.perm + slot);
    const V3 p0 = mk(__ldg(v), __ldg(v + 1), __ldg(v + 2)), p1 = mk(__ldg(v + 3), __ldg(v + 4), __ldg(v + 5)),
             p2 = mk(__ldg(v + 6), __ldg(v + 7), __ldg(v + 8));
    const V3 lo = vmin(vmin(p0, p1), p2), hi = vmax(vmax(p0, p1), p2);
    return box_hit_fast(make_float4(lo.x, lo.y, lo.z, 0.0f), make_float4(hi.x, hi.y, hi.z, 0.0f), r, tmin, tmax, enter);
}

// The walk, one node or leaf per step, for kernels that refill their lanes between steps.
template <int STRIDE>
struct ClosestWalk {
    Stack<STRIDE> stk;
    Ray r;
    float tmin, tmax, bound, bt, lim, bb, bg, second;
    int c, best;
    bool sure;
    __device__ __forceinline__ void start(const DevScene &s, const Ray &ray, float t0, float t1) {
        r = ray;
        tmin = t0;
        tmax = bound = bt = t1;
        lim = t0;
        bb = bg = 0.0f;
        second = INFINITY;
        best = -1;
        stk.top = -1;
        sure = s.n_nodes > 0 && closest_covered(s, r);
        c = sure ? __float_as_int(__ldg(&s.ctrav[2].w)) : 0;
    }
    // true when the walk is over (finish() has the answer)
    __device__ __forceinline__ bool step(const DevScene &s) {
        if (!sure) return true;
        if (c < 0) {
            float4 ta, tb, tc;
            load_tri(s, -1 - c, ta, tb, tc);
            float t, b, g, enter = 0.0f;
            if (tri_hit<true>(ta, tb, tc, r, tmin, bound, &t, &b, &g) && own_box_hit(s, -1 - c, r, tmin, tmax, enter)) {
                if (t < bt || best < 0) {
                    if (best >= 0) second = fminf(second, bt);
                    best = -1 - c;
                    bt = t; bb = b; bg = g;
                    lim = enter;
                    bound = fmaxf(t, enter);
                } else {
                    second = fminf(second, t);
                }
            }
            if (stk.empty()) return true;
            c = stk.pop();
            return false;
        }
        float4 l0, l1, r0, r1;
        load_pair(s.ctrav + 2 * (c + 1), l0, l1, r0, r1);
        float tl, tr;
        const bool hl = box_hit_fast(l0, l1, r, tmin, bound, tl);
        const bool hr = box_hit_fast(r0, r1, r, tmin, bound, tr);
        if (hl && hr) {
            const bool lf = tl <= tr;
            if (!stk.push(__float_as_int(lf ? r0.w : l0.w))) sure = false;   // not met: as deep as the tree
            c = __float_as_int(lf ? l0.w : r0.w);
        } else if (hl || hr) {
            c = __float_as_int(hl ? l0.w : r0.w);
        } else {
            if (stk.empty()) return true;
            c = stk.pop();
        }
        return false;
    }
    // the answer; `stack`: room for the reference's own walk, STACK_CAP entries STRIDE2 apart
    template <int STRIDE2>
    __device__ __forceinline__ int finish(const DevScene &s, int *stack) {
        if (s.n_nodes == 0) return -1;
        if (!sure || (best >= 0 && second <= fmaxf(bt, lim))) {
            const ClosestHit h = closest_reference<STRIDE2>(s.nodes, s.tri_isect, s.err, r, tmin, tmax, stack);
            best = h.slot;
            bt = h.t; bb = h.beta; bg = h.gamma;
        }
        return best;
    }
};

// stk: STACK_CAP entries
template <int STRIDE>
__device__ __forceinline__ int closest_hit(const DevScene &s, const Ray &r, float tmin, float tmax,
                                           Stack<STRIDE> &stk, float *t_out, float *beta_out,
                                           float *gamma_out) {
    ClosestWalk<STRIDE> w;
    w.stk = stk;
    w.start(s, r, tmin, tmax);
    while (!w.step(s)) {}
    const int slot = w.template finish<STRIDE>(s, stk.base);
    if (slot >= 0) { *t_out = w.bt; *beta_out = w.bb; *gamma_out = w.bg; }
    return slot;
}

struct HitGeo {
    V3 p, ng, ns;
    Onb uvn;
    int mat, light;
    float t;
};

// Triangle::fill_hit_record (triangle.cc:277-296) + Surface::fill_hit_record
// (surface.cc:62-96) + the hit point r.org() + t * r.dir().
__device__ __forceinline__ void fill_hit(const DevScene &s, const Ray &r, int slot, float t,
                                         float beta, float gamma, HitGeo &h) {
    float4 s0 = __ldg(s.tri_shade + 2 * slot), s1 = __ldg(s.tri_shade + 2 * slot + 1);
    V3 n = mk(s0.x, s0.y, s0.z), u = mk(s1.x, s1.y, s1.z);
    int4 sf = __ldg(s.surf + __float_as_int(s0.w));
    V3 normal = n;
    V3 dn = sub(n, n);
    V3 shading = unit(add(add(n, scl(dn, beta)), scl(dn, gamma)));
    if (sf.y & RZK_SURF_FLIPPED) { normal = neg(normal); shading = neg(shading); }
    if ((sf.y & RZK_SURF_TWO_SIDED) && dot(shading, r.d) > 0.0f) {
        if (sf.x >= 0) { shading = neg(shading); normal = neg(normal); }
    }
    h.uvn = onb_from_nu(shading, u);
    h.p = add(r.o, scl(r.d, t));
    h.ng = normal;
    h.ns = shading;
    h.mat = sf.x;
    h.light = sf.z;
    h.t = t;
}

__device__ __forceinline__ void write_receiver(const HitGeo &h, const Ray &r, rzk_receiver *o) {
    float w[24];
    st3(w + 0, h.p); st3(w + 3, h.ng); st3(w + 6, h.ns); st3(w + 9, neg(r.d));
    st3(w + 12, h.uvn.u); st3(w + 15, h.uvn.v); st3(w + 18, h.uvn.n);
    w[21] = __int_as_float(h.mat); w[22] = __int_as_float(h.light); w[23] = __int_as_float(1);
    float4 *dst = reinterpret_cast<float4 *>(o);
#pragma unroll
    for (int k = 0; k < 6; ++k) dst[k] = make_float4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
}

__device__ __forceinline__ void write_miss(rzk_receiver *o) {
    float4 *dst = reinterpret_cast<float4 *>(o);
    float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < 5; ++k) dst[k] = z;
    dst[5] = make_float4(0.0f, __int_as_float(-1), __int_as_float(-1), __int_as_float(0));
}

// Camera::shoot_ray (camera.cc:52-65) followed by the Ray constructor.
__device__ __forceinline__ Ray camera_ray(const rzk_camera &c, int i, int j) {
    float H = (float)c.height;
    float px = (float)j + 0.5f;
    float py = H - 1 - (float)i + 0.5f;
    float fx = (px - c.cop[0]) / c.scale[0];
    float fy = (py - c.cop[1]) / c.scale[1];
    Onb o{ld3(c.u), ld3(c.v), ld3(c.n)};
    V3 dir = unit(l2w(o, mk(fx, fy, -c.focal)));
    return make_ray(ld3(c.eye), dir);
}

}  // namespace rzk
