// rzk_gather_dev.cuh - device building blocks of the gather kernels (rzk_gather.cu,
// rzk_batch.cu): bulk-copy / mbarrier helpers, receiver and material loads, the exact-zero
// pair test, the pair's radiance, the warp-packet any-hit and one persistent work item.
#pragma once

#include "rzk_traverse.cuh"

namespace rzk {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Bounded wait on a bulk-copy barrier: gives up after ~2^24 polls and reports it.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint32_t *err) {
    for (uint32_t it = 0; it < (1u << 24); ++it)
        if (mbar_try_wait(bar, parity)) return true;
    if (err) atomicOr(err, ERR_TIMEOUT);
    return false;
}

struct RecvRegs {
    V3 p, ng, ns, wo;
    Onb uvn;
    int mat;
};

__device__ __forceinline__ RecvRegs load_receiver(const rzk_receiver *r) {
    const float4 *q = reinterpret_cast<const float4 *>(r);
    float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2), d = __ldg(q + 3), e = __ldg(q + 4),
           f = __ldg(q + 5);
    RecvRegs o;
    o.p = mk(a.x, a.y, a.z);
    o.ng = mk(a.w, b.x, b.y);
    o.ns = mk(b.z, b.w, c.x);
    o.wo = mk(c.y, c.z, c.w);
    o.uvn.u = mk(d.x, d.y, d.z);
    o.uvn.v = mk(d.w, e.x, e.y);
    o.uvn.n = mk(e.z, e.w, f.x);
    o.mat = __float_as_int(f.y);
    return o;
}

// A VPL record in registers: six 16-byte loads (the library's VPL arrays are 16-byte aligned).
__device__ __forceinline__ rzk_vpl load_vpl(const rzk_vpl *v) {
    union {
        float4 f[6];
        rzk_vpl l;
    } u;
    static_assert(sizeof(u.f) == sizeof(u.l), "96-byte records");
#pragma unroll
    for (int k = 0; k < 6; ++k) u.f[k] = __ldg(reinterpret_cast<const float4 *>(v) + k);
    return u.l;
}

// r with its tangent basis vectors u, v read again from the receiver record
__device__ __forceinline__ RecvRegs reload_basis(RecvRegs r, const rzk_receiver *rec) {
    const float4 *q = reinterpret_cast<const float4 *>(rec);
    const float4 d = __ldg(q + 3), e = __ldg(q + 4);
    r.uvn.u = mk(d.x, d.y, d.z);
    r.uvn.v = mk(d.w, e.x, e.y);
    return r;
}

__device__ __forceinline__ rzk_material load_material(const rzk_material *m) {
    const float4 *q = reinterpret_cast<const float4 *>(m);
    float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    rzk_material o;
    o.type = __float_as_int(a.x);
    o.kd[0] = a.y; o.kd[1] = a.z; o.kd[2] = a.w;
    o.ks[0] = b.x; o.ks[1] = b.y; o.ks[2] = b.z;
    o.p0 = b.w; o.p1 = c.x;
    o.pad[0] = o.pad[1] = o.pad[2] = 0.0f;
    return o;
}

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ bool finite3(Rgb c) {
    return isfinite(c.r) && isfinite(c.g) && isfinite(c.b);
}

// Receiver index of a lane: a TW x (32 / TW) pixel tile of a row-major image of width
// img_w (8 x 4 by default; the autotuner also tries 4 x 8, 16 x 2 and 32 x 1), or 32
// consecutive receivers when img_w == 0.  -1 outside the receiver range.
template <int TW = 8>
__device__ __forceinline__ int lane_receiver(int gwarp, int lane, int n_recv, int img_w) {
    static_assert(TW == 4 || TW == 8 || TW == 16 || TW == 32, "warp tile width");
    constexpr int TH = 32 / TW;
    if (img_w <= 0) {
        int ri = gwarp * 32 + lane;
        return ri < n_recv ? ri : -1;
    }
    int tiles_x = (img_w + TW - 1) / TW;
    int x = (gwarp % tiles_x) * TW + (lane % TW);
    int y = (gwarp / tiles_x) * TH + (lane / TW);
    if (x >= img_w) return -1;
    long long ri = (long long)y * img_w + x;
    return ri < n_recv ? (int)ri : -1;
}

struct PairGeo {
    V3 q;
    float G;
    V3 wi;
    Rgb power;
};

// The VPL-only facts the per-pair tests use: its power is finite (all three components),
// and it was reached from behind its surface (a BRDF VPL whose stored incident direction
// makes a cosine <= ZERO_EPSILON with its normal: its BRDF's early-out then fires for every
// receiver).  The gathers form them once per VPL, one VPL per lane, instead of in every
// lane for every VPL.
__device__ __forceinline__ bool vpl_power_finite(const rzk_vpl &l) {
    return isfinite(l.contrib[0]) && isfinite(l.contrib[1]) && isfinite(l.contrib[2]);
}
__device__ __forceinline__ bool vpl_from_behind(const rzk_vpl &l) {
    return l.mat >= 0 && dot(ld3(l.wi), ld3(l.nn)) <= ZERO_EPSILON;
}

__device__ __forceinline__ PairGeo pair_geo(const RecvRegs &r, const rzk_vpl &l) {
    PairGeo pg;
    pg.q = ld3(l.p);
    pg.G = form_factor_abs(r.p, r.ns, pg.q, ld3(l.n));
    pg.wi = unit(sub(pg.q, r.p));
    pg.power = crgb(l.contrib[0], l.contrib[1], l.contrib[2]);
    return pg;
}

// Geometry of a pair and the exact-zero test of its term: returns false when either
// BRDF's early-out makes the term exactly zero (G and the power finite).  `fin` and
// `behind` are vpl_power_finite(l) and vpl_from_behind(l).
__device__ __forceinline__ bool pair_survives(const RecvRegs &r, const rzk_vpl &l, PairGeo &pg, bool fin,
                                              bool behind) {
    pg = pair_geo(r, l);
    if (isfinite(pg.G) && fin) {
        if (dot(pg.wi, r.uvn.n) <= ZERO_EPSILON || dot(r.wo, r.uvn.n) <= ZERO_EPSILON) return false;
        if (behind) return false;
        if (l.mat >= 0 && dot(neg(pg.wi), ld3(l.nn)) <= ZERO_EPSILON) return false;
    }
    return true;
}

__device__ __forceinline__ bool pair_survives(const RecvRegs &r, const rzk_vpl &l, PairGeo &pg) {
    return pair_survives(r, l, pg, vpl_power_finite(l), vpl_from_behind(l));
}

__device__ __forceinline__ Rgb pair_radiance(const GatherScene &s, const RecvRegs &r, const rzk_material &rm,
                                             const rzk_vpl &l, const PairGeo &pg, int mode, float tau) {
    Rgb sb = brdf_eval(rm, r.uvn, r.wo, pg.wi);
    Rgb lb;
    if (l.mat >= 0) {
        rzk_material lm = load_material(s.mats + l.mat);
        Onb lu{ld3(l.u), ld3(l.v), ld3(l.nn)};
        lb = brdf_eval(lm, lu, ld3(l.wi), neg(pg.wi));
    } else {
        lb = crgb(1.0f, 1.0f, 1.0f);
    }
    return radiance_terms(pg.power, sb, lb, pg.G, mode, tau);
}

__device__ __forceinline__ float warp_min_f(float x) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float warp_max_f(float x) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

// The shaft of a warp's shadow segments: all end at the VPL q, so a point of any of them is
// q + s (p - q) with s in [0, 1] and, per axis, p - q within [umin, umax] over the live lanes.
// A box [lo, hi] meets the shaft only if some s lies, on every axis, between the least and the
// largest s for which an s u of that interval reaches into [lo - q, hi - q].  The test below
// passes every box that box_hit_fast passes for one of the segments: a float slab test accepts
// points within 3 u (|plane| + |origin|) of the box, the float direction is within 4 u of
// (q - p) / |q - p|, and a direction component below 1e-6 is replaced by it (2e-6 of the
// distance); the planes are moved out by 8e-6 of the coordinates' size, the interval of u by as
// much, and the quotients by 2e-6 of themselves.  Comparisons that a NaN spoils pass.
struct Shaft {
    float qa[3], qb[3];   // q plus and minus the margin
    float n1[3], n2[3];   // entry: max((lo - qa) n1, (hi - qb) n2)
    float f[3], g[3];     // exit:  ((hi - qb), or where u < 0 (lo - qa)) f + g
    bool neg[3];
    __device__ __forceinline__ void set(V3 q, V3 p, bool live) {
        const float qv[3] = {q.x, q.y, q.z}, pv[3] = {p.x, p.y, p.z};
        float lo[3], hi[3], size = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float u = pv[a] - qv[a];
            lo[a] = warp_min_f(live ? u : INFINITY);
            hi[a] = warp_max_f(live ? u : -INFINITY);
            size = fmaxf(size, fabsf(qv[a]) + fmaxf(fabsf(lo[a]), fabsf(hi[a])));
        }
        const float eps = 8e-6f * size;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            qa[a] = qv[a] + eps;
            qb[a] = qv[a] - eps;
            const float u0 = lo[a] - eps, u1 = hi[a] + eps;
            const float r0 = __fdividef(1.0f, u0), r1 = __fdividef(1.0f, u1);
            const bool pos = u0 >= 0.0f;   // at zero 1 / u0 is +inf, which bounds the exit and not the entry
            neg[a] = u1 < 0.0f;
            n1[a] = neg[a] ? 0.0f : 0.999998f * r1;
            n2[a] = pos ? 0.0f : 0.999998f * r0;
            f[a] = 1.000002f * (pos ? r0 : neg[a] ? r1 : 0.0f);
            g[a] = pos || neg[a] ? 0.0f : 1e30f;
        }
    }
    __device__ __forceinline__ bool meets(float4 lo, float4 hi) const {
        const float l[3] = {lo.x - qa[0], lo.y - qa[1], lo.z - qa[2]};
        const float h[3] = {hi.x - qb[0], hi.y - qb[1], hi.z - qb[2]};
        float near = -2e-6f, far = 1.000002f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            near = fmaxf(near, fmaxf(l[a] * n1[a], h[a] * n2[a]));
            far = fminf(far, __fmaf_rn(neg[a] ? l[a] : h[a], f[a], g[a]));
        }
        return !(near > far);
    }
};

// Packet any-hit over the 8-wide any-hit tree.  Returns whether this lane's segment is
// unoccluded (lanes with act == false return false).
//
// `cache` and `cache2` (per lane) name the entries of the tree whose triangles last
// occluded this lane's receiver (most recent first), or -1.  They are tried first, then the
// entries cached by five neighbouring lanes: a triangle whose own box and triangle tests pass
// occludes the segment whichever way it was found, so a hit there is the traversal's
// answer; the entry of any triangle found becomes the lane's `cache`, the previous one its
// `cache2`.
//
// The walk tests nodes against the whole packet, not rays against nodes: a lane holds one child
// of one of up to four 8-wide nodes and tests its box against the packet's shaft, so a step
// covers 32 boxes; every leaf whose box meets the shaft is then tested by each live lane with its
// own ray (box, then triangle).  The answer is exact: a triangle is looked at whenever its own
// box passes for some lane, because the shaft test passes wherever box_hit_fast does, and it
// occludes a lane only by that lane's own tests.  A packet whose rays are far apart for the
// triangles' size (a 192-pixel image: 81 leaves in the shaft, 6 of them entered) refines a step's
// boxes by the rays themselves, each lane its box against every live ray.
//
// Bound by the issue rate.  One ray per lane and two boxes a step took about 95 instructions for
// 2 boxes, 40 steps a packet; this takes about 80 for 32, 7 to 12 steps.  512 x 512 x 32,768 VPLs,
// 300k triangles 103 -> 61 ms; ten requests of up to 192 x 192 x 3,000, 10k to 30k triangles
// 37.5 -> 23.7 (64 without the refinement; its limit at 4 m > live + 8: 25.0, m > live: 33.2,
// 2 m > live + 12: 24.3); LightSlice's tracing 11.6 -> 5.4; 36 triangles 8.1 -> 7.5 (B200, with
// VPL tiles of 16 instead of 32, which leave L1 124 KB instead of 28: 103 -> 73 ms with 32).
constexpr int kWideFan = 8;
constexpr int kWideMulti = 64;    // most pending nodes with which four are taken at once
// from at most kWideMulti + 28 pending, one node at a time adds at most 7 a level; 21 levels of a
// 62-deep binary tree taken three at a time
constexpr int kWideStack = (kWideMulti + 28 + 7 * 21 + 1 + 3) / 4 * 4;
constexpr int kPacketInts = kWideStack + 64;   // a packet's shared memory: pending nodes, 16 VPLs' margins
static_assert(kWideStack % 4 == 0, "the margins are read as float4");

__device__ __forceinline__ bool entry_occludes(const GatherScene &s, int entry, const Ray &ray, float tmax) {
    const float4 *p = s.wide8 + 2 * (size_t)entry;
    const float4 lo = __ldg(p), hi = __ldg(p + 1);
    float t = 0.0f;
    if (!box_hit_fast(lo, hi, ray, s.tmin, tmax, t)) return false;
    float4 ta, tb, tc;
    load_tri(s, -1 - __float_as_int(lo.w), ta, tb, tc);
    return tri_hit<false>(ta, tb, tc, ray, s.tmin, tmax, nullptr, nullptr, nullptr);
}

__device__ __forceinline__ bool packet_visible(const GatherScene &s, V3 p, V3 q, const Ray &ray, float tmax, bool act,
                                               int *stk, int &cache, int &cache2) {
    if (s.n_nodes == 0) return act;
    const int lane = threadIdx.x & 31;
    bool alive = act;
    // The lane's own two entries, then those cached by the lanes at xor distances 1, 8, 2, 16 and
    // 4: in an 8 x 4 pixel tile those are the neighbouring pixels, whose shadow rays toward the
    // same VPL run almost parallel and are often blocked by the same triangle.  The same rule
    // applies (own box and triangle tests), so the answer is still exact; a lane blocked by
    // a neighbour's entry adopts it.  Every lane takes part in each shuffle.  One copy of the
    // tests: unrolled, the kernels outgrow the instruction cache.
    constexpr unsigned long long kDistance = 0x041002080100ull << 8;   // one byte a round: 0, 0, 1, 8, 2, 16, 4
#pragma unroll 1
    for (int k = 0; k < 7; ++k) {
        const int other = __shfl_xor_sync(kFull, k == 1 ? cache2 : cache, (int)((kDistance >> (8 * k)) & 31u));
        if (alive && other >= 0 && (k == 0 || other != cache) && entry_occludes(s, other, ray, tmax)) {
            alive = false;
            if (k > 0) {
                cache2 = cache;
                cache = other;
            }
        }
        if (!__any_sync(kFull, alive)) return false;
    }

    Shaft sh;
    sh.set(q, p, alive);
    int n = 1;
    if (lane == 0) stk[0] = 0;
    __syncwarp();
    const unsigned below = (1u << lane) - 1u;
    do {
        const int take = n <= kWideMulti ? min(n, 4) : 1;
        n -= take;
        bool meets = false;
        int entry = 0, code = 0;
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
        if ((lane >> 3) < take) {
            entry = stk[n + (lane >> 3)] * kWideFan + (lane & 7);
            const float4 *e = s.wide8 + 2 * (size_t)entry;
            lo = __ldg(e);
            hi = __ldg(e + 1);
            code = __float_as_int(lo.w);
            meets = code != kWideEmpty && sh.meets(lo, hi);
        }
        // a wide packet's shaft holds many boxes that no ray enters: where they are many against
        // the live lanes, each lane tests its box with every live ray
        unsigned live = __ballot_sync(kFull, alive);
        if (2 * __popc(__ballot_sync(kFull, meets)) > __popc(live) + 8) {
            bool entered = false;
            for (; live; live &= live - 1u) {
                const int k = __ffs(live) - 1;
                Ray other;
                other.inv_d = mk(__shfl_sync(kFull, ray.inv_d.x, k), __shfl_sync(kFull, ray.inv_d.y, k),
                                 __shfl_sync(kFull, ray.inv_d.z, k));
                other.org_inv_d = mk(__shfl_sync(kFull, ray.org_inv_d.x, k), __shfl_sync(kFull, ray.org_inv_d.y, k),
                                     __shfl_sync(kFull, ray.org_inv_d.z, k));
                const float far = __shfl_sync(kFull, tmax, k);
                float t = 0.0f;
                entered |= box_hit_fast(lo, hi, other, s.tmin, far, t);
            }
            meets = meets && entered;
        }
        const unsigned inner = __ballot_sync(kFull, meets && code >= 0);
        if (inner) {
            if (n + __popc(inner) > kWideStack) {   // not met: a tree deeper than the stack covers
                if (lane == 0 && s.err) atomicOr(s.err, ERR_STACK);
                break;
            }
            if (meets && code >= 0) stk[n + __popc(inner & below)] = code;
            n += __popc(inner);
            __syncwarp();
        }
        for (unsigned leaf = __ballot_sync(kFull, meets && code < 0); leaf; leaf &= leaf - 1u) {
            const int e = __shfl_sync(kFull, entry, __ffs(leaf) - 1);
            const float4 *pe = s.wide8 + 2 * (size_t)e;
            const float4 lo = __ldg(pe), hi = __ldg(pe + 1);
            float t = 0.0f;
            const bool in = alive && box_hit_fast(lo, hi, ray, s.tmin, tmax, t);
            if (!__any_sync(kFull, in)) continue;
            float4 ta, tb, tc;
            load_tri(s, -1 - __float_as_int(lo.w), ta, tb, tc);
            if (in && tri_hit<false>(ta, tb, tc, ray, s.tmin, tmax, nullptr, nullptr, nullptr)) {
                alive = false;
                if (cache != e) { cache2 = cache; cache = e; }
            }
            if (!__any_sync(kFull, alive)) return false;
        }
    } while (n > 0);
    return alive;
}

// Which of 32 receivers x 16 VPLs can have a term at all, from the tensor cores: the receiver
// behind the VPL's surface, or the VPL behind the receiver's, is the sign of a dot product with
// q - p, and with both taken relative to a point c of the tile
//   n_r . (q - p)  = (n_r, -n_r . (p - c)) . (q - c, 1)
//   nn_v . (q - p) = (p - c, 1) . (-nn_v, nn_v . (q - c))
// so the two tests of a block are two products with an inner dimension of 4 (operands rounded to
// tf32).  A pair is dropped only where a product is past zero by more than
// 2.4e-3 (|q - c| + R) + 1e-8, R the largest |p - c|: the rounded operands are within 2^-11 of
// themselves, so a product of unit normals is within 1e-3 |q - c| + 0.5e-3 R (or the other way
// round), and what is left bounds the rounding of the exact test and keeps |q - p| above 1e-8;
// normals that are not unit vectors, powers that are not finite and coordinates past 1e8 drop
// nothing (an infinite margin, which no product is past).  Every dropped pair fails pair_survives,
// which decides the others, so the surviving pairs are the same.  The division-free test it
// replaces took about 55 instructions a VPL, this about 12: 512^2 x 32,768 VPLs 61.0 -> 45.8 ms,
// its clustered gather 7.1 -> 6.7.
__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

struct FaceTest {
    uint32_t a1[4], a2[4];   // rows g and g + 8 of the two 16-receiver blocks, component lane % 4
    V3 c;
    float R;
    bool ok;                 // this lane's receiver may be dropped
    __device__ __forceinline__ void init(const RecvRegs &r, bool active, int lane) {
        const int src = __ffs(__ballot_sync(kFull, active)) - 1;   // the caller has an active lane
        c = mk(__shfl_sync(kFull, r.p.x, src), __shfl_sync(kFull, r.p.y, src), __shfl_sync(kFull, r.p.z, src));
        const V3 x = sub(r.p, c), n = r.uvn.n;
        R = warp_max_f(active ? len(x) : 0.0f);
        const float nn = dot(n, n);
        ok = active && nn >= 0.98f && nn <= 1.02f && dot(r.ns, r.ns) <= 4.0f;
        const float k1 = -dot(n, x);
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = 8 * i + g;
            const float n0 = __shfl_sync(kFull, n.x, row), n1 = __shfl_sync(kFull, n.y, row),
                        n2 = __shfl_sync(kFull, n.z, row), n3 = __shfl_sync(kFull, k1, row);
            const float x0 = __shfl_sync(kFull, x.x, row), x1 = __shfl_sync(kFull, x.y, row),
                        x2 = __shfl_sync(kFull, x.z, row);
            a1[i] = to_tf32(t == 0 ? n0 : t == 1 ? n1 : t == 2 ? n2 : n3);
            a2[i] = to_tf32(t == 0 ? x0 : t == 1 ? x1 : t == 2 ? x2 : 1.0f);
        }
    }
    // bit v of the result: this lane's receiver may have a term with VPL v of `vpls` (shared
    // memory; the first `count` of 16, fin as from vpl_power_finite for VPL lane % 16).
    // margin: 16 x float4 of the warp's shared memory.
    __device__ __forceinline__ uint32_t candidates(const rzk_vpl *vpls, int count, bool fin, float4 *margin,
                                                   int lane) const {
        const int g = lane >> 2, t = lane & 3;
        {
            const rzk_vpl &l = vpls[min(lane & 15, count - 1)];
            const V3 x = sub(ld3(l.p), c), ln = ld3(l.n), lnn = ld3(l.nn);
            const float reach = len(x) + R, m = 2.4e-3f * reach + 1e-8f, un = dot(lnn, lnn);
            const bool use = fin && dot(ln, ln) <= 4.0f && reach < 1e8f;
            if (lane < 16)
                margin[lane] = make_float4(dot(lnn, x), use ? m : INFINITY,
                                           use && l.mat >= 0 && un >= 0.98f && un <= 1.02f ? m : INFINITY, 0.0f);
        }
        __syncwarp();
        uint32_t rows[2] = {0u, 0u};   // receivers g | g + 8 << 16, and the same of the second block
        const float ct = t == 0 ? c.x : t == 1 ? c.y : c.z;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const rzk_vpl &l = vpls[8 * h + g];
            const uint32_t b1 = to_tf32(t < 3 ? l.p[t < 3 ? t : 0] - ct : 1.0f);
            const uint32_t b2 = to_tf32(t < 3 ? -l.nn[t < 3 ? t : 0] : margin[8 * h + g].x);
            const float4 m0 = margin[8 * h + 2 * t], m1 = margin[8 * h + 2 * t + 1];
            const uint32_t bit = 1u << (8 * h + 2 * t);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float d[4], e[4];
                asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
                    : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                    : "r"(a1[2 * i]), "r"(a1[2 * i + 1]), "r"(b1), "f"(0.0f));
                asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
                    : "=f"(e[0]), "=f"(e[1]), "=f"(e[2]), "=f"(e[3])
                    : "r"(a2[2 * i]), "r"(a2[2 * i + 1]), "r"(b2), "f"(0.0f));
                if (!(d[0] < -m0.y) && !(e[0] > m0.z)) rows[i] |= bit;
                if (!(d[1] < -m1.y) && !(e[1] > m1.z)) rows[i] |= bit << 1;
                if (!(d[2] < -m0.y) && !(e[2] > m0.z)) rows[i] |= bit << 16;
                if (!(d[3] < -m1.y) && !(e[3] > m1.z)) rows[i] |= bit << 17;
            }
        }
        // the four lanes of a group hold two columns of each eight
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            rows[i] |= __shfl_xor_sync(kFull, rows[i], 1);
            rows[i] |= __shfl_xor_sync(kFull, rows[i], 2);
        }
        const uint32_t lo = __shfl_sync(kFull, rows[0], 4 * (lane & 7)), hi = __shfl_sync(kFull, rows[1], 4 * (lane & 7));
        const uint32_t mine = ((lane & 16 ? hi : lo) >> (2 * (lane & 8))) & 0xffffu;
        __syncwarp();   // the margins are read before the next block's are written
        return (ok ? mine : 0xffffu) & ((1u << count) - 1u);
    }
};

// Per-warp staging state of the persistent gathers: the warp's two VPL tiles, their
// barriers (with the number of completed phases of each) and its packet stack.
template <int TILE>
struct WarpStage {
    rzk_vpl (*tl)[TILE];
    uint64_t *mb;
    int *stk;
    uint32_t uses[2];
    __device__ __forceinline__ void init(rzk_vpl (*tiles)[TILE], uint64_t *bar, int *stack, int lane) {
        tl = tiles;
        mb = bar;
        stk = stack;
        uses[0] = uses[1] = 0u;
        if (lane == 0) {
            mbar_init(&mb[0], 1);
            mbar_init(&mb[1], 1);
            fence_barrier_init();
        }
        __syncwarp();
    }
};

// Warp tiles of an image (TW x (32 / TW) pixels each), or of 32 consecutive receivers
// without an image width.
template <int TW = 8>
__host__ __device__ __forceinline__ long long warp_tiles(long long n_recv, int img_w) {
    if (img_w <= 0) return (n_recv + 31) / 32;
    const long long img_h = (n_recv + img_w - 1) / img_w;
    return (long long)((img_w + TW - 1) / TW) * ((img_h + 32 / TW - 1) / (32 / TW));
}

// One work item of the persistent gathers: the 32 receivers of warp tile `wt` against VPL
// chunk `chunk`.  Each lane hands `sink(ri, sum, ok)` its receiver's index (-1 for none)
// and the sum of its terms over the chunk's VPLs in VPL order (zero without a receiver);
// ok is false, and the sum incomplete, if a bounded wait gave up (reported in the error
// word), and the item then returns false.  The tile shape changes which receivers share a
// packet, never a receiver's sum.
template <int TILE, int TW = 8, class Sink>
__device__ __forceinline__ bool gather_item(const GatherScene &s, const rzk_receiver *recv, int n_recv, int img_w,
                                            const rzk_vpl *vpls, int n_vpl, int chunk, int wt, int chunk_len,
                                            int mode, float tau, WarpStage<TILE> &ws, int lane, Sink &&sink) {
    const int ri = lane_receiver<TW>(wt, lane, n_recv, img_w);
    const int j0 = chunk * chunk_len;
    const int j1 = min(n_vpl, j0 + chunk_len);
    const int n_tiles = (j1 - j0 + TILE - 1) / TILE;

    RecvRegs r;
    r.p = mk(0.0f, 0.0f, 0.0f);   // lanes without a receiver still form (unused) rays
    bool active = false;
    if (ri >= 0) {
        r = load_receiver(recv + ri);
        active = r.mat >= 0;
    }
    // a tile of inactive lanes, or an empty chunk, contributes nothing: no VPL stream (an
    // empty chunk must not arm a barrier phase that no wait consumes)
    if (n_tiles <= 0 || !__any_sync(kFull, active)) {
        sink(ri, crgb(0.0f, 0.0f, 0.0f), true);
        return true;
    }
    Rgb sum = crgb(0.0f, 0.0f, 0.0f);
    unsigned long long n_rays = 0;         // shadow rays of this item (lane 0's count)
    int occ_cache = -1, occ_cache2 = -1;   // this lane's last two occluders (any-hit tree leaves)
    if (lane == 0) {
        int cnt = min(TILE, j1 - j0);
        fence_proxy_async();
        mbar_expect_tx(&ws.mb[0], cnt * (uint32_t)sizeof(rzk_vpl));
        bulk_g2s(&ws.tl[0][0], vpls + j0, cnt * (uint32_t)sizeof(rzk_vpl), &ws.mb[0]);
    }
    FaceTest face;
    face.init(r, active, lane);
    float4 *margin = reinterpret_cast<float4 *>(ws.stk + kWideStack);
    for (int k = 0; k < n_tiles; ++k) {
        const int buf = k & 1;
        if (lane == 0 && k + 1 < n_tiles) {
            int jn = j0 + (k + 1) * TILE;
            int cnt = min(TILE, j1 - jn);
            fence_proxy_async();
            mbar_expect_tx(&ws.mb[buf ^ 1], cnt * (uint32_t)sizeof(rzk_vpl));
            bulk_g2s(&ws.tl[buf ^ 1][0], vpls + jn, cnt * (uint32_t)sizeof(rzk_vpl), &ws.mb[buf ^ 1]);
        }
        bool ok = mbar_wait_bounded(&ws.mb[buf], ws.uses[buf] & 1u, lane == 0 ? s.err : nullptr);
        ws.uses[buf]++;
        if (__any_sync(kFull, !ok)) {
            sink(ri, sum, false);
            return false;
        }
        const rzk_vpl *tile = ws.tl[buf];
        const int cnt = min(TILE, j1 - (j0 + k * TILE));
        // the VPL-only facts of the tile's VPLs, one VPL per lane
        static_assert(TILE <= 32, "one VPL per lane");
        const rzk_vpl &mine = tile[lane < cnt ? lane : 0];
        const unsigned fin_mask = __ballot_sync(kFull, lane < cnt && vpl_power_finite(mine));
        const unsigned behind_mask = __ballot_sync(kFull, lane < cnt && vpl_from_behind(mine));
        uint32_t cand = face.candidates(tile, min(cnt, 16), (fin_mask >> (lane & 15)) & 1u, margin, lane);
        if (TILE > 16 && cnt > 16)
            cand |= face.candidates(tile + 16, cnt - 16, (fin_mask >> (16 + (lane & 15))) & 1u, margin, lane) << 16;
        if (!active) cand = 0u;
        for (unsigned todo = __reduce_or_sync(kFull, cand); todo; todo &= todo - 1u) {
            const int v = __ffs(todo) - 1;
            const rzk_vpl &l = tile[v];
            const bool fin = (fin_mask >> v) & 1u, behind = (behind_mask >> v) & 1u;
            PairGeo pg;
            bool act = ((cand >> v) & 1u) && pair_survives(r, l, pg, fin, behind);
            const unsigned am = __ballot_sync(kFull, act);
            if (!am) continue;
            n_rays += (unsigned)__popc(am);
            Ray ray = make_ray(r.p, sub(pg.q, r.p));
            float tmax = len(sub(pg.q, r.p)) - s.tmin;
            if (packet_visible(s, r.p, ld3(l.p), ray, tmax, act, ws.stk, occ_cache, occ_cache2)) {
                // the pair's geometry (recomputed: the same operations on the same values),
                // the material and the receiver's tangent basis are read or formed again here
                // rather than held in registers through the traversal
                PairGeo pv;
                pair_survives(r, l, pv, fin, behind);
                sum = cadd(sum, pair_radiance(s, reload_basis(r, recv + ri), load_material(s.mats + r.mat), l, pv,
                                              mode, tau));
            }
        }
        __syncwarp();
    }
    if (lane == 0 && s.rays && n_rays) atomicAdd(s.rays, n_rays);
    sink(ri, sum, true);
    return true;
}

// Sink of gather_item writing an item's partial sums to chunk `chunk`'s plane of `partial`
// (planes of n_recv x 3 floats); nothing is written for an item whose wait gave up.
struct PlaneSink {
    float *partial;
    int n_recv, chunk;
    __device__ __forceinline__ void operator()(int ri, Rgb sum, bool ok) const {
        if (ok && ri >= 0) {
            // partial sums are read once by the chunk reduction: streaming stores keep them
            // from displacing the traversal working set in L2
            float *o = partial + 3 * ((size_t)chunk * n_recv + ri);
            __stcs(o, sum.r); __stcs(o + 1, sum.g); __stcs(o + 2, sum.b);
        }
    }
};

// Visibility half of gather_item, for gathers split into a tracing pass and a summing
// pass: the 32 receivers of warp tile `wt` (img_w as in lane_receiver) against VPLs [j0, j1); masks[j - j0] = ballot of
// the lanes whose pair's term is not exactly zero (pair_survives) and whose shadow segment
// is unoccluded - exactly the pairs gather_item adds.  Returns false if a bounded wait gave
// up (reported in the error word).  FACE: with the facing test; without it every VPL goes to
// pair_survives, which in items of few VPLs is the shorter way.
template <int TILE, bool FACE = true>
__device__ __forceinline__ bool visibility_item(const GatherScene &s, const rzk_receiver *recv, int n_recv, int img_w,
                                                const rzk_vpl *vpls, int j0, int j1, int wt, WarpStage<TILE> &ws,
                                                int lane, uint32_t *masks) {
    const int ri = lane_receiver(wt, lane, n_recv, img_w);
    const int n_tiles = (j1 - j0 + TILE - 1) / TILE;
    RecvRegs r;
    r.p = mk(0.0f, 0.0f, 0.0f);
    bool active = false;
    if (ri >= 0) {
        r = load_receiver(recv + ri);
        active = r.mat >= 0;
    }
    if (n_tiles <= 0 || !__any_sync(kFull, active)) {
        for (int j = j0 + lane; j < j1; j += 32) masks[j - j0] = 0u;
        return true;
    }
    int occ_cache = -1, occ_cache2 = -1;
    unsigned long long n_rays = 0;
    if (lane == 0) {
        int cnt = min(TILE, j1 - j0);
        fence_proxy_async();
        mbar_expect_tx(&ws.mb[0], cnt * (uint32_t)sizeof(rzk_vpl));
        bulk_g2s(&ws.tl[0][0], vpls + j0, cnt * (uint32_t)sizeof(rzk_vpl), &ws.mb[0]);
    }
    FaceTest face;
    if (FACE) face.init(r, active, lane);
    float4 *margin = reinterpret_cast<float4 *>(ws.stk + kWideStack);
    for (int k = 0; k < n_tiles; ++k) {
        const int buf = k & 1;
        if (lane == 0 && k + 1 < n_tiles) {
            int jn = j0 + (k + 1) * TILE;
            int cnt = min(TILE, j1 - jn);
            fence_proxy_async();
            mbar_expect_tx(&ws.mb[buf ^ 1], cnt * (uint32_t)sizeof(rzk_vpl));
            bulk_g2s(&ws.tl[buf ^ 1][0], vpls + jn, cnt * (uint32_t)sizeof(rzk_vpl), &ws.mb[buf ^ 1]);
        }
        bool ok = mbar_wait_bounded(&ws.mb[buf], ws.uses[buf] & 1u, lane == 0 ? s.err : nullptr);
        ws.uses[buf]++;
        if (__any_sync(kFull, !ok)) return false;
        const rzk_vpl *tile = ws.tl[buf];
        const int cnt = min(TILE, j1 - (j0 + k * TILE));
        // the VPL-only facts of the tile's VPLs, one VPL per lane (as in gather_item)
        static_assert(TILE <= 32, "one VPL per lane");
        const rzk_vpl &mine = tile[lane < cnt ? lane : 0];
        const unsigned fin_mask = __ballot_sync(kFull, lane < cnt && vpl_power_finite(mine));
        const unsigned behind_mask = __ballot_sync(kFull, lane < cnt && vpl_from_behind(mine));
        uint32_t word = 0u;   // the ballot of the tile's VPL `lane`
        uint32_t cand = cnt == 32 ? kFull : (1u << cnt) - 1u;
        if (FACE) cand = face.candidates(tile, min(cnt, 16), (fin_mask >> (lane & 15)) & 1u, margin, lane);
        if (FACE && TILE > 16 && cnt > 16)
            cand |= face.candidates(tile + 16, cnt - 16, (fin_mask >> (16 + (lane & 15))) & 1u, margin, lane) << 16;
        if (!active) cand = 0u;
        for (unsigned todo = __reduce_or_sync(kFull, cand); todo; todo &= todo - 1u) {
            const int v = __ffs(todo) - 1;
            const rzk_vpl &l = tile[v];
            const bool fin = (fin_mask >> v) & 1u, behind = (behind_mask >> v) & 1u;
            PairGeo pg;
            const bool act = ((cand >> v) & 1u) && pair_survives(r, l, pg, fin, behind);
            const unsigned am = __ballot_sync(kFull, act);
            if (!am) continue;
            n_rays += (unsigned)__popc(am);
            Ray ray = make_ray(r.p, sub(pg.q, r.p));
            float tmax = len(sub(pg.q, r.p)) - s.tmin;
            const unsigned vis =
                __ballot_sync(kFull, packet_visible(s, r.p, ld3(l.p), ray, tmax, act, ws.stk, occ_cache, occ_cache2));
            if (lane == v) word = vis;
        }
        if (lane < cnt) masks[k * TILE + lane] = word;
        __syncwarp();
    }
    if (lane == 0 && s.rays && n_rays) atomicAdd(s.rays, n_rays);
    return true;
}

// Summing half for one warp: each lane's sum, in VPL order, of its receiver's terms with the VPLs
// of [j0, j1) that `masks` (first word: VPL j0's, from visibility_item) marks.  A lane that is not
// `active` (no receiver, or one without a material) adds nothing whatever its bits say: an item
// whose bounded wait gave up leaves its words unwritten.
__device__ __forceinline__ Rgb shade_marked(const GatherScene &s, const RecvRegs &r, const rzk_material &rm,
                                            bool active, const rzk_vpl *vpls, int j0, int j1,
                                            const uint32_t *masks, int mode, float tau, int lane) {
    Rgb sum = crgb(0.0f, 0.0f, 0.0f);
    for (int b = j0; b < j1; b += 32) {
        const uint32_t word = b + lane < j1 ? __ldcs(masks + (b - j0) + lane) : 0u;
        for (unsigned todo = __ballot_sync(kFull, word != 0u); todo; todo &= todo - 1u) {
            const int v = __ffs(todo) - 1;
            const bool marked = (__shfl_sync(kFull, word, v) >> lane) & 1u;
            if (!marked || !active) continue;
            const rzk_vpl l = load_vpl(vpls + b + v);
            sum = cadd(sum, pair_radiance(s, r, rm, l, pair_geo(r, l), mode, tau));
        }
    }
    return sum;
}

// Summing half with one order of additions per sum but the terms formed in parallel: the warps
// of a block (at least three) take the VPLs of [j0, j1) in turn, 32 VPLs at a time, and leave the
// terms in `terms`; then thread t < 96 adds channel t / 32 of receiver t % 32 in VPL order.
// Returns that thread's sum.  `masks` as from visibility_item, its first word VPL j0's; `active` as
// in shade_marked.
template <int WARPS>
__device__ __forceinline__ float shade_chunk(const GatherScene &s, const RecvRegs &r, bool active, const rzk_vpl *vpls,
                                             int j0, int j1, const uint32_t *masks, int mode, float tau,
                                             float (*terms)[3][32]) {
    static_assert(WARPS >= 3, "a warp per channel");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float acc = 0.0f;
    for (int b = j0; b < j1; b += 32) {
        const uint32_t word = b + lane < j1 ? __ldg(masks + (b - j0) + lane) : 0u;
        const unsigned some = __ballot_sync(kFull, word != 0u);   // the same in every warp
        if (!some) continue;
        int k = 0;
        for (unsigned todo = some; todo; todo &= todo - 1u, ++k) {
            if (k % WARPS != w) continue;
            const int v = __ffs(todo) - 1;
            const bool marked = (__shfl_sync(kFull, word, v) >> lane) & 1u;
            if (!marked || !active) continue;
            const rzk_vpl l = load_vpl(vpls + b + v);
            const PairGeo pg = pair_geo(r, l);
            const Rgb L = pair_radiance(s, r, load_material(s.mats + r.mat), l, pg, mode, tau);
            terms[v][0][lane] = L.r;
            terms[v][1][lane] = L.g;
            terms[v][2][lane] = L.b;
        }
        __syncthreads();
        if (w < 3) {
            for (unsigned todo = some; todo; todo &= todo - 1u) {
                const int v = __ffs(todo) - 1;
                const bool marked = (__shfl_sync(kFull, word, v) >> lane) & 1u;
                if (marked && active) acc += terms[v][w][lane];
            }
        }
        __syncthreads();
    }
    return acc;
}

// Summing half: the 32 receivers of warp tile `wt` add, in VPL order, the terms of the
// pairs that `masks` (one word per VPL, from visibility_item) marks - the same values in
// the same order as gather_item with one chunk, so the sums are bit-identical to it.
// WEIGHTED: VPL j's radiance is multiplied by weights[j] before it is added (a cluster
// representative standing for its cluster).  Writes partial[3 * ri ...].
template <bool WEIGHTED>
__device__ __forceinline__ void shade_item(const GatherScene &s, const rzk_receiver *recv, int n_recv, int img_w,
                                           const rzk_vpl *vpls, int n_vpl, const uint32_t *masks, int wt, int mode,
                                           float tau, float *partial, int lane, const float *weights) {
    const int ri = lane_receiver(wt, lane, n_recv, img_w);
    if (ri < 0) return;
    RecvRegs r = load_receiver(recv + ri);
    Rgb sum = crgb(0.0f, 0.0f, 0.0f);
    if (r.mat >= 0) {
        const rzk_material rm = load_material(s.mats + r.mat);
        const unsigned bit = 1u << lane;
        for (int j = 0; j < n_vpl; ++j) {
            if (!(masks[j] & bit)) continue;
            const rzk_vpl &l = vpls[j];
            PairGeo pg;
            pair_survives(r, l, pg);
            Rgb L = pair_radiance(s, r, rm, l, pg, mode, tau);
            if (WEIGHTED) {
                const float w = weights[j];
                L = crgb(w * L.r, w * L.g, w * L.b);
            }
            sum = cadd(sum, L);
        }
    }
    float *o = partial + 3 * (size_t)ri;
    o[0] = sum.r; o[1] = sum.g; o[2] = sum.b;
}

}  // namespace rzk
