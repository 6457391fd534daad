// rzk_sah.cu - a surface-area-heuristic tree over the scene's triangles for any-hit
// (shadow-ray) traversal.
//
// The any-hit answer is "some triangle whose own box passes the slab test and whose
// triangle test passes": every inner box is the exact min/max of the boxes below it and the
// rounded slab test is monotone in the bounds, so which tree leads to a triangle never
// changes whether it is tested under its own box.  Any tree with one triangle per leaf,
// leaf box = the triangle's box (the reference's leaf box, aggregate_bvh.cc:183-209) and
// inner box = the exact union of its children therefore returns the reference's visibility
// bit for bit; a tree with less overlap than the Morton LBVH simply reaches the answer in
// fewer steps.  Closest hits walk this tree's nodes in inflated boxes (below) and go back to the
// reference tree, whose visit order decides ties, only where a tie is possible or those boxes do
// not cover the ray.
//
// Binned SAH: 32 bins on the centroid axis of largest extent; past depth 32 or when no split
// separates the centroids, the median of the Morton order the slots came in.  Nodes are
// numbered depth-first with siblings adjacent and packed like the reference tree (two float4
// per node slot).
//
// Built on the device in two phases.  A node of more than kSmall triangles is split by one
// block (bounds, bins in shared memory, stable partition), all such nodes of a level in one
// launch; a node of at most kSmall triangles is finished by one warp, its boxes in shared
// memory and its whole subtree built there without another launch.  Both phases stay short
// because the top levels move the most data per block and there are few of them.  Every
// result is independent of scheduling: bounds and bins are exact minima, maxima and counts,
// the partition is stable, and a node's number follows from its range alone - an inner node
// over the positions [begin, end) reached through `lefts` left turns has begin + lefts inner
// nodes before it in depth-first order, so its children are nodes 1 + 2 (begin + lefts) and
// the next.
#include "rzk_internal.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>

namespace rzk {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBins = 32;          // one bin per lane of the warp that chooses the split
constexpr int kMedianDepth = 32;   // deeper nodes are halved: depth stays under 32 + log2(n)
constexpr int kSmall = 256;        // triangles whose subtree one warp builds
constexpr int kLargeThreads = 1024;
constexpr int kSmallWarps = 4;     // 4 x 10.8 KB of shared memory per block
constexpr int kMaxLevels = 64;

// A node to build: the triangles idx[begin, end), its node index, and depth | lefts << 8 |
// buffer << 16 (which of the two index buffers holds the range).
struct Task {
    int begin, end, node, info;
};
static_assert(sizeof(Task) == 16, "one 16-byte load");

struct Box {
    V3 mn, mx;
    __device__ __forceinline__ void reset() {
        mn = mk(FLT_MAX, FLT_MAX, FLT_MAX);
        mx = mk(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    }
    __device__ __forceinline__ void grow(V3 a, V3 b) {
        mn = mk(fminf(mn.x, a.x), fminf(mn.y, a.y), fminf(mn.z, a.z));
        mx = mk(fmaxf(mx.x, b.x), fmaxf(mx.y, b.y), fmaxf(mx.z, b.z));
    }
    __device__ __forceinline__ float area() const {
        const float dx = mx.x - mn.x, dy = mx.y - mn.y, dz = mx.z - mn.z;
        return dx < 0.0f ? 0.0f : dx * dy + dy * dz + dz * dx;
    }
};

__device__ __forceinline__ V3 centroid(float4 lo, float4 hi) {
    return mk(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
}
__device__ __forceinline__ V3 xyz(float4 f) { return mk(f.x, f.y, f.z); }
__device__ __forceinline__ float comp(V3 v, int d) { return d == 0 ? v.x : d == 1 ? v.y : v.z; }

// floats as ints of the same order, for integer min / max reductions and atomics
__device__ __forceinline__ int ord(float f) {
    const int i = __float_as_int(f);
    return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float unord(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

__device__ __forceinline__ V3 warp_min(V3 v) {
    return mk(unord(__reduce_min_sync(kFull, ord(v.x))), unord(__reduce_min_sync(kFull, ord(v.y))),
              unord(__reduce_min_sync(kFull, ord(v.z))));
}
__device__ __forceinline__ V3 warp_max(V3 v) {
    return mk(unord(__reduce_max_sync(kFull, ord(v.x))), unord(__reduce_max_sync(kFull, ord(v.y))),
              unord(__reduce_max_sync(kFull, ord(v.z))));
}

// The axis of largest centroid extent and the binning along it.
struct Binning {
    int axis;
    float lo, k, ext;
    __device__ __forceinline__ void set(const Box &c) {
        const V3 e = sub(c.mx, c.mn);
        axis = 0;
        if (e.y > e.x) axis = 1;
        if (e.z > comp(e, axis)) axis = 2;
        ext = comp(e, axis);
        lo = comp(c.mn, axis);
        k = kBins / ext;
    }
    __device__ __forceinline__ int bin(V3 cen) const {
        const int b = (int)((comp(cen, axis) - lo) * k);
        return min(max(b, 0), kBins - 1);
    }
};

// Lane b holds bin b's box and count.  Returns the bin after which to split (the first of
// least cost), or -1 if none separates the triangles; `left` = the triangles up to it.
__device__ __forceinline__ int choose_split(const Box &bin, int count, int lane, int &left) {
    Box l = bin, r = bin;
    int lc = count, rc = count;
#pragma unroll
    for (int o = 1; o < kBins; o <<= 1) {
        const V3 a = mk(__shfl_up_sync(kFull, l.mn.x, o), __shfl_up_sync(kFull, l.mn.y, o), __shfl_up_sync(kFull, l.mn.z, o));
        const V3 b = mk(__shfl_up_sync(kFull, l.mx.x, o), __shfl_up_sync(kFull, l.mx.y, o), __shfl_up_sync(kFull, l.mx.z, o));
        const V3 c = mk(__shfl_down_sync(kFull, r.mn.x, o), __shfl_down_sync(kFull, r.mn.y, o), __shfl_down_sync(kFull, r.mn.z, o));
        const V3 d = mk(__shfl_down_sync(kFull, r.mx.x, o), __shfl_down_sync(kFull, r.mx.y, o), __shfl_down_sync(kFull, r.mx.z, o));
        const int n = __shfl_up_sync(kFull, lc, o), m = __shfl_down_sync(kFull, rc, o);
        if (lane >= o) { l.grow(a, b); lc += n; }
        if (lane + o < kBins) { r.grow(c, d); rc += m; }
    }
    const float ra = __shfl_down_sync(kFull, r.area(), 1);
    const int rn = __shfl_down_sync(kFull, rc, 1);
    float cost = FLT_MAX;
    if (lane < kBins - 1 && lc > 0 && rn > 0) cost = lc * l.area() + rn * ra;
    const int best = __reduce_min_sync(kFull, ord(cost));
    if (!(unord(best) < FLT_MAX)) return -1;
    const int b = __ffs(__ballot_sync(kFull, ord(cost) == best)) - 1;
    left = __shfl_sync(kFull, lc, b);
    return b;
}

__device__ __forceinline__ void write_node(float4 *out, int node, const Box &b, int code) {
    out[2 * (node + 1)] = make_float4(b.mn.x, b.mn.y, b.mn.z, __int_as_float(code));
    out[2 * (node + 1) + 1] = make_float4(b.mx.x, b.mx.y, b.mx.z, __int_as_float(0));
}

// Box of every sorted triangle slot as two float4 (one 32-byte sector), and the initial
// order: the slots' own, which is the Morton order.
__global__ void sah_boxes_kernel(int n, const int *perm, const float *bmin, const float *bmax, float4 *box, int *idx) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const size_t t = perm[s];
    box[2 * (size_t)s] = make_float4(bmin[3 * t], bmin[3 * t + 1], bmin[3 * t + 2], 0.0f);
    box[2 * (size_t)s + 1] = make_float4(bmax[3 * t], bmax[3 * t + 1], bmax[3 * t + 2], 0.0f);
    idx[s] = s;
}

__global__ void sah_root_kernel(int n, Task *large, int *n_large, Task *small, int *n_small) {
    const Task t{0, n, 0, 0};
    if (n > kSmall) { large[0] = t; *n_large = 1; } else { small[0] = t; *n_small = 1; }
}

// One block per node of more than kSmall triangles: its node record, its triangles
// partitioned into the other index buffer, and its children appended to the next level's
// list or to the small list.
__global__ void __launch_bounds__(kLargeThreads) sah_large_kernel(const float4 *box, int *idx0, int *idx1,
                                                                  const Task *tasks, const int *n_tasks, Task *next,
                                                                  int *n_next, Task *small, int *n_small, float4 *out) {
    constexpr int W = kLargeThreads / 32;
    __shared__ int red[W][12];
    __shared__ int bins[kBins][7];
    __shared__ int wcnt[W];
    __shared__ Binning s_bin;
    __shared__ int s_best, s_left;
    __shared__ Box s_box;
    if ((int)blockIdx.x >= *n_tasks) return;
    const Task t = tasks[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int depth = t.info & 255, lefts = (t.info >> 8) & 255, buf = t.info >> 16;
    const int *in = buf ? idx1 : idx0;
    int *to = buf ? idx0 : idx1;

    Box b, c;
    b.reset();
    c.reset();
    for (int i = t.begin + tid; i < t.end; i += kLargeThreads) {
        const size_t s = in[i];
        const float4 lo = box[2 * s], hi = box[2 * s + 1];
        const V3 m = centroid(lo, hi);
        b.grow(xyz(lo), xyz(hi));
        c.grow(m, m);
    }
    b.mn = warp_min(b.mn);
    b.mx = warp_max(b.mx);
    c.mn = warp_min(c.mn);
    c.mx = warp_max(c.mx);
    if (lane == 0) {
        const V3 v[4] = {b.mn, b.mx, c.mn, c.mx};
        for (int k = 0; k < 4; ++k) {
            red[w][3 * k] = ord(v[k].x);
            red[w][3 * k + 1] = ord(v[k].y);
            red[w][3 * k + 2] = ord(v[k].z);
        }
    }
    if (tid < kBins * 7) {
        const int f = tid % 7;
        bins[tid / 7][f] = f < 3 ? ord(FLT_MAX) : f < 6 ? ord(-FLT_MAX) : 0;
    }
    __syncthreads();
    if (w == 0) {   // lane = warp of the block
        auto get = [&](int k) { return mk(unord(red[lane][k]), unord(red[lane][k + 1]), unord(red[lane][k + 2])); };
        b.mn = warp_min(get(0));
        b.mx = warp_max(get(3));
        c.mn = warp_min(get(6));
        c.mx = warp_max(get(9));
        if (lane == 0) {
            s_box = b;
            s_bin.set(c);
            s_best = -1;
            s_left = (t.end - t.begin) / 2;
        }
    }
    __syncthreads();
    const Binning bn = s_bin;
    if (bn.ext > 0.0f && depth < kMedianDepth) {
        // consecutive positions are close along the Morton curve and fall into few bins: the
        // warp reduces bin by bin and one lane updates the block's bin
        for (int i0 = t.begin + 32 * w; i0 < t.end; i0 += kLargeThreads) {
            const int i = i0 + lane;
            int bin = -1;
            float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
            if (i < t.end) {
                const size_t s = in[i];
                lo = box[2 * s];
                hi = box[2 * s + 1];
                bin = bn.bin(centroid(lo, hi));
            }
            unsigned todo = __ballot_sync(kFull, bin >= 0);
            while (todo) {
                const int cur = __shfl_sync(kFull, bin, __ffs(todo) - 1);
                const bool mine = bin == cur;
                const unsigned group = __ballot_sync(kFull, mine);
                const int a0 = __reduce_min_sync(kFull, mine ? ord(lo.x) : INT_MAX);
                const int a1 = __reduce_min_sync(kFull, mine ? ord(lo.y) : INT_MAX);
                const int a2 = __reduce_min_sync(kFull, mine ? ord(lo.z) : INT_MAX);
                const int a3 = __reduce_max_sync(kFull, mine ? ord(hi.x) : INT_MIN);
                const int a4 = __reduce_max_sync(kFull, mine ? ord(hi.y) : INT_MIN);
                const int a5 = __reduce_max_sync(kFull, mine ? ord(hi.z) : INT_MIN);
                if (lane < 7) {
                    int *p = &bins[cur][lane];
                    const int v = lane == 0 ? a0 : lane == 1 ? a1 : lane == 2 ? a2 : lane == 3 ? a3 : lane == 4 ? a4 : a5;
                    if (lane < 3) atomicMin(p, v);
                    else if (lane < 6) atomicMax(p, v);
                    else atomicAdd(p, __popc(group));
                }
                todo &= ~group;
            }
        }
        __syncthreads();
        if (w == 0) {
            Box bb;
            bb.mn = mk(unord(bins[lane][0]), unord(bins[lane][1]), unord(bins[lane][2]));
            bb.mx = mk(unord(bins[lane][3]), unord(bins[lane][4]), unord(bins[lane][5]));
            int left = 0;
            const int best = choose_split(bb, bins[lane][6], lane, left);
            if (lane == 0 && best >= 0) { s_best = best; s_left = left; }
        }
        __syncthreads();
    }
    const int best = s_best, mid = t.begin + s_left;
    int lrun = t.begin, rrun = mid;   // next free left and right position
    for (int i0 = t.begin; i0 < t.end; i0 += kLargeThreads) {
        const int i = i0 + tid;
        int s = 0;
        bool left = false;
        if (i < t.end) {
            s = in[i];
            left = best >= 0 ? bn.bin(centroid(box[2 * (size_t)s], box[2 * (size_t)s + 1])) <= best : i < mid;
        }
        const unsigned m = __ballot_sync(kFull, left);
        if (lane == 0) wcnt[w] = __popc(m);
        __syncthreads();
        const int mine = wcnt[lane];
        const int before = __reduce_add_sync(kFull, lane < w ? mine : 0);
        const int total = __reduce_add_sync(kFull, mine);
        const int lrank = before + __popc(m & ((1u << lane) - 1u));
        if (i < t.end) to[left ? lrun + lrank : rrun + (tid - lrank)] = s;
        lrun += total;
        rrun += min(kLargeThreads, t.end - i0) - total;
        __syncthreads();
    }
    if (tid == 0) {
        const int child = 1 + 2 * (t.begin + lefts);
        write_node(out, t.node, s_box, child);
        for (int k = 0; k < 2; ++k) {
            Task n;
            n.begin = k ? mid : t.begin;
            n.end = k ? t.end : mid;
            n.node = child + k;
            n.info = (depth + 1) | (lefts + (k ? 0 : 1)) << 8 | (buf ^ 1) << 16;
            if (n.end - n.begin > kSmall) next[atomicAdd(n_next, 1)] = n;
            else small[atomicAdd(n_small, 1)] = n;
        }
    }
}

// One warp per subtree of at most kSmall triangles.
struct SmallMem {
    float4 box[2 * kSmall];
    int slot[kSmall];
    uint8_t order[2][kSmall];   // local triangles in position order, and the partition's target
    Task stack[64];             // pending right children, positions relative to the subtree's
};

__global__ void __launch_bounds__(32 * kSmallWarps) sah_small_kernel(const float4 *box, const int *idx0, const int *idx1,
                                                                     const Task *tasks, const int *n_tasks, float4 *out,
                                                                     int *max_depth) {
    __shared__ SmallMem mem[kSmallWarps];
    static_assert(kSmall <= 256, "order holds bytes");
    const int lane = threadIdx.x & 31;
    SmallMem &m = mem[threadIdx.x >> 5];
    const int total = *n_tasks, step = gridDim.x * kSmallWarps;
    for (int k = blockIdx.x * kSmallWarps + (threadIdx.x >> 5); k < total; k += step) {
        const Task t = tasks[k];
        const int *in = t.info >> 16 ? idx1 : idx0;
        const int n = t.end - t.begin;
        for (int i = lane; i < n; i += 32) {
            const int s = in[t.begin + i];
            m.slot[i] = s;
            m.box[2 * i] = box[2 * (size_t)s];
            m.box[2 * i + 1] = box[2 * (size_t)s + 1];
            m.order[0][i] = (uint8_t)i;
        }
        __syncwarp();
        int begin = 0, end = n, node = t.node, depth = t.info & 255, lefts = (t.info >> 8) & 255, top = 0;
        int deepest = depth;
        for (;;) {
            const int cnt = end - begin;
            Box b, c;
            b.reset();
            c.reset();
            for (int i = begin + lane; i < end; i += 32) {
                const int q = m.order[0][i];
                const float4 lo = m.box[2 * q], hi = m.box[2 * q + 1];
                const V3 ce = centroid(lo, hi);
                b.grow(xyz(lo), xyz(hi));
                c.grow(ce, ce);
            }
            b.mn = warp_min(b.mn);
            b.mx = warp_max(b.mx);
            if (cnt == 1) {
                deepest = max(deepest, depth);
                if (lane == 0) write_node(out, node, b, -1 - m.slot[m.order[0][begin]]);
                if (top == 0) break;
                const Task e = m.stack[--top];
                __syncwarp();
                begin = e.begin;
                end = e.end;
                node = e.node;
                depth = e.info & 255;
                lefts = e.info >> 8;
                continue;
            }
            c.mn = warp_min(c.mn);
            c.mx = warp_max(c.mx);
            Binning bn;
            bn.set(c);
            int best = -1, left = cnt / 2;
            if (bn.ext > 0.0f && depth < kMedianDepth) {
                Box bb;   // this lane's bin
                bb.reset();
                int bc = 0;
                for (int i = begin; i < end; ++i) {
                    const int q = m.order[0][i];
                    const float4 lo = m.box[2 * q], hi = m.box[2 * q + 1];
                    if (bn.bin(centroid(lo, hi)) == lane) {
                        bb.grow(xyz(lo), xyz(hi));
                        ++bc;
                    }
                }
                int nl = 0;
                best = choose_split(bb, bc, lane, nl);
                if (best >= 0) left = nl;
            }
            if (best >= 0) {   // stable partition (a median split keeps the order)
                int lrun = begin, rrun = begin + left;
                for (int i0 = begin; i0 < end; i0 += 32) {
                    const int i = i0 + lane;
                    int q = 0;
                    bool l = false;
                    if (i < end) {
                        q = m.order[0][i];
                        l = bn.bin(centroid(m.box[2 * q], m.box[2 * q + 1])) <= best;
                    }
                    const unsigned lm = __ballot_sync(kFull, l);
                    const int lrank = __popc(lm & ((1u << lane) - 1u));
                    if (i < end) m.order[1][l ? lrun + lrank : rrun + (lane - lrank)] = (uint8_t)q;
                    lrun += __popc(lm);
                    rrun += min(32, end - i0) - __popc(lm);
                }
                __syncwarp();
                for (int i = begin + lane; i < end; i += 32) m.order[0][i] = m.order[1][i];
                __syncwarp();
            }
            const int child = 1 + 2 * (t.begin + begin + lefts);
            if (lane == 0) {
                write_node(out, node, b, child);
                m.stack[top] = Task{begin + left, end, child + 1, (depth + 1) | lefts << 8};
            }
            __syncwarp();
            ++top;
            end = begin + left;
            node = child;
            ++depth;
            ++lefts;
        }
        if (lane == 0) atomicMax(max_depth, deepest);
        __syncwarp();
    }
}

// The closest-hit tree: the any-hit tree's nodes with inflated boxes, so that a ray which passes
// a triangle's test at distance t (tri_hit: floats, Cramer's rule, |denom| >= 1e-6) never enters
// a box around that triangle later than at t as box_hit_fast computes it.  With u = 2^-24,
// P = |e1| |e2|, A = |e1 x e2|, J = p0 - o and D the largest distance of a covered origin from a
// vertex:
//   - a cross product is within 2.42 u of its factors' lengths (two products, one difference per
//     component), a dot product with it within 3 u more: the determinants are within 5.42 u P,
//     5.42 u |J| |e2|, 5.42 u |J| |e1| and 5.42 u P |J| of their exact values;
//   - so t, beta |e1| and gamma |e2| are together within 21.7 u P (D + E) / |denom| of the exact
//     solution's, E the longest edge, while 5.42 u P is at most 0.01 |denom|; with beta and gamma
//     in [0, 1] the point o + t d lies within 22.5 u P (D + E) / |denom| of the triangle;
//   - off the triangle's plane it is far closer: only t's error leaves the plane, by its part
//     along the normal, which takes the grazing angle out of denom: 5.42 u P (2 D + E) / (0.98 A);
//   - on an axis-aligned triangle the edges' components along the normal are exactly zero, so
//     denom, the numerator of t and, with K = t d_n, those of beta and gamma all carry the factor
//     d_n (the direction's component along the normal) and their errors are relative to it: at
//     most 4 u P |d_n|, 9 u |J| |e2| |d_n| and so on, over A |d_n|, whatever the angle: the point
//     lies within u (P / A) (25 D + 12 E) of the triangle;
//   - the slab test places a plane within 4 u (|plane| + |origin|) of where it is, and where it
//     replaces a component below 1e-6 by 1e-6 it moves the point at t by at most 2e-6 t.
// A triangle that a bound says nothing about gets a box that every ray enters at once.
struct Inflate {
    float D, pad;   // largest |p0 - o|; rounding of planes and of p0 - o, replaced components
    __device__ __forceinline__ V3 by(float4 a, float4 b, float4 c) const {
        const V3 e1 = mk(a.w, b.x, b.y), e2 = mk(b.z, b.w, c.x);
        const float l1 = len(e1), l2 = len(e2), P = l1 * l2, E = fmaxf(l1, l2);
        constexpr float u = 5.9604645e-8f, kRound = 1.05f;   // kRound: this arithmetic's own rounding
        const V3 x = cross(e1, e2);
        const float A = len(x);
        const bool thin = !(A > 1e-3f * P);   // the normal is not known well enough
        const bool aligned = (e1.x == 0.0f && e2.x == 0.0f) || (e1.y == 0.0f && e2.y == 0.0f) ||
                             (e1.z == 0.0f && e2.z == 0.0f);
        if (aligned && !thin) {
            const float r = kRound * u * (P / A) * (25.0f * D + 12.0f * E) + pad;
            return mk(r, r, r);
        }
        const float denom = 0.999e-6f;
        if (!(5.42f * u * P * kRound <= 0.01f * denom)) return mk(1e30f, 1e30f, 1e30f);
        const float in_plane = kRound * 22.5f * u * P * (D + E) / denom;
        if (thin) return mk(in_plane + pad, in_plane + pad, in_plane + pad);
        const float off = kRound * 5.6f * u * P * (2.0f * D + E) / A + pad;
        // the share of an in-plane distance along an axis, from the normal's lean towards it
        auto along = [&](float xi) {
            const float ni = 0.999f * fabsf(xi) / A;
            return in_plane * sqrtf(fmaxf(1.0f - ni * ni, 0.0f)) + off;
        };
        return mk(along(x.x), along(x.y), along(x.z));
    }
};

// Leaves' inflated boxes and every node's parent.  A node index or slot out of range (a saved
// tree that was damaged) is passed over.
__global__ void closest_leaves_kernel(int n, const float4 *trav, const float4 *tri_isect, Inflate inf, float4 *ctrav,
                                      int *parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * n - 1) return;
    const float4 lo = trav[2 * (i + 1)], hi = trav[2 * (i + 1) + 1];
    const int code = __float_as_int(lo.w);
    if (code >= 0) {
        if (code >= 1 && code + 1 < 2 * n - 1) parent[code] = parent[code + 1] = i;
        return;
    }
    if (-1 - code >= n) return;
    const float4 *t = tri_isect + 3 * (size_t)(-1 - code);
    Box b;
    b.mn = xyz(lo);
    b.mx = xyz(hi);
    const V3 by = inf.by(t[0], t[1], t[2]);
    b.mn = sub(b.mn, by);
    b.mx = add(b.mx, by);
    write_node(ctrav, i, b, code);
}

// Inner boxes bottom-up: the thread that comes second to a node unites its children and goes on.
// cost[0], cost[1]: expected visits of a random ray's walk, exact and inflated (box areas over
// the root's).
__global__ void __launch_bounds__(256) closest_refit_kernel(int n, const float4 *trav, float4 *ctrav, const int *parent,
                                                            int *count, double *cost) {
    __shared__ float red[8][2];
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    Box root;
    root.mn = xyz(trav[2]);
    root.mx = xyz(trav[3]);
    const float whole = fmaxf(root.area(), 1e-30f);
    float exact = 0.0f, inflated = 0.0f;
    if (i0 < 2 * n - 1 && __float_as_int(trav[2 * (i0 + 1)].w) < 0) {
        int i = i0;
        Box b;
        b.mn = xyz(ctrav[2 * (i + 1)]);
        b.mx = xyz(ctrav[2 * (i + 1) + 1]);
        for (;;) {
            Box own;
            own.mn = xyz(trav[2 * (i + 1)]);
            own.mx = xyz(trav[2 * (i + 1) + 1]);
            exact += fminf(own.area() / whole, 1.0f);
            inflated += fminf(b.area() / whole, 1.0f);
            const int p = i > 0 ? parent[i] : -1;
            if (p < 0) break;
            __threadfence();   // this node's box before the count
            if (atomicAdd(count + p, 1) != 1) break;
            __threadfence();
            const int other = ((i - 1) ^ 1) + 1;
            b.grow(xyz(__ldcg(ctrav + 2 * (other + 1))), xyz(__ldcg(ctrav + 2 * (other + 1) + 1)));
            write_node(ctrav, p, b, __float_as_int(trav[2 * (p + 1)].w));
            i = p;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        exact += __shfl_xor_sync(kFull, exact, o);
        inflated += __shfl_xor_sync(kFull, inflated, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5][0] = exact;
        red[threadIdx.x >> 5][1] = inflated;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double sum = 0.0;
        for (int w = 0; w < 8; ++w) sum += red[w][threadIdx.x];
        atomicAdd(cost + threadIdx.x, sum);
    }
}

}  // namespace

// The 8-wide any-hit tree of the packet gathers: every inner node at a depth divisible by three
// becomes a node of up to eight entries, its descendants three levels down (or the leaves above).
// Entry = {box min, code}, {box max, -}: code = a wide node's index, -1 - sorted triangle slot, or
// kWideEmpty.  A parent or child index out of range (a saved tree that was damaged) is passed over.
__global__ void wide8_parent_kernel(int nn, const float4 *tree, int *parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const int c = __float_as_int(tree[2 * (i + 1)].w);
    if (c >= 1 && c + 1 < nn) parent[c] = parent[c + 1] = i;
}

__global__ void wide8_flag_kernel(int nn, const float4 *tree, const int *parent, int *flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    int depth = 0;
    for (int k = i; k > 0 && depth < 4 * STACK_CAP; ++depth) k = parent[k];
    flag[i] = i == 0 || (__float_as_int(tree[2 * (i + 1)].w) >= 0 && depth % 3 == 0) ? 1 : 0;
}

__global__ void wide8_fill_kernel(int nn, const float4 *tree, const int *flag, const int *index, float4 *wide) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn || !flag[i]) return;
    int node[8] = {i}, count = 1;
    for (int round = 0; round < 3; ++round) {
        int next[8], m = 0;
        for (int k = 0; k < count; ++k) {
            const int c = __float_as_int(tree[2 * (node[k] + 1)].w);
            if (c >= 1 && c + 1 < nn) {
                next[m++] = c;
                next[m++] = c + 1;
            } else {
                next[m++] = node[k];
            }
        }
        count = m;
        for (int k = 0; k < m; ++k) node[k] = next[k];
    }
    float4 *rec = wide + 16 * (size_t)index[i];
    for (int k = 0; k < 8; ++k) {
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(kWideEmpty)), hi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k < count) {
            lo = tree[2 * (node[k] + 1)];
            hi = tree[2 * (node[k] + 1) + 1];
            hi.w = 0.0f;
            if (__float_as_int(lo.w) >= 0) lo.w = __int_as_float(index[node[k]]);
        }
        rec[2 * k] = lo;
        rec[2 * k + 1] = hi;
    }
}

static rzk_status drop_closest_tree(rzk_scene *s) {
    if (s->d_ctrav) {
        cudaFree(s->d_ctrav);
        s->d_ctrav = nullptr;
        s->device_bytes -= s->ctrav_bytes;
        s->ctrav_bytes = 0;
    }
    return RZK_OK;
}

// Makes the closest-hit tree from the any-hit tree (on a fresh build and on a restored scene);
// leaves the scene without one where closest hits are better off in the reference's order: no
// any-hit tree, few triangles (36: 740 us for 4 M rays in the reference's order, 880 in this
// one; 3,012: 1,420 and 1,060), a reference tree near the traversal stack's depth (whose dropped
// pushes are part of its answer), coordinates the bound cannot handle, no memory for it, or boxes
// inflated so far (large slanted triangles, or a scene in large units) that a ray would visit
// kMaxInflation times as many nodes (the rooms here: 1.00 to 1.15 times).
rzk_status build_closest_tree(rzk_scene *s, cudaStream_t st) {
    constexpr double kMaxInflation = 2.5;
    constexpr int kMinTris = 128;
    const int n = s->n_tris;
    float ext = 0.0f, top = 0.0f, diag2 = 0.0f, c[3];
    for (int d = 0; d < 3; ++d) {
        const float e = s->box[3 + d] - s->box[d];
        c[d] = 0.5f * (s->box[d] + s->box[3 + d]);
        ext = std::max(ext, e);
        diag2 += e * e;
        top = std::max(top, std::max(std::fabs(s->box[d]), std::fabs(s->box[3 + d])));
    }
    const bool wanted = n >= kMinTris && s->d_trav && s->n_levels <= STACK_CAP - 4 && ext > 1e-6f && top < 1e6f;
    if (wanted) {
        const size_t bytes = sizeof(float4) * 4 * (size_t)n;
        if (s->d_ctrav && s->ctrav_bytes != bytes) {
            cudaFree(s->d_ctrav);
            s->d_ctrav = nullptr;
            s->device_bytes -= s->ctrav_bytes;
        }
        const size_t nn = 2 * (size_t)n - 1;
        CallScratch mem;   // first: without it the scene must not be left with a tree that is not filled
        cudaError_t e = mem.alloc(2 * sizeof(double) + 2 * sizeof(int) * nn, st);
        const bool make = e == cudaSuccess && !s->d_ctrav;
        if (make) e = cudaMalloc((void **)&s->d_ctrav, bytes);
        if (e == cudaErrorMemoryAllocation) {   // a scene that fits without the tree does without it
            (void)cudaGetLastError();
            if (make) s->d_ctrav = nullptr;
            return drop_closest_tree(s);
        }
        RZK_CUDA_TRY(e);
        if (make) {
            s->ctrav_bytes = bytes;
            s->device_bytes += bytes;
            // slot 0; the kernels write every node (not cleared on a rebuild: queries may be reading)
            RZK_CUDA_TRY(cudaMemsetAsync(s->d_ctrav, 0, 2 * sizeof(float4), st));
        }
        const float radius = 2.0f * ext;   // the covered origins: a sphere about the scene's centre
        Inflate inf;
        inf.D = 1.01f * (radius + 0.5f * std::sqrt(diag2));
        inf.pad = 1e-6f * (top + radius) + 6e-6f * inf.D;
        for (int d = 0; d < 3; ++d) s->cguard[d] = c[d];
        s->cguard[3] = radius * radius;
        double *cost = (double *)mem.get();
        int *count = (int *)(cost + 2), *parent = count + nn;
        RZK_CUDA_TRY(cudaMemsetAsync(cost, 0, 2 * sizeof(double) + sizeof(int) * nn, st));
        RZK_CUDA_TRY(cudaMemsetAsync(parent, 0xff, sizeof(int) * nn, st));
        const unsigned grid = (unsigned)((nn + 255) / 256);
        closest_leaves_kernel<<<grid, 256, 0, st>>>(n, s->d_trav, s->d_tri_isect, inf, s->d_ctrav, parent);
        closest_refit_kernel<<<grid, 256, 0, st>>>(n, s->d_trav, s->d_ctrav, parent, count, cost);
        RZK_CUDA_TRY(cudaGetLastError());
        double h[2];
        RZK_CUDA_TRY(cudaMemcpyAsync(h, cost, sizeof(h), cudaMemcpyDeviceToHost, st));
        mem.release();
        RZK_CUDA_TRY(cudaStreamSynchronize(st));
        if (h[1] <= kMaxInflation * h[0]) return RZK_OK;
    }
    return drop_closest_tree(s);
}

// Makes the packet gathers' 8-wide tree from the any-hit tree (from the reference's where there is
// none), on a fresh build and on a restored scene.
rzk_status build_wide_tree(rzk_scene *s, cudaStream_t st) {
    const int nn = s->d_trav ? 2 * s->n_tris - 1 : s->n_nodes;
    if (nn <= 0) return RZK_OK;
    const float4 *tree = s->d_trav ? s->d_trav : s->d_nodes;
    CallScratch mem;
    const size_t scan_bytes = exclusive_scan_tmp_bytes(nn);
    RZK_CUDA_TRY(mem.alloc(sizeof(int) * (3 * (size_t)nn + 64) + scan_bytes, st));
    int *total = (int *)mem.get(), *parent = total + 64, *flag = parent + nn, *index = flag + nn;
    const unsigned grid = (unsigned)((nn + 255) / 256);
    RZK_CUDA_TRY(cudaMemsetAsync(parent, 0, sizeof(int) * (size_t)nn, st));
    wide8_parent_kernel<<<grid, 256, 0, st>>>(nn, tree, parent);
    wide8_flag_kernel<<<grid, 256, 0, st>>>(nn, tree, parent, flag);
    RZK_CUDA_TRY(cudaGetLastError());
    RZK_TRY(exclusive_scan_i32(flag, index, nn, total, index + nn, scan_bytes, st));
    int n = 0;
    RZK_CUDA_TRY(cudaMemcpyAsync(&n, total, sizeof(int), cudaMemcpyDeviceToHost, st));
    RZK_CUDA_TRY(cudaStreamSynchronize(st));
    if (s->n_wide8 < n) {
        if (s->d_wide8) {
            cudaFree(s->d_wide8);
            s->device_bytes -= 16 * sizeof(float4) * (size_t)s->n_wide8;
        }
        s->d_wide8 = nullptr;
        s->n_wide8 = 0;
        RZK_CUDA_TRY(cudaMalloc((void **)&s->d_wide8, 16 * sizeof(float4) * (size_t)n));
        s->n_wide8 = n;
        s->device_bytes += 16 * sizeof(float4) * (size_t)n;
    }
    wide8_fill_kernel<<<grid, 256, 0, st>>>(nn, tree, flag, index, s->d_wide8);
    RZK_CUDA_TRY(cudaGetLastError());
    mem.release();
    RZK_CUDA_TRY(cudaStreamSynchronize(st));
    return RZK_OK;
}

rzk_status build_sah_tree(rzk_scene *s, cudaStream_t st) {
    const int n = s->n_tris;
    if (n <= 0) return RZK_OK;
    const size_t bytes = sizeof(float4) * 4 * (size_t)n;   // 2n - 1 nodes and the unused slot 0
    if (s->d_trav && s->trav_bytes != bytes) {
        cudaFree(s->d_trav);
        s->d_trav = nullptr;
        s->device_bytes -= s->trav_bytes;
    }
    if (!s->d_trav) {
        s->trav_bytes = 0;
        RZK_CUDA_TRY(cudaMalloc((void **)&s->d_trav, bytes));
        s->trav_bytes = bytes;
        s->device_bytes += bytes;
    }
    // nodes of one level are disjoint ranges of more than kSmall triangles; every small node
    // holds at least one triangle of its own
    const int max_large = n / (kSmall + 1) + 1;
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t o_idx0 = up(2 * sizeof(float4) * (size_t)n), o_idx1 = o_idx0 + up(sizeof(int) * (size_t)n);
    const size_t o_small = o_idx1 + up(sizeof(int) * (size_t)n), o_l0 = o_small + up(sizeof(Task) * (size_t)n);
    const size_t o_l1 = o_l0 + up(sizeof(Task) * (size_t)max_large), o_cnt = o_l1 + up(sizeof(Task) * (size_t)max_large);
    CallScratch mem;
    RZK_CUDA_TRY(mem.alloc(o_cnt + sizeof(int) * (kMaxLevels + 3), st));
    char *buf = mem.get();
    float4 *box = (float4 *)buf;
    int *idx0 = (int *)(buf + o_idx0), *idx1 = (int *)(buf + o_idx1);
    Task *small = (Task *)(buf + o_small), *large[2] = {(Task *)(buf + o_l0), (Task *)(buf + o_l1)};
    int *n_small = (int *)(buf + o_cnt), *max_depth = n_small + 1,
        *n_large = n_small + 2;   // n_large[level]
    RZK_CUDA_TRY(cudaMemsetAsync(n_small, 0, sizeof(int) * (kMaxLevels + 3), st));
    RZK_CUDA_TRY(cudaMemsetAsync(s->d_trav, 0, 2 * sizeof(float4), st));
    sah_boxes_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, s->d_perm, s->d_bmin, s->d_bmax, box, idx0);
    sah_root_kernel<<<1, 1, 0, st>>>(n, large[0], n_large, small, n_small);
    RZK_CUDA_TRY(cudaGetLastError());
    int pending = n > kSmall ? 1 : 0;
    for (int level = 0; pending && level < kMaxLevels; ++level) {
        const int grid = level < 30 ? std::min(max_large, 1 << level) : max_large;
        sah_large_kernel<<<grid, kLargeThreads, 0, st>>>(box, idx0, idx1, large[level & 1], n_large + level,
                                                         large[(level + 1) & 1], n_large + level + 1, small, n_small,
                                                         s->d_trav);
        RZK_CUDA_TRY(cudaGetLastError());
        // a level has nodes only if the one before it had: look once in four levels, the first
        // time when an even split would be done
        if ((level & 3) == 3 && (level >= 23 || (kSmall << level) >= n)) {   // past 2^30: any n
            RZK_CUDA_TRY(cudaMemcpyAsync(&pending, n_large + level + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
            RZK_CUDA_TRY(cudaStreamSynchronize(st));
        }
    }
    sah_small_kernel<<<(n + 128 * kSmallWarps - 1) / (128 * kSmallWarps), 32 * kSmallWarps, 0, st>>>(
        box, idx0, idx1, small, n_small, s->d_trav, max_depth);
    RZK_CUDA_TRY(cudaGetLastError());
    RZK_CUDA_TRY(cudaMemcpyAsync(&s->trav_depth, max_depth, sizeof(int), cudaMemcpyDeviceToHost, st));
    mem.release();
    RZK_CUDA_TRY(cudaStreamSynchronize(st));
    return s->trav_depth >= STACK_CAP - 2 ? RZK_ERR_STACK : RZK_OK;
}

}  // namespace rzk
