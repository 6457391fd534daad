// rzk_trace.cu - batched visibility and closest-hit queries (the Aggregate interface).
#include "rzk_traverse.cuh"

#include <algorithm>

namespace rzk {

namespace {

constexpr int kTraceBlock = 128;

// A query's traversal stack has as many entries as the tree walked is deep, so that it does not
// limit the resident warps (64 entries: 24 per SM; 200,000 rays on 30k triangles 167 and 156 us).
// Large batches in large scenes keep their lanes busy by refilling them: a warp owns a run of
// rays, and when kRefill of its lanes have finished theirs they take the next ones together,
// while the others go on.  One ray per thread left 6.7 (closest) and 8.4 (any hit) of 32 lanes
// active on average there, each warp waiting for its longest ray.
constexpr int kRefill = 8;

struct RayRun {   // the warp's rays [next, end)
    int next, end;
    __device__ __forceinline__ RayRun(int n, int per_warp) {
        const long long w = ((long long)blockIdx.x * kTraceBlock + threadIdx.x) >> 5;
        next = (int)min((long long)n, w * per_warp);
        end = (int)min((long long)n, w * per_warp + per_warp);
    }
    // hands the idle lanes (idx < 0) their next rays' indices; false when the run is over
    __device__ __forceinline__ bool refill(int &idx, int lane) {
        const unsigned idle = __ballot_sync(0xffffffffu, idx < 0);
        if (idle == 0xffffffffu && next >= end) return false;
        if (next < end && (__popc(idle) >= kRefill)) {
            const int k = next + __popc(idle & ((1u << lane) - 1u));
            if (idx < 0 && k < end) idx = k;
            next += __popc(idle);
        }
        return true;
    }
};

// Aggregate::hit(p, q, tmin, time) (aggregate.cc:84-90): Ray(p, q - p) over
// [tmin, |q - p| - tmin].
__global__ void __launch_bounds__(kTraceBlock) occluded_kernel(DevScene s, const float *p, const float *q, int n,
                                                               int per_warp, int cap, uint8_t *out) {
    extern __shared__ int stack_mem[];
    const int lane = threadIdx.x & 31;
    RayRun run(n, per_warp);
    AnyHitWalk<kTraceBlock> walk;
    walk.stk.init(stack_mem + threadIdx.x, cap);
    int idx = -1;
    for (;;) {
        const int was = idx;
        if (!run.refill(idx, lane)) break;
        if (idx != was) {
            const V3 a = ld3(p + 3 * (size_t)idx), b = ld3(q + 3 * (size_t)idx);
            walk.start(s, make_ray(a, sub(b, a)), s.tmin, len(sub(b, a)) - s.tmin);
        }
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            if (idx < 0) break;
            if (walk.step(s)) {
                out[idx] = walk.hit ? 1 : 0;
                idx = -1;
            }
        }
    }
}

__global__ void __launch_bounds__(kTraceBlock) occluded_plain_kernel(GatherScene s, const float *p, const float *q,
                                                                     int n, int cap, uint8_t *out) {
    extern __shared__ int stack_mem[];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Stack<kTraceBlock> stk;
    stk.init(stack_mem + threadIdx.x, cap);
    const V3 a = ld3(p + 3 * (size_t)i), b = ld3(q + 3 * (size_t)i);
    const Ray r = make_ray(a, sub(b, a));
    out[i] = any_hit<kTraceBlock, false, true>(s, r, s.tmin, len(sub(b, a)) - s.tmin, stk) ? 1 : 0;
}

// TREE: the scene has a closest-hit tree; otherwise cap is STACK_CAP.
template <bool TREE>
__global__ void __launch_bounds__(kTraceBlock) closest_plain_kernel(DevScene s, const float *o, const float *d, int n,
                                                                    int cap, float *t_out, rzk_receiver *recv) {
    extern __shared__ int stack_mem[];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Ray r = make_ray(ld3(o + 3 * (size_t)i), ld3(d + 3 * (size_t)i));
    float t = RAY_TMAX, b = 0.0f, g = 0.0f;
    int slot = -1;
    if (TREE) {
        ClosestWalk<kTraceBlock> walk;
        walk.stk.init(stack_mem + threadIdx.x, cap);
        walk.start(s, r, s.tmin, RAY_TMAX);
        while (!walk.step(s)) {}
        int mem[STACK_CAP];   // rarely needed: local memory
        slot = walk.template finish<1>(s, mem);
        t = walk.bt; b = walk.bb; g = walk.bg;
    } else if (s.n_nodes > 0) {
        const ClosestHit c =
            closest_in_order<kTraceBlock>(s.nodes, s.tri_isect, s.err, r, s.tmin, RAY_TMAX, stack_mem + threadIdx.x);
        slot = c.slot; t = c.t; b = c.beta; g = c.gamma;
    }
    if (t_out) t_out[i] = slot < 0 ? -1.0f : t;
    if (!recv) return;
    if (slot < 0) {
        write_miss(recv + i);
        return;
    }
    HitGeo h;
    fill_hit(s, r, slot, t, b, g, h);
    write_receiver(h, r, recv + i);
}

__global__ void __launch_bounds__(kTraceBlock) closest_kernel(DevScene s, const float *o, const float *d, int n,
                                                              int per_warp, int cap, float *t_out,
                                                              rzk_receiver *recv) {
    extern __shared__ int stack_mem[];
    const int lane = threadIdx.x & 31;
    RayRun run(n, per_warp);
    ClosestWalk<kTraceBlock> walk;
    walk.stk.init(stack_mem + threadIdx.x, cap);
    int idx = -1, done = -1;   // done: a finished ray whose result is not written yet
    for (;;) {
        const int was = idx;
        const bool more = run.refill(idx, lane);
        if (done >= 0 && (!more || idx != was)) {
            int mem[STACK_CAP];   // rarely needed: local memory
            const int slot = walk.template finish<1>(s, mem);
            if (t_out) t_out[done] = slot < 0 ? -1.0f : walk.bt;
            if (recv && slot < 0) {
                write_miss(recv + done);
            } else if (recv) {
                HitGeo h;
                fill_hit(s, walk.r, slot, walk.bt, walk.bb, walk.bg, h);
                write_receiver(h, walk.r, recv + done);
            }
            done = -1;
        }
        if (!more) break;
        if (idx != was)
            walk.start(s, make_ray(ld3(o + 3 * (size_t)idx), ld3(d + 3 * (size_t)idx)), s.tmin, RAY_TMAX);
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            if (idx < 0) break;
            if (walk.step(s)) {
                done = idx;
                idx = -1;
            }
        }
    }
}

// Queries on rays the caller constructed (the reference's Ray fields, its own interval):
// the caller's ray is used as stored.  Any-hit walks the any-hit tree (same answer, see
// rzk_sah.cu); closest-hit walks the reference tree in the reference's visit order, which
// decides ties.
__global__ void __launch_bounds__(kTraceBlock) ray_query_kernel(DevScene s, const int *perm, const rzk_ray *rays,
                                                                int n, int closest, rzk_ray_hit *out) {
    __shared__ int stack_mem[STACK_CAP * kTraceBlock];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Stack<kTraceBlock> stk;
    stk.init(stack_mem + threadIdx.x);
    const rzk_ray &q = rays[i];
    Ray r;
    r.o = ld3(q.o);
    r.d = ld3(q.d);
    r.inv_d = ld3(q.inv_d);
    r.org_inv_d = ld3(q.org_inv_d);
    rzk_ray_hit h{0, 0.0f, 0.0f, 0.0f, -1, {0, 0, 0}};
    if (closest) {
        if (s.n_nodes > 0) {
            const ClosestHit c = closest_in_order<kTraceBlock>(s.nodes, s.tri_isect, s.err, r, q.tmin, q.tmax, stk.base);
            if (c.slot >= 0) {
                h.hit = 1;
                h.t = c.t;
                h.beta = c.beta;
                h.gamma = c.gamma;
                h.tri = perm[c.slot];
            }
        }
    } else {
        h.hit = any_hit<kTraceBlock, false, true, false>(s, r, q.tmin, q.tmax, stk) ? 1 : 0;
    }
    out[i] = h;
}

// One thread per pixel; a block covers an 16 x 8 pixel tile so that a warp's primary
// rays are spatially coherent.
__global__ void __launch_bounds__(kTraceBlock) primary_kernel(DevScene s, rzk_camera cam,
                                                              rzk_receiver *out) {
    __shared__ int stack_mem[STACK_CAP * kTraceBlock];
    int j = blockIdx.x * 16 + (threadIdx.x & 15);
    int i = blockIdx.y * 8 + (threadIdx.x >> 4);
    if (i >= cam.height || j >= cam.width) return;
    Stack<kTraceBlock> stk;
    stk.init(stack_mem + threadIdx.x);
    Ray r = camera_ray(cam, i, j);
    float t, b, g;
    rzk_receiver *o = out + (size_t)i * cam.width + j;
    int slot = closest_hit<kTraceBlock>(s, r, s.tmin, RAY_TMAX, stk, &t, &b, &g);
    if (slot < 0) { write_miss(o); return; }
    HitGeo h;
    fill_hit(s, r, slot, t, b, g, h);
    write_receiver(h, r, o);
}

}  // namespace

static int stack_entries(int depth) { return std::max(2, std::min(STACK_CAP, depth + 1)); }

// Refilling pays where a walk is long and a lane has several rays to do; elsewhere the longest
// ray's steps are the time and the extra work of a step only adds to them.  us on B200, one ray
// per thread and refilled: 300k triangles 524,288 rays 586 and 515, segments 374 and 342, 200,000
// rays 286 and 288, segments 203 and 212, 5,000 rays 129 and 142; 105k triangles 1,000,003 rays
// 686 and 655, 524,288 390 and 378; 30k triangles 1,000,003 rays 463 and 478; 36 triangles
// 400,000 segments 31 and 45.
constexpr int kRefillRays = 384 << 10, kRefillTris = 64 << 10;

// Grid of a refilling kernel: a run of whole warps' worth of rays per resident warp, at most
// kMaxRun.
struct RunGrid {
    unsigned blocks;
    int per_warp, cap;
    size_t smem;
};
template <class K>
static cudaError_t run_grid(K kernel, int n, int depth, RunGrid &g) {
    constexpr int kMaxRun = 512;
    g.cap = stack_entries(depth);
    g.smem = sizeof(int) * kTraceBlock * (size_t)g.cap;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTraceBlock, g.smem);
    if (e != cudaSuccess) return e;
    const long long warps = (long long)sms * std::max(1, per_sm) * (kTraceBlock / 32);
    g.per_warp = (int)std::min<long long>(kMaxRun, ((n + warps - 1) / warps + 31) / 32 * 32);
    const long long runs = ((long long)n + g.per_warp - 1) / g.per_warp;
    g.blocks = (unsigned)((runs + kTraceBlock / 32 - 1) / (kTraceBlock / 32));
    return cudaSuccess;
}

rzk_status launch_occluded(const DevScene &s, int depth, const float *p, const float *q, int n, uint8_t *out,
                           cudaStream_t st) {
    if (n <= 0) return RZK_OK;
    if (n < kRefillRays || s.n_tris < kRefillTris) {
        const int cap = stack_entries(depth);
        occluded_plain_kernel<<<(n + kTraceBlock - 1) / kTraceBlock, kTraceBlock, sizeof(int) * kTraceBlock * cap, st>>>(
            s, p, q, n, cap, out);
        RZK_CUDA_TRY(cudaGetLastError());
        return RZK_OK;
    }
    RunGrid g;
    RZK_CUDA_TRY(run_grid(occluded_kernel, n, depth, g));
    occluded_kernel<<<g.blocks, kTraceBlock, g.smem, st>>>(s, p, q, n, g.per_warp, g.cap, out);
    RZK_CUDA_TRY(cudaGetLastError());
    return RZK_OK;
}

rzk_status launch_closest(const DevScene &s, int depth, const float *o, const float *d, int n, float *t,
                          rzk_receiver *recv, cudaStream_t st) {
    if (n <= 0) return RZK_OK;
    if (!s.ctrav || n < kRefillRays || s.n_tris < kRefillTris) {
        const auto kernel = s.ctrav ? closest_plain_kernel<true> : closest_plain_kernel<false>;
        const int cap = s.ctrav ? stack_entries(depth) : STACK_CAP;
        kernel<<<(n + kTraceBlock - 1) / kTraceBlock, kTraceBlock, sizeof(int) * kTraceBlock * cap, st>>>(s, o, d, n, cap,
                                                                                                         t, recv);
        RZK_CUDA_TRY(cudaGetLastError());
        return RZK_OK;
    }
    RunGrid g;
    RZK_CUDA_TRY(run_grid(closest_kernel, n, depth, g));
    closest_kernel<<<g.blocks, kTraceBlock, g.smem, st>>>(s, o, d, n, g.per_warp, g.cap, t, recv);
    RZK_CUDA_TRY(cudaGetLastError());
    return RZK_OK;
}

rzk_status launch_ray_query(const DevScene &s, const int *perm, const rzk_ray *rays, int n, int closest,
                            rzk_ray_hit *out, cudaStream_t st) {
    if (n <= 0) return RZK_OK;
    ray_query_kernel<<<(n + kTraceBlock - 1) / kTraceBlock, kTraceBlock, 0, st>>>(s, perm, rays, n, closest, out);
    RZK_CUDA_TRY(cudaGetLastError());
    return RZK_OK;
}

rzk_status launch_primary(const DevScene &s, const rzk_camera &cam, rzk_receiver *out,
                          cudaStream_t st) {
    if (cam.width <= 0 || cam.height <= 0) return RZK_OK;
    dim3 grid((cam.width + 15) / 16, (cam.height + 7) / 8);
    primary_kernel<<<grid, kTraceBlock, 0, st>>>(s, cam, out);
    RZK_CUDA_TRY(cudaGetLastError());
    return RZK_OK;
}

}  // namespace rzk
