// rzk_internal.cuh - library-internal types shared by the .cu files of librzk_cuda.so.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

#include "../../include/rzk.h"
#include "rzk_math.cuh"

#define RZK_CUDA_TRY(expr)                                   \
    do {                                                     \
        cudaError_t _e = (expr);                             \
        if (_e != cudaSuccess) {                             \
            rzk::set_last_cuda_error(_e, #expr, __FILE__, __LINE__); \
            return _e == cudaErrorMemoryAllocation ? RZK_ERR_NOMEM : RZK_ERR_CUDA; \
        }                                                    \
    } while (0)
#define RZK_TRY(expr) do { rzk_status _s = (expr); if (_s != RZK_OK) return _s; } while (0)

namespace rzk {

void set_last_cuda_error(cudaError_t e, const char *what, const char *file, int line);

// While it lives, allocations of this thread do not break a stream capture that another thread has
// in progress (they are "potentially unsafe" calls, which a capture in global mode, the default,
// is invalidated by).
class RelaxedCapture {
public:
    RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode_); }
    RelaxedCapture(const RelaxedCapture &) = delete;
    RelaxedCapture &operator=(const RelaxedCapture &) = delete;
    ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode_); }

private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// Device scratch of one call, ordered on the call's stream: taken from a memory pool that the
// library keeps per device and given back to it, on the same stream, when the object dies.
// A cudaMalloc and cudaFree pair costs 100-400 us each and waits for the whole device (VPL
// generation of the 24,000-particle frame: 0.64 of 1.1 ms; clustering 10,000 columns: 1.8 of
// 2.6 ms; many milliseconds now and then); from the pool it is a few microseconds.  The pool
// serves any number of threads and streams (the runtime orders reuse across streams).  What it
// holds beyond kPoolKeep without a call using it goes back to the device when a stream is next
// waited for, so a call that waits releases its scratch before it does.  It is emptied when the
// device's last context is destroyed, and not destroyed with it: another thread's call may be using
// it (destroying it then crashed the process).
constexpr unsigned long long kPoolKeep = 256ull << 20;
class CallScratch {
public:
    CallScratch() = default;
    CallScratch(const CallScratch &) = delete;
    CallScratch &operator=(const CallScratch &) = delete;
    ~CallScratch() { release(); }
    void release() {   // after the last kernel that uses the memory has been launched
        if (!p_) return;
        RelaxedCapture relaxed;
        cudaFreeAsync(p_, st_);
        p_ = nullptr;
    }
    cudaError_t alloc(size_t bytes, cudaStream_t st);   // once per object, on the current device
    char *get() const { return (char *)p_; }

private:
    void *p_ = nullptr;
    cudaStream_t st_ = nullptr;
};
void pool_context_created(int device);
void pool_context_destroyed(int device);

// Device error word bits (written by kernels, read by rzk_context_check).
enum : uint32_t { ERR_TIMEOUT = 1u, ERR_STACK = 2u, ERR_BOUNDS = 4u };

// Code of an unused entry of a 4-wide traversal node.
constexpr int kWideEmpty = 0x7fffffff;

// Area light as the VPL generator samples it (area_light.cc:27-46, quad.cc:73-87).
struct DevLight {
    float4 p0[2], p1[2], p2[2];   // the (one or two) triangles of the light's shape
    float4 n[2];                  // their facet normals; .w = area
    float4 basis_n, basis_u;      // Surface::get_basis: larger triangle's n and tangent
    float4 emit;                  // radiance; .w unused
    float t0_ratio;
    int kind, flags, n_tris;
};

// What the gather kernels need of a scene.
struct GatherScene {
    const float4 *wide8;      // 8-wide any-hit tree: 16 x float4 per node (rzk_sah.cu)
    const float4 *trav;       // any-hit tree, same packing as nodes (rzk_sah.cu; = nodes without it)
    const float4 *tri_isect;  // 3 x float4 per sorted triangle (see tri_hit)
    const rzk_material *mats;
    uint32_t *err;            // device error word (context-owned)
    unsigned long long *rays; // shadow rays traced by the gather kernels (context-owned counter)
    int n_nodes;
    float tmin;
};

// Everything a kernel needs to trace and shade in one scene (passed by value).
struct DevScene : GatherScene {
    const float4 *nodes;      // 2 x float4 per slot, slot = BFS node index + 1
    const float4 *tri_shade;  // 2 x float4 per sorted triangle: {n, surf}, {u, -}
    const float4 *wide;       // 8 x float4 per 4-wide traversal node (see rzk_bvh.cu K6)
    const float4 *ctrav;      // closest-hit tree: trav with inflated boxes (rzk_sah.cu), or null
    const float *verts;       // 9 per triangle in input order
    const int *perm;          // sorted triangle slot -> input triangle
    const int4 *surf;         // per surface {mat, flags, light, -}
    const DevLight *lights;
    const float *light_pdf;
    const float *light_cdf;
    int n_tris, n_mats, n_lights;
    float cguard[4];          // origins ctrav covers: centre, squared radius
};

struct Scene;

struct BatchPlan;   // rzk_batch.cu: a batch of gathers split into launch tables

}  // namespace rzk

struct rzk_context {
    int device = 0;
    uint32_t *d_err = nullptr;             // error word (the first 8 bytes of a 16-byte allocation)
    unsigned long long *d_rays = nullptr;  // shadow rays traced by the gather kernels (its last 8)
    // reusable gather scratch: per-(VPL chunk, receiver) partial sums
    float *d_partial = nullptr;
    size_t partial_bytes = 0;
    // staging for rzk_gather_host
    void *d_stage = nullptr;
    size_t stage_bytes = 0;
    double *d_mean = nullptr;
    // work counter of the persistent gather and its resident grid size per variant
    int *d_work = nullptr;
    // spatially ordered VPL copy of a chunked gather, its sort keys and sort scratch
    void *d_order = nullptr;
    size_t order_bytes = 0;
    int persistent_grid[16] = {0};
    int gather_kernels = 0;   // kernels the last gather launched
    int vis_grid = 0;   // resident grid of the two-pass gather's tracing kernel
    // ballots of two-pass gathers: buffer k holds 2^(kMaskLog0 + k) words.  None is freed before
    // the context is, so that a captured gather stays good whatever gathers run after it.
    static constexpr int kMaskLog0 = 16, kMaskLogMax = 26;   // 256 KB to 256 MB
    uint32_t *d_masks[kMaskLogMax - kMaskLog0 + 1] = {};
};

struct rzk_scene {
    rzk_context *ctx = nullptr;
    int n_tris = 0, n_nodes = 0, n_levels = 0, n_surfs = 0, n_mats = 0, n_lights = 0;
    float tmin = 1e-3f;
    float box[6] = {0, 0, 0, 0, 0, 0};   // Aggregate::box (min xyz, max xyz), incl. the origin
    // original (flattened, input-order) triangles
    float *d_v = nullptr;        // [n][9]
    float *d_tp = nullptr;       // [n][3] tangent reference vertex
    int *d_tri_surf = nullptr;   // [n]
    float *d_tri_n = nullptr;    // [n][3] facet normal
    float *d_tri_u = nullptr;    // [n][3] tangent
    float *d_tri_area = nullptr; // [n]
    float *d_bmin = nullptr, *d_bmax = nullptr;   // [n][3] triangle boxes
    // build products
    uint32_t *d_codes = nullptr, *d_sorted_codes = nullptr;
    int *d_perm = nullptr;
    int *d_start = nullptr, *d_end = nullptr, *d_left = nullptr, *d_right = nullptr,
        *d_level = nullptr;
    float *d_nbmin = nullptr, *d_nbmax = nullptr;  // [nodes][3]
    std::vector<int> level_first, level_last;
    // packed traversal layout
    float4 *d_nodes = nullptr, *d_tri_isect = nullptr, *d_tri_shade = nullptr;
    float4 *d_wide = nullptr;
    int n_wide = 0, n_wide_cap = 0;
    float4 *d_trav = nullptr;    // SAH any-hit tree (rzk_sah.cu)
    float4 *d_wide8 = nullptr;   // 8-wide any-hit tree of the packet gathers (rzk_sah.cu), not saved
    int n_wide8 = 0;             // nodes it has room for
    float4 *d_ctrav = nullptr;   // closest-hit tree (rzk_sah.cu), not saved: made from d_trav
    size_t ctrav_bytes = 0;
    float cguard[4] = {0, 0, 0, -1};
    int trav_depth = 0;
    size_t trav_bytes = 0;
    bool build_trav = true;
    int4 *d_surf = nullptr;
    rzk_material *d_mats = nullptr;
    rzk::DevLight *d_lights = nullptr;
    float *d_light_pdf = nullptr, *d_light_cdf = nullptr;
    std::vector<int> light_surf;   // host: surface index of each light
    size_t device_bytes = 0;
    // most entries a walk of the any-hit or closest-hit tree pushes (the reference tree's own
    // limit where there is neither)
    int walk_depth() const { return d_trav && trav_depth > 0 ? trav_depth : rzk::STACK_CAP; }
    // scratch for the build (freed after)
    rzk::DevScene dev() const {
        rzk::DevScene s;
        s.nodes = d_nodes; s.tri_isect = d_tri_isect; s.tri_shade = d_tri_shade; s.wide = d_wide;
        s.trav = d_trav ? d_trav : d_nodes;
        s.wide8 = d_wide8;
        s.ctrav = d_ctrav;
        for (int i = 0; i < 4; ++i) s.cguard[i] = cguard[i];
        s.verts = d_v;
        s.perm = d_perm;
        s.surf = d_surf; s.mats = d_mats; s.lights = d_lights; s.light_pdf = d_light_pdf;
        s.light_cdf = d_light_cdf; s.n_tris = n_tris; s.n_nodes = n_nodes; s.n_mats = n_mats;
        s.n_lights = n_lights; s.tmin = tmin; s.err = ctx ? ctx->d_err : nullptr;
        s.rays = ctx ? ctx->d_rays : nullptr;
        return s;
    }
};

namespace rzk {
// rzk_bvh.cu
rzk_status bvh_build(rzk_scene *s, cudaStream_t st);
// rzk_sah.cu
rzk_status build_sah_tree(rzk_scene *s, cudaStream_t st);
rzk_status build_closest_tree(rzk_scene *s, cudaStream_t st);
rzk_status build_wide_tree(rzk_scene *s, cudaStream_t st);
// utilities (rzk_bvh.cu)
rzk_status exclusive_scan_i32(const int *d_in, int *d_out, int n, int *d_total, void *d_tmp,
                              size_t tmp_bytes, cudaStream_t st);
size_t exclusive_scan_tmp_bytes(int n);
size_t radix_sort_scratch_bytes(int n);
rzk_status radix_sort_u32(uint32_t *keys, int *vals, int n, int bits, void *scratch, cudaStream_t st);
int exclusive_scan_launches(int n, bool total);   // kernels one exclusive_scan_i32 call launches
int radix_sort_launches(int n, int bits);         // kernels one radix_sort_u32 call launches

// rzk_gather.cu: spatial VPL order of chunked gathers.  Each segment is one gather's VPL
// set; ordering writes every segment's VPLs, stably sorted by the Hilbert-curve index of
// their positions' cells on a 256^3 grid over that gather's scene box, to
// out[begin, begin + n).
constexpr int kOrderSegs = 128;
struct OrderSeg {
    const rzk_vpl *src;
    int begin, n;
    float lo[3], k[3];
};
struct OrderTable {
    OrderSeg seg[kOrderSegs];
    int n_segs, total;
};
void order_table_init(OrderTable &t);
// appends a segment (no device work); false when the table is full
bool order_table_add(OrderTable &t, const rzk_vpl *src, int n, const float *box);
size_t order_scratch_bytes(int total);
int order_launches(const OrderTable &t);
rzk_status order_vpls(const OrderTable &t, void *scratch, rzk_vpl *out, cudaStream_t st, const int **from = nullptr);
// rzk_gather.cu: every (receiver, VPL) pair into a column-major [n_vpl][n_recv][3] matrix;
// kind 0 radiance, 1 incident radiance, 2 visible x incident radiance (+ visibility)
rzk_status launch_matrix(const DevScene &s, int depth, const float *box, const rzk_receiver *recv, int n_recv, const rzk_vpl *vpls,
                         int n_vpl, int mode, float tau, float *mat, uint8_t *vis, int kind,
                         cudaStream_t st);
// Chunk ring of the persistent gather on fixed scratch (rzk_gather.cu, used by
// rzk_gather_noalloc): the per-chunk sums of at most `slots` warp tiles at a time.  Tile t writes its chunks to slot t % slots once the slot
// has finished t / slots tiles (`round`); the warp that writes a tile's last chunk (`done`)
// adds the chunks in chunk order, writes the tile's pixels and frees the slot.  The
// counters start at zero (one memset of ring_counter_bytes); the sums need no clearing.
struct ChunkRing {
    int *done;     // [slots] chunks of the slot's current tile written
    int *round;    // [slots] tiles the slot has finished
    float *sums;   // [slots][n_chunks][32 lanes][3]
    int slots;
};
constexpr int kRingSlots = 8192;   // most slots a ring is given (96 MiB at 32 chunks)
size_t ring_counter_bytes(int slots);
size_t ring_bytes(int slots, int n_chunks);
int ring_slots_fitting(size_t bytes, int n_chunks);   // slots whose ring fits in `bytes`
ChunkRing ring_at(void *base, int slots);
// the ring's slot wait on a slot nothing frees, limited to timeout_ms (rzk_debug_ring_wait)
rzk_status launch_ring_wait_probe(rzk_context *ctx, int timeout_ms, int *h_acquired, cudaStream_t st);
// rzk_gather.cu: make the context's scratch (d_partial) at least `bytes` long
rzk_status ensure_scratch(rzk_context *ctx, size_t bytes);
// rzk_batch.cu: plan a batch (validates jobs; no device work), then launch it on a partial
// buffer of batch_plan_partial_floats floats, an ordering buffer of batch_plan_order_bytes
// bytes (16-byte aligned; null when that is 0) and batch_plan_tables work counters;
// grid 0 = the variant's resident grid.
rzk_status batch_plan_create(const rzk_gather_job *jobs, int n_jobs, int chunk_len, int tile_width,
                             BatchPlan **out);
int batch_variant_tile_width(int variant);   // warp tile width (pixels) of a batch variant
void batch_plan_destroy(BatchPlan *p);
size_t batch_plan_partial_floats(const BatchPlan *p);
size_t batch_plan_order_bytes(const BatchPlan *p);
int batch_plan_tables(const BatchPlan *p);
int batch_plan_launches(const BatchPlan *p);   // kernels the plan's last batch_plan_launch launched
// masks: null, or batch_plan_mask_words words, with which the tables that a two-pass launch
// suits run in two passes (as rzk_gather does; variant 0 only, the same images).
size_t batch_plan_mask_words(const BatchPlan *p);
rzk_status batch_plan_launch(BatchPlan *p, float *partial, void *order, int *work, uint32_t *masks, int variant, int grid,
                             cudaStream_t st);
}  // namespace rzk
