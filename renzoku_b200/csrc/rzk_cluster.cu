// rzk_cluster.cu - light-transport-matrix statistics and column clustering on the device.
//
//   LightTransportMatrix::generate_alphas_for_clustering (light_transport_matrix.cc:72-106)
//   LightTransportMatrix::get_column_norms                (light_transport_matrix.cc:118-130)
//   ClusterBuilder::cluster_by_sampling                   (cluster_builder.cc:82-273)
//
// Matrix layout: column-major MatrixC<Rgb> (matrix_c.h:177-184), [cols][rows][3] floats,
// as rzk_gather_matrix writes it.  Every reduction the reference forms is a plain loop in
// float; here each is one thread's loop in the same order (and the library is built
// without FMA contraction), so alphas, norms, distances and the argmin are bit-identical.
// The column-to-cluster distances |‖K_j‖‖m_i‖ − m_i·K_j| are a cols x clusters x 3·rows
// contraction: a shared-memory tiled product in which every output accumulates over the
// 3·rows index in increasing order.  The reference's random draws (centre sampling and
// one representative per cluster) are sequential and stay on the host, drawing from the
// counter-based stream (seed, 1, 0) in the reference's order.
#include "rzk_internal.cuh"
#include "rzk_hostutil.h"
#include "rzk_cluster.cuh"

#include <algorithm>
#include <vector>

namespace rzk {

namespace {

// The column sums run over the rows in order and the row sums over the columns in order, each
// in one thread (a float sum has one order), so they are bound by the latency of one addition
// per element, not by memory.  What the additions read - the magnitudes, with their square
// roots - is formed by the whole block, tile by tile in shared memory, from coalesced loads
// issued one tile ahead.  One thread per sum reading the matrix itself left that thread waiting
// for a strided load and a square root at every step: at 256 rows x 10,000 columns the row sums
// took 2,430 us, the column statistics 70, c 131 and alpha 70 (B200).
constexpr int kColTile = 32;    // columns per block of the column kernels, rows per tile
constexpr int kStatThreads = 256;

// ALPHA = false, per column j: the magnitude-matrix norm (Rmag = |R_ij|, then sqrt Σ Rmag²),
// the get_column_norms norm (sqrt Σ (r² + g² + b²)) and magnitude() of the flattened column
// (sqrt Σ over r, g, b in order), each in row order; null outputs are left out.
// ALPHA = true: alpha_j = ‖R_j‖ c - (Rᵀ u)_j with Rᵀu summed over rows in order (MatrixC::mul).
template <bool ALPHA>
__global__ void __launch_bounds__(kStatThreads) column_kernel(const float *mat, int rows, int cols, float *rmag_norm,
                                                              float *col_norm, float *flat_norm, const float *u,
                                                              const float *c0, float *alphas) {
    constexpr int W = kStatThreads / 32, T = kColTile;
    __shared__ float raw[T][3 * T + 1];    // [column][rgb of the tile's rows]
    __shared__ float mag[T][T + 1];        // [row][column]
    __shared__ float sq[T][T + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j0 = blockIdx.x * T;
    float next[T / W][3];
    auto fetch = [&](int r0) {
        const int nf = 3 * min(T, rows - r0);
#pragma unroll
        for (int a = 0; a < T / W; ++a) {
            const int j = j0 + w + W * a;
            const float *c = mat + ((size_t)j * rows + r0) * 3;
#pragma unroll
            for (int k = 0; k < 3; ++k) next[a][k] = (j < cols && lane + 32 * k < nf) ? c[lane + 32 * k] : 0.0f;
        }
    };
    if (rows > 0) fetch(0);
    float s_mag = 0.0f, s_cn = 0.0f, s_flat = 0.0f;
    for (int r0 = 0; r0 < rows; r0 += T) {
#pragma unroll
        for (int a = 0; a < T / W; ++a)
#pragma unroll
            for (int k = 0; k < 3; ++k) raw[w + W * a][lane + 32 * k] = next[a][k];
        if (r0 + T < rows) fetch(r0 + T);
        __syncthreads();
#pragma unroll
        for (int a = 0; a < T / W; ++a) {
            const int r = w + W * a;   // lane = column
            const float x = raw[lane][3 * r], y = raw[lane][3 * r + 1], z = raw[lane][3 * r + 2];
            const float d = x * x + y * y + z * z;
            mag[r][lane] = sqrtf(d);   // MatrixC<Rgb>::flatten_magnitude (matrix_c.cc:49-58)
            sq[r][lane] = d;
        }
        __syncthreads();
        const int nr = min(T, rows - r0);
        if (w == 0) {
            if (ALPHA) {
                for (int r = 0; r < nr; ++r) s_mag += mag[r][lane] * u[r0 + r];
            } else {
                for (int r = 0; r < nr; ++r) s_mag += mag[r][lane] * mag[r][lane];
            }
        } else if (!ALPHA && w == 1) {
            for (int r = 0; r < nr; ++r) s_cn += sq[r][lane];
        } else if (!ALPHA && w == 2) {
            for (int r = 0; r < nr; ++r) {
                const float x = raw[lane][3 * r], y = raw[lane][3 * r + 1], z = raw[lane][3 * r + 2];
                s_flat += x * x;
                s_flat += y * y;
                s_flat += z * z;
            }
        }
        __syncthreads();
    }
    const int j = j0 + lane;
    if (j >= cols) return;
    if (ALPHA) {
        if (w == 0) alphas[j] = rmag_norm[j] * (*c0) - s_mag;
        return;
    }
    if (w == 0 && rmag_norm) rmag_norm[j] = sqrtf(s_mag);
    if (w == 1 && col_norm) col_norm[j] = sqrtf(s_cn);
    if (w == 2 && flat_norm) flat_norm[j] = sqrtf(s_flat);
}

// u = R * 1 (MatrixC::row_sum, matrix_c.h:236-245): per row, over columns in order; one block
// per kRowTile rows.  The last block forms c = column_norms.row_sum (one value, columns in
// order) meanwhile.
// 256 columns a tile: the 256 additions of a tile then take longer than the next tile's loads
// (128 columns: 119 us at 256 x 10,000, the loads' latency showing).
constexpr int kRowTile = 8, kRowCols = 256, kRowThreads = 512, kSumTile = 4 * kRowThreads;
__global__ void __launch_bounds__(kRowThreads) rowsum_kernel(const float *mat, int rows, int cols, float *u,
                                                              const float *rmag_norm, float *c0) {
    constexpr int RF = 3 * kRowTile, PER = kRowCols * RF / kRowThreads;
    static_assert(kRowCols * RF % kRowThreads == 0 && 2 * kRowTile * (kRowCols + 4) >= 2 * kSumTile, "tile shapes");
    __shared__ float raw[kRowCols][RF + 1];
    __shared__ __align__(16) float mag[2][kRowTile][kRowCols + 4];   // 4 apart modulo the 32 banks
    const int tid = threadIdx.x;
    int buf = 0;
    float acc = 0.0f;
    if (blockIdx.x == gridDim.x - 1) {
        float *x = &mag[0][0][0];
        float v[4];
        auto fetch = [&](int k0) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = k0 + kRowThreads * k + tid;
                v[k] = i < cols ? rmag_norm[i] : 0.0f;
            }
        };
        fetch(0);
        for (int k0 = 0; k0 < cols; k0 += kSumTile, buf ^= 1) {
            float *t = x + buf * kSumTile;
#pragma unroll
            for (int k = 0; k < 4; ++k) t[kRowThreads * k + tid] = v[k];
            if (k0 + kSumTile < cols) fetch(k0 + kSumTile);
            __syncthreads();
            if (tid == 0) {   // the zeros past the end leave the sum unchanged
                const float4 *q = reinterpret_cast<const float4 *>(t);
#pragma unroll 8
                for (int i = 0; i < kSumTile / 4; ++i) {
                    const float4 f = q[i];
                    acc += f.x;
                    acc += f.y;
                    acc += f.z;
                    acc += f.w;
                }
            }
        }
        if (tid == 0) *c0 = acc;
        return;
    }
    const int i0 = blockIdx.x * kRowTile, nr = min(kRowTile, rows - i0);
    float next[PER];
    auto fetch = [&](int c) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int e = tid + kRowThreads * k, j = c + e / RF, f = e % RF;
            next[k] = (j < cols && f < 3 * nr) ? mat[((size_t)j * rows + i0) * 3 + f] : 0.0f;
        }
    };
    fetch(0);
    for (int c = 0; c < cols; c += kRowCols, buf ^= 1) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int e = tid + kRowThreads * k;
            raw[e / RF][e % RF] = next[k];
        }
        if (c + kRowCols < cols) fetch(c + kRowCols);
        __syncthreads();
#pragma unroll
        for (int e = tid; e < kRowTile * kRowCols; e += kRowThreads) {
            const float *p = &raw[e / kRowTile][3 * (e % kRowTile)];
            mag[buf][e % kRowTile][e / kRowTile] = sqrtf(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
        }
        __syncthreads();
        if (tid < kRowTile) {   // the other warps go on to the next tile
            const float4 *q = reinterpret_cast<const float4 *>(mag[buf][tid]);
#pragma unroll 8
            for (int i = 0; i < kRowCols / 4; ++i) {
                const float4 f = q[i];
                acc += f.x;
                acc += f.y;
                acc += f.z;
                acc += f.w;
            }
        }
    }
    if (tid < nr) u[i0 + tid] = acc;
}

// K = selected columns, each scaled by its cluster weight (cluster_builder.cc:176-190).
__global__ void gather_centers_kernel(const float *mat, int rows, const int *centers, const float *w,
                                      int count, float *K) {
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t n3 = 3 * (size_t)rows;
    if (e >= n3 * count) return;
    int c = (int)(e / n3);
    size_t k = e - (size_t)c * n3;
    K[e] = mat[(size_t)centers[c] * n3 + k] * w[c];
}

// Two floats side by side, each lane rounded like the scalar multiply and add.  The multiply
// is a fused multiply-add of -0 (which leaves every product as it rounds, signed zeros
// included), with the -0 pair a kernel argument: a packed multiply whose result a packed add
// consumes is contracted into one fused operation, whatever its rounding modifier and
// -fmad=false, and would round once instead of twice.
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b, uint64_t neg0) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg0));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
constexpr uint64_t kNeg0Pair = 0x8000000080000000ull;

// D[i][j] = |kn_j * nm_i - Σ_e R[i][e] K[j][e]|, e in increasing order per output; the product
// and the sum round separately, which neither a fused multiply-add nor the tensor cores do.
// Bound by the FP32 pipe: a thread keeps 8 x 4 outputs as pairs of columns, K's values stand
// twice in shared memory so that a load yields them as pairs, and each step issues 16 packed
// multiplies and 16 packed adds on 4 16-byte loads (4 x 4 scalar outputs: 32 on 8 loads).
constexpr int TI = 64, TJ = 64, TE = 16, kDistThreads = TI * TJ / 32;
__global__ void __launch_bounds__(kDistThreads) distance_kernel(const float *R, const float *K, int n3, int cols,
                                                       int count, const float *kn, const float *nm, uint64_t neg0, float *D) {
    __shared__ __align__(16) float As[TE][TI + 4];
    __shared__ __align__(16) float2 Bs[TE][TJ + 2];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int i0 = blockIdx.x * TI, j0 = blockIdx.y * TJ;
    uint64_t acc[4][4];   // [pair of columns][cluster]
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0;
    constexpr int RS = kDistThreads / TE;   // rows a load round covers
    float na[TI / RS], nb[TJ / RS];
    auto fetch = [&](int e0) {
        const int e = e0 + (threadIdx.x & 15), r = threadIdx.x >> 4;
#pragma unroll
        for (int k = 0; k < TI / RS; ++k) {
            const int i = i0 + r + RS * k;
            na[k] = (i < cols && e < n3) ? R[(size_t)i * n3 + e] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < TJ / RS; ++k) {
            const int j = j0 + r + RS * k;
            nb[k] = (j < count && e < n3) ? K[(size_t)j * n3 + e] : 0.0f;
        }
    };
    fetch(0);
    for (int e0 = 0; e0 < n3; e0 += TE) {
        const int ee = threadIdx.x & 15, r = threadIdx.x >> 4;
#pragma unroll
        for (int k = 0; k < TI / RS; ++k) As[ee][r + RS * k] = na[k];
#pragma unroll
        for (int k = 0; k < TJ / RS; ++k) Bs[ee][r + RS * k] = make_float2(nb[k], nb[k]);
        __syncthreads();
        if (e0 + TE < n3) fetch(e0 + TE);
        const int emax = min(TE, n3 - e0);
        auto step = [&](int e) {
            const ulonglong2 a01 = *reinterpret_cast<const ulonglong2 *>(&As[e][ty * 8]);
            const ulonglong2 a23 = *reinterpret_cast<const ulonglong2 *>(&As[e][ty * 8 + 4]);
            const ulonglong2 b01 = *reinterpret_cast<const ulonglong2 *>(&Bs[e][tx * 2]);
            const ulonglong2 b23 = *reinterpret_cast<const ulonglong2 *>(&Bs[e][TJ / 2 + tx * 2]);
            const uint64_t av[4] = {a01.x, a01.y, a23.x, a23.y}, bv[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = add2(acc[a][b], mul2(av[a], bv[b], neg0));
        };
        if (emax == TE) {
#pragma unroll
            for (int e = 0; e < TE; ++e) step(e);
        } else {
            for (int e = 0; e < emax; ++e) step(e);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const int i = i0 + ty * 8 + a;
        if (i >= cols) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int j = j0 + (b >> 1) * (TJ / 2) + tx * 2 + (b & 1);
            const float v = __uint_as_float((uint32_t)(acc[a >> 1][b] >> (32 * (a & 1))));
            if (j < count) D[(size_t)i * count + j] = fabsf(kn[j] * nm[i] - v);
        }
    }
}

// Nearest cluster of each column: strict < over clusters in order (lowest index wins).
__global__ void argmin_kernel(const float *D, int cols, int count, int *owner) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cols) return;
    const float *d = D + (size_t)i * count;
    int best = -1;
    float bd = 3.402823466e+38f;   // FLT_MAX
    for (int j = 0; j < count; ++j) {
        float x = d[j];
        if (x < bd) { best = j; bd = x; }
    }
    owner[i] = best;
}

template <class T>
struct DevBuf {
    CallScratch mem;
    T *p = nullptr;
    cudaError_t alloc(size_t n, cudaStream_t st) {
        const cudaError_t e = mem.alloc(sizeof(T) * n, st);
        p = (T *)mem.get();
        return e;
    }
    void release() {
        mem.release();
        p = nullptr;
    }
};

}  // namespace

// flat_norms (optional): magnitude() of each flattened column, from the same pass.
static rzk_status column_stats_and_alphas(const float *mat, int rows, int cols, float *alphas, float *col_norms,
                                          float *flat_norms, cudaStream_t st) {
    if (cols <= 0) return RZK_OK;
    if (rows <= 0) return RZK_ERR_INVALID;
    DevBuf<float> buf;   // [rmag: cols | u: rows | c]
    RZK_CUDA_TRY(buf.alloc((size_t)cols + rows + 1, st));
    float *rmag = buf.p, *u = rmag + cols, *c0 = u + rows;
    const int grid = (cols + kColTile - 1) / kColTile;
    column_kernel<false><<<grid, kStatThreads, 0, st>>>(mat, rows, cols, rmag, col_norms, flat_norms, nullptr, nullptr,
                                                        nullptr);
    rowsum_kernel<<<(rows + kRowTile - 1) / kRowTile + 1, kRowThreads, 0, st>>>(mat, rows, cols, u, rmag, c0);
    column_kernel<true><<<grid, kStatThreads, 0, st>>>(mat, rows, cols, rmag, nullptr, nullptr, u, c0, alphas);
    RZK_CUDA_TRY(cudaGetLastError());
    buf.release();
    RZK_CUDA_TRY(cudaStreamSynchronize(st));
    return RZK_OK;
}

rzk_status ltm_alphas(const float *mat, int rows, int cols, float *alphas, float *col_norms, cudaStream_t st) {
    return column_stats_and_alphas(mat, rows, cols, alphas, col_norms, nullptr, st);
}

rzk_status cluster_by_sampling(const float *mat, int rows, int cols, int num_clusters, uint32_t seed,
                               int *h_n, int32_t *h_center, int32_t *h_rep, float *h_weight,
                               int32_t *h_assign, cudaStream_t st, float *h_mags) {
    HostRng g{seed, 1u, 0u};
    return cluster_by_sampling(mat, rows, cols, num_clusters, g, h_n, h_center, h_rep, h_weight, h_assign, st,
                               h_mags);
}

rzk_status cluster_by_sampling(const float *mat, int rows, int cols, int num_clusters, HostRng &g, int *h_n,
                               int32_t *h_center, int32_t *h_rep, float *h_weight, int32_t *h_assign,
                               cudaStream_t st, float *h_mags) {
    for (int j = 0; j < cols; ++j) h_assign[j] = -1;
    if (cols < num_clusters) {   // cluster_builder.cc:90-101
        for (int i = 0; i < cols; ++i) { h_center[i] = i; h_weight[i] = 1.0f; h_rep[i] = -1; }
        *h_n = cols;
        return RZK_OK;
    }
    DevBuf<float> alphas, nm;
    RZK_CUDA_TRY(alphas.alloc(cols, st));
    RZK_CUDA_TRY(nm.alloc(cols, st));
    rzk_status e = column_stats_and_alphas(mat, rows, cols, alphas.p, nullptr, nm.p, st);
    if (e != RZK_OK) return e;
    std::vector<float> a(cols);
    RZK_CUDA_TRY(cudaMemcpyAsync(a.data(), alphas.p, sizeof(float) * cols, cudaMemcpyDeviceToHost, st));
    RZK_CUDA_TRY(cudaStreamSynchronize(st));
    // centre sampling (cluster_builder.cc:110-156)
    DPdf pa;
    pa.set(a.data(), cols);
    std::vector<int> cen;
    std::vector<float> w;
    std::vector<int> slot(cols, -1);
    // The reference draws until it holds num_clusters distinct centres, which never ends
    // when fewer columns than that can be drawn at all (zero alpha); the target is capped
    // at the drawable count, and a draw budget bounds a pathological distribution.
    int drawable = 0;
    for (int i = 0; i < cols; ++i) drawable += pa.pdf[i] > 0.0f;
    const int target = std::min(num_clusters, drawable);
    long long draws = 0;
    const long long max_draws = 100000000LL;
    while ((int)cen.size() < target && draws++ < max_draws) {
        int k;
        float pk;
        pa.sample(g.next(), k, pk);
        if (pk == 0.0f) continue;
        if (slot[k] < 0) {
            slot[k] = (int)cen.size();
            cen.push_back(k);
            w.push_back(1.0f / pk);
        } else {
            w[slot[k]] += 1.0f / pk;
        }
    }
    const int count = (int)cen.size();
    if (count == 0) {   // nothing can be drawn: no cluster, no assignment
        *h_n = 0;
        if (h_mags) std::fill(h_mags, h_mags + cols, 0.0f);
        return RZK_OK;
    }
    const size_t n3 = 3 * (size_t)rows;
    DevBuf<int> d_cen, d_owner;
    DevBuf<float> d_w, K, kn, D;
    RZK_CUDA_TRY(d_cen.alloc(count, st));
    RZK_CUDA_TRY(d_w.alloc(count, st));
    RZK_CUDA_TRY(K.alloc(n3 * count, st));
    RZK_CUDA_TRY(kn.alloc(count, st));
    RZK_CUDA_TRY(d_owner.alloc(cols, st));
    RZK_CUDA_TRY(D.alloc((size_t)cols * count, st));
    RZK_CUDA_TRY(cudaMemcpyAsync(d_cen.p, cen.data(), sizeof(int) * count, cudaMemcpyHostToDevice, st));
    RZK_CUDA_TRY(cudaMemcpyAsync(d_w.p, w.data(), sizeof(float) * count, cudaMemcpyHostToDevice, st));
    size_t tot = n3 * count;
    gather_centers_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(mat, rows, d_cen.p, d_w.p, count, K.p);
    column_kernel<false><<<(count + kColTile - 1) / kColTile, kStatThreads, 0, st>>>(
        K.p, rows, count, nullptr, kn.p, nullptr, nullptr, nullptr, nullptr);
    dim3 grid((cols + TI - 1) / TI, (count + TJ - 1) / TJ);
    distance_kernel<<<grid, kDistThreads, 0, st>>>(mat, K.p, (int)n3, cols, count, kn.p, nm.p, kNeg0Pair, D.p);
    argmin_kernel<<<(cols + 127) / 128, 128, 0, st>>>(D.p, cols, count, d_owner.p);
    RZK_CUDA_TRY(cudaGetLastError());
    std::vector<int> owner(cols);
    std::vector<float> mags(cols);
    RZK_CUDA_TRY(cudaMemcpyAsync(owner.data(), d_owner.p, sizeof(int) * cols, cudaMemcpyDeviceToHost, st));
    RZK_CUDA_TRY(cudaMemcpyAsync(mags.data(), nm.p, sizeof(float) * cols, cudaMemcpyDeviceToHost, st));
    for (DevBuf<float> *b : {&alphas, &nm, &d_w, &K, &kn, &D}) b->release();
    for (DevBuf<int> *b : {&d_cen, &d_owner}) b->release();
    RZK_CUDA_TRY(cudaStreamSynchronize(st));
    if (h_mags) std::copy(mags.begin(), mags.end(), h_mags);
    // members in column order, pdf over magnitudes, representative (cluster_builder.cc:228-272)
    std::vector<std::vector<int>> members(count);
    for (int i = 0; i < cols; ++i)
        if (owner[i] >= 0) members[owner[i]].push_back(i);
    std::vector<int> rep(count);
    std::vector<float> wf(count);
    for (int c = 0; c < count; ++c) {
        std::vector<float> mm(members[c].size());
        for (size_t t = 0; t < mm.size(); ++t) mm[t] = mags[members[c][t]];
        DPdf pc;
        pc.set(mm.data(), (int)mm.size());
        int j;
        float pj;
        pc.sample(g.next(), j, pj);
        if (j < 0) {
            rep[c] = members[c].empty() ? -1 : members[c][members[c].size() / 2];
            wf[c] = 0.0f;
        } else {
            rep[c] = members[c][j];
            wf[c] = 1.0f / pj;
        }
    }
    int n = 0;
    std::vector<int> map(count, -1);
    for (int c = 0; c < count; ++c) {
        if (rep[c] < 0) continue;
        map[c] = n;
        h_center[n] = cen[c];
        h_rep[n] = rep[c];
        h_weight[n] = wf[c];
        n++;
    }
    for (int i = 0; i < cols; ++i) h_assign[i] = owner[i] >= 0 ? map[owner[i]] : -1;
    *h_n = n;
    return RZK_OK;
}

}  // namespace rzk

extern "C" {

rzk_status rzk_ltm_alphas(const float *d_matrix, int rows, int cols, float *d_alphas, float *d_col_norms,
                          void *stream) {
    if (rows < 0 || cols < 0 || (cols > 0 && (!d_matrix || !d_alphas))) return RZK_ERR_INVALID;
    return rzk::ltm_alphas(d_matrix, rows, cols, d_alphas, d_col_norms, (cudaStream_t)stream);
}

rzk_status rzk_cluster_by_sampling(const float *d_matrix, int rows, int cols, int num_clusters, uint32_t seed,
                                   int *h_n_clusters, int32_t *h_center, int32_t *h_representative,
                                   float *h_weight, int32_t *h_assign, void *stream) {
    if (rows < 0 || cols < 0 || num_clusters <= 0 || !h_n_clusters || !h_center || !h_representative ||
        !h_weight || (cols > 0 && (!d_matrix || !h_assign)))
        return RZK_ERR_INVALID;
    return rzk::cluster_by_sampling(d_matrix, rows, cols, num_clusters, seed, h_n_clusters, h_center,
                                    h_representative, h_weight, h_assign, (cudaStream_t)stream);
}

}  // extern "C"
