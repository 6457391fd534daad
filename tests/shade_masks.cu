// shade_masks.cu - one warp tile through both summing halves of the two-pass gather, on given
// ballots: out[0] by shade_marked, out[1] by shade_chunk (planes of 32 receivers x 3 floats).
#include "../renzoku_b200/csrc/rzk_gather_dev.cuh"

using namespace rzk;

constexpr int kWarps = 8;

__global__ void __launch_bounds__(32 * kWarps) shade_kernel(GatherScene s, const rzk_receiver *recv, int n_recv,
                                                            const rzk_vpl *vpls, int n_vpl, const uint32_t *masks,
                                                            float *out) {
    __shared__ float terms[32][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ri = lane_receiver(0, lane, n_recv, 0);
    RecvRegs r;
    rzk_material rm;
    bool active = false;
    if (ri >= 0) {
        r = load_receiver(recv + ri);
        active = r.mat >= 0;
        if (active) rm = load_material(s.mats + r.mat);
    }
    if (w == 0) {
        const Rgb sum = shade_marked(s, r, rm, active, vpls, 0, n_vpl, masks, RZK_CLAMP_NONE, 0.0f, lane);
        out[3 * lane] = sum.r;
        out[3 * lane + 1] = sum.g;
        out[3 * lane + 2] = sum.b;
    }
    const float c = shade_chunk<kWarps>(s, r, active, vpls, 0, n_vpl, masks, RZK_CLAMP_NONE, 0.0f, terms);
    if (w < 3) out[96 + 3 * lane + w] = c;
}

extern "C" int shade(const rzk_receiver *recv, int n_recv, const rzk_vpl *vpls, int n_vpl, const uint32_t *masks,
                     const rzk_material *mats, float *out) {
    GatherScene s = {};
    s.mats = mats;
    s.tmin = 1e-3f;
    shade_kernel<<<1, 32 * kWarps>>>(s, recv, n_recv, vpls, n_vpl, masks, out);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return (int)e;
}
