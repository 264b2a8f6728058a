// Chooses the instantiated hidden-units-per-lane count K for an RBM of M hidden units.
#include "kernels.h"

namespace rbmg {

template <int K>
cudaError_t rbm_mc_launch_k(const RbmDev&, const OpDev*, const McLaunch&, cudaStream_t);
template <int K>
cudaError_t rbm_est_launch_k(const RbmDev&, const OpDev*, const RbmDev*, const EstLaunch&, cudaStream_t);

// Every pass evaluates all 32 K units, the padding too, so the counts are at most a third (above
// 32 units) over what M needs.  With 1, 2, 4, 8, 13 and 18 alone M = 75 ran 128 units and M = 150
// ran 256.  Microseconds a sweep of 1024 and
// 16384 walkers with those and now: N = 30, M = 75: 15 / 14 and 109 / 93; N = 40, M = 150: 34 / 24 and
// 260 / 176; N = 64, M = 180: 54 / 45 and 411 / 324; N = 80, M = 300: 118 / 93 and 893 / 671; the
// energies of 10007 configurations at N = 75, M = 150: 0.64 / 0.50 ms with their log psi.
static const int kInstantiated[] = {1, 2, 3, 4, 5, 6, 8, 10, 13, 18};

int rbm_lanes_k(int M) {
    const int need = (M + 31) / 32;
    for (int k : kInstantiated)
        if (k >= need) return k;
    return -1;
}

int rbm_range_top(int M) {
    for (int top : {32, 64, 128, 256, 416})
        if (M <= top) return top;
    return 576;
}
bool rbm_pairable(int Ma, int Mb) { return rbm_range_top(Ma) == rbm_range_top(Mb); }

cudaError_t launch_rbm_mc(const RbmDev& P, const OpDev* op, const McLaunch& L, cudaStream_t st) {
    switch (P.Mpad / 32) {
        case 1: return rbm_mc_launch_k<1>(P, op, L, st);
        case 2: return rbm_mc_launch_k<2>(P, op, L, st);
        case 3: return rbm_mc_launch_k<3>(P, op, L, st);
        case 4: return rbm_mc_launch_k<4>(P, op, L, st);
        case 5: return rbm_mc_launch_k<5>(P, op, L, st);
        case 6: return rbm_mc_launch_k<6>(P, op, L, st);
        case 8: return rbm_mc_launch_k<8>(P, op, L, st);
        case 10: return rbm_mc_launch_k<10>(P, op, L, st);
        case 13: return rbm_mc_launch_k<13>(P, op, L, st);
        case 18: return rbm_mc_launch_k<18>(P, op, L, st);
        default: return cudaErrorInvalidValue;
    }
}

// Wq [N][KP][32], bq [KP][32] (KP = ceil(K / 2)): entry (row, kk, lane) holds units
// j0 = lane + 32 (2 kk) and j1 = j0 + 32; row N is the bias
__global__ void rbm_pairs_kernel(int N, int Mpad, int KP, const float2* W, const float2* b, float4* Wq, float4* bq) {
    const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long per_row = static_cast<long>(KP) * 32;
    if (idx >= (N + 1) * per_row) return;
    const int row = static_cast<int>(idx / per_row);
    const int rem = static_cast<int>(idx - row * per_row);
    const int kk = rem / 32, lane = rem % 32;
    const int j0 = lane + 32 * (2 * kk), j1 = j0 + 32;
    const float2* src = row < N ? W + static_cast<long>(row) * Mpad : b;
    const float2 a = j0 < Mpad ? src[j0] : make_float2(0.0f, 0.0f);
    const float2 c = j1 < Mpad ? src[j1] : make_float2(0.0f, 0.0f);
    (row < N ? Wq[idx] : bq[rem]) = make_float4(a.x, c.x, a.y, c.y);
}

// Wg [N][K H][G], bg [K H][G] (kernels.h); row N is the bias
__global__ void rbm_group_pairs_kernel(int N, int Mpad, int G, const float2* W, const float2* b, float4* Wg,
                                       float4* bg) {
    const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int per_row = Mpad / 2;
    if (idx >= static_cast<long>(N + 1) * per_row) return;
    const int row = static_cast<int>(idx / per_row), rem = static_cast<int>(idx - static_cast<long>(row) * per_row);
    const int g = rem % G, pp = rem / G, H = 16 / G;
    const int j0 = 32 * (pp / H) + 2 * G * (pp % H) + g;
    const float2* src = row < N ? W + static_cast<long>(row) * Mpad : b;
    const float2 a = src[j0], c = src[j0 + G];
    (row < N ? Wg[idx] : bg[rem]) = make_float4(a.x, c.x, a.y, c.y);
}

// Wt4 [Mpad / 2][N]: entry (p, i) = (x_j, x_j+4, y_j, y_j+4) of W[i], j = 8 (p / 4) + p % 4
__global__ void rbm_transpose_kernel(int N, int Mpad, const float2* W, float4* Wt4) {
    const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<long>(N) * (Mpad / 2)) return;
    const int p = static_cast<int>(idx / N), i = static_cast<int>(idx - static_cast<long>(p) * N);
    const int j = 8 * (p / 4) + p % 4;
    const float2 a = W[static_cast<long>(i) * Mpad + j], c = W[static_cast<long>(i) * Mpad + j + 4];
    Wt4[idx] = make_float4(a.x, c.x, a.y, c.y);
}

cudaError_t launch_rbm_pairs(int N, int Mpad, const float2* W, const float2* b, float4* Wq, float4* bq,
                             float4* Wt, float4* Wg, float4* bg, cudaStream_t st) {
    const int KP = (Mpad / 32 + 1) / 2;
    const long n = static_cast<long>(N + 1) * KP * 32;
    rbm_pairs_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, st>>>(N, Mpad, KP, W, b, Wq, bq);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long q = static_cast<long>(N + 1) * (Mpad / 2);
    if (rbm_group(Mpad / 32) < 32)
        rbm_group_pairs_kernel<<<static_cast<int>((q + 255) / 256), 256, 0, st>>>(N, Mpad, rbm_group(Mpad / 32), W, b, Wg,
                                                                              bg);
    e = cudaGetLastError();
    if (e != cudaSuccess || !Wt) return e;
    const long m = static_cast<long>(N) * (Mpad / 2);
    rbm_transpose_kernel<<<static_cast<int>((m + 255) / 256), 256, 0, st>>>(N, Mpad, W, Wt);
    return cudaGetLastError();
}

cudaError_t launch_rbm_estimate(const RbmDev& P, const OpDev* op, const RbmDev* PP, const EstLaunch& L,
                                cudaStream_t st) {
    if (PP && PP->Mpad != P.Mpad) {   // a launch per network: the kernel has one number of units
        if (!rbm_pairable(P.M, PP->M)) return cudaErrorInvalidValue;
        EstLaunch own = L, prime = L;
        own.flags &= ~EST_PRIME;
        prime.flags &= EST_PRIME | EST_ENUMERATE;
        const cudaError_t e = launch_rbm_estimate(P, op, nullptr, own, st);
        return e != cudaSuccess ? e : launch_rbm_estimate(*PP, nullptr, PP, prime, st);
    }
    switch (P.Mpad / 32) {
        case 1: return rbm_est_launch_k<1>(P, op, PP, L, st);
        case 2: return rbm_est_launch_k<2>(P, op, PP, L, st);
        case 3: return rbm_est_launch_k<3>(P, op, PP, L, st);
        case 4: return rbm_est_launch_k<4>(P, op, PP, L, st);
        case 5: return rbm_est_launch_k<5>(P, op, PP, L, st);
        case 6: return rbm_est_launch_k<6>(P, op, PP, L, st);
        case 8: return rbm_est_launch_k<8>(P, op, PP, L, st);
        case 10: return rbm_est_launch_k<10>(P, op, PP, L, st);
        case 13: return rbm_est_launch_k<13>(P, op, PP, L, st);
        case 18: return rbm_est_launch_k<18>(P, op, PP, L, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace rbmg
