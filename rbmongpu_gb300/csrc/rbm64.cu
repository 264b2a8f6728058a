// FP64 per-sample pass for the Hilbert-space distance of complex RBMs.
//
// The distance between nearby states is a difference of nearly equal averages
// (d^2 = 1 - |<omega>|^2 / (<norm><ratio>) is ~1e-6 for the perturbed copies the
// reference tests), so the per-sample terms omega_s = exp(conj(log psi'_s - log psi_s)) E_s
// and ratio_s are computed here in FP64, from FP64 copies of the parameters,
// with log psi' - log psi summed angle by angle as differences.  One warp per sample,
// angles and activations of the warp's sample in shared memory.
#include <cuda_runtime.h>

#include "kernels.h"
#include "math64.cuh"
#include "rbm64.h"

namespace rbmg {

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ double2 warp_sum64(double2 v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
    }
    return v;
}

__device__ __forceinline__ bool spin_up(const uint64_t* s, int i) { return (s[i >> 6] >> (i & 63)) & 1ull; }

// six consecutive spins of a configuration, from spin 6 g on
__device__ __forceinline__ int spin_group(const uint64_t* s, int g, int N) {
    const int i = kTab64Spins * g, w = i >> 6, sh = i & 63;
    uint64_t v = s[w] >> sh;
    if (sh > 64 - kTab64Spins && w + 1 < kMaxWords) v |= s[w + 1] << (64 - sh);
    return static_cast<int>(v & ((1u << min(kTab64Spins, N - i)) - 1u));
}

// tab[g][m][j] = sum over the spins i of group g of +-W[i][j], signs by the bits of m; group 0
// carries b[j].  An angle is then one entry per six spins (2 FP64 additions for 12).
__global__ void table64_kernel(Rbm64 P, double2* tab) {
    const int groups = (P.N + kTab64Spins - 1) / kTab64Spins;
    const long total = static_cast<long>(groups) * kTab64Size * P.M;
    for (long e = blockIdx.x * 256L + threadIdx.x; e < total; e += static_cast<long>(gridDim.x) * 256) {
        const int j = static_cast<int>(e % P.M);
        const int m = static_cast<int>(e / P.M) % kTab64Size, g = static_cast<int>(e / P.M / kTab64Size);
        double2 a = g == 0 ? P.b[j] : make_double2(0.0, 0.0);
        for (int i = kTab64Spins * g; i < min(P.N, kTab64Spins * (g + 1)); i++) {
            const double2 w = P.W[static_cast<long>(i) * P.M + j];
            const double sg = (m >> (i - kTab64Spins * g)) & 1 ? 1.0 : -1.0;
            a.x = fma(sg, w.x, a.x);
            a.y = fma(sg, w.y, a.y);
        }
        tab[e] = a;
    }
}

__device__ __forceinline__ double2 angle64(const Rbm64& P, const uint64_t* s, int j) {
    if (P.tab) {
        double2 a = make_double2(0.0, 0.0);
        const int groups = (P.N + kTab64Spins - 1) / kTab64Spins;
#pragma unroll 2
        for (int g = 0; g < groups; g++) {
            const double2 t = P.tab[(static_cast<long>(g) * kTab64Size + spin_group(s, g, P.N)) * P.M + j];
            a.x += t.x;
            a.y += t.y;
        }
        return a;
    }
    double2 a = P.b[j];
    for (int i = 0; i < P.N; i++) {
        const double2 w = P.W[static_cast<long>(i) * P.M + j];
        if (spin_up(s, i)) { a.x += w.x; a.y += w.y; }
        else { a.x -= w.x; a.y -= w.y; }
    }
    return a;
}

// coefficient and phase of string n on the configuration s
__device__ __forceinline__ double2 string_factor64(const OpDev& op, int n, const uint64_t* s) {
    int parity = 0;
    for (int k = 0; k < kMaxWords; k++) parity += __popcll(op.zmask[n * kMaxWords + k] & ~s[k]);
    const double2 c = op.coef[n];
    const int yp = op.ypow[n] & 3;
    const double2 r = yp == 0 ? c : (yp == 1 ? make_double2(c.y, -c.x) : (yp == 2 ? make_double2(-c.x, -c.y)
                                                                                : make_double2(-c.y, c.x)));
    return (parity & 1) ? make_double2(-r.x, -r.y) : r;
}

// The warp's sums of eight complex values a lane, in one folding butterfly: lanes 4 u .. 4 u + 3
// receive the sum of value u (9 complex additions a lane against 40 of eight butterflies)
__device__ __forceinline__ double2 warp_fold8(double2 (&d)[8], int lane) {
#pragma unroll
    for (int half = 4, off = 16; half >= 1; half >>= 1, off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const double2 send = up ? d[i] : d[i + half], keep = up ? d[i + half] : d[i];
            d[i].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, off);
            d[i].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, off);
        }
    }
#pragma unroll
    for (int off = 2; off >= 1; off >>= 1) {
        d[0].x += __shfl_xor_sync(0xffffffffu, d[0].x, off);
        d[0].y += __shfl_xor_sync(0xffffffffu, d[0].y, off);
    }
    return d[0];
}

// One warp per configuration, its lanes over the hidden units.  Shared memory per warp:
// theta[M], f[M] + C (double2 each).  op.S = 0 skips the local energy and PP.W = null skips
// log psi'; with both it is the FP64 log psi pass that the exact-summation weights and the psi
// vector use.  Bound: the FP64 pipe.  The off-diagonal strings are taken eight at a time
// (their lane sums folded together), and their exp, cos and sin 32 at a time, one string per
// lane, so that no FP64 instruction repeats in the 32 lanes what one could do: N = 16, M = 32
// over 2^16 configurations (one pass with log psi', one for the weights) takes 2670 us,
// 9350 us with one string at a time in all lanes; 1.8 ms is the issue time of the strings'
// activations alone.
__global__ void rbm_hsd64_kernel(Rbm64 P, Rbm64 PP, OpDev op, Hsd64Launch L) {
    extern __shared__ double2 smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long t = static_cast<long>(blockIdx.x) * kWarpsPerBlock + warp;
    if (t >= L.count) return;
    const int M = P.M, N = P.N;
    double2* th = smem + static_cast<long>(warp) * 2 * M;
    double2* f = th + M;
    uint64_t s[kMaxWords] = {0, 0, 0, 0};
    const int nw = (N + 63) / 64;
    if (L.enumerate) {
        const uint64_t idx = L.enum_base + static_cast<uint64_t>(t);
        s[0] = N >= 64 ? idx : (idx & ((1ull << N) - 1ull));
    } else {
#pragma unroll
        for (int k = 0; k < kMaxWords; k++)
            if (k < nw) s[k] = L.spins[t * nw + k];
    }
    double2 lp = make_double2(0.0, 0.0);
    for (int j = lane; j < M; j += 32) {
        const double2 a = angle64(P, s, j);
        const double2 v = lc64(a).open();
        th[j] = a;
        f[j] = v;
        lp.x += v.x - kLcC;
        lp.y += v.y;
    }
    lp = warp_sum64(lp);
    __syncwarp();
    // local energy (include/operator/Operator.hpp:90-115) with per-angle differences
    double2 e = make_double2(0.0, 0.0);
    for (int n = lane; n < op.S; n += 32) {
        if (op.nflip[n] != 0) continue;
        const double2 cf = string_factor64(op, n, s);
        e.x += cf.x;
        e.y += cf.y;
    }
    const int strings = op.S > 0 ? op.num_offdiag : 0;
    for (int q0 = 0; q0 < strings; q0 += 32) {
        double2 mine = make_double2(0.0, 0.0);   // log psi(s'_n) - log psi(s) of string q0 + lane
        for (int b = 0; b < 4 && q0 + 8 * b < strings; b++) {
            double2 d[8];
            int site[8], flips[8];
            double two_s[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                d[u] = make_double2(0.0, 0.0);
                const int n = op.offdiag[min(q0 + 8 * b + u, strings - 1)];
                flips[u] = op.nflip[n];
                site[u] = op.flip_off[n];
                const int first = op.flip_sites[site[u]];
                two_s[u] = spin_up(s, first) ? -2.0 : 2.0;
                if (flips[u] == 1) site[u] = first;
            }
            for (int j = lane; j < M; j += 32) {
                const double2 a0 = th[j], f0 = f[j];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    double2 a = a0;
                    if (flips[u] == 1) {
                        const double2 w = P.W[static_cast<long>(site[u]) * M + j];
                        a.x = fma(two_s[u], w.x, a.x);
                        a.y = fma(two_s[u], w.y, a.y);
                    } else {
                        for (int k = 0; k < flips[u]; k++) {
                            const int i = op.flip_sites[site[u] + k];
                            const double2 w = P.W[static_cast<long>(i) * M + j];
                            const double sg = spin_up(s, i) ? -2.0 : 2.0;
                            a.x = fma(sg, w.x, a.x);
                            a.y = fma(sg, w.y, a.y);
                        }
                    }
                    lc64(a).add_difference(f0, d[u]);
                }
            }
            const double2 sum = warp_fold8(d, lane);
            const double vx = __shfl_sync(0xffffffffu, sum.x, 4 * (lane & 7));
            const double vy = __shfl_sync(0xffffffffu, sum.y, 4 * (lane & 7));
            if (lane >> 3 == b) mine = make_double2(vx, vy);
        }
        if (q0 + lane < strings) {
            const double2 cf = string_factor64(op, op.offdiag[q0 + lane], s);
            const double m = exp(mine.x);
            double sn, cs;
            sincos(mine.y, &sn, &cs);
            const double2 x = make_double2(m * cs, m * sn);
            e.x += cf.x * x.x - cf.y * x.y;
            e.y += cf.x * x.y + cf.y * x.x;
        }
    }
    if (op.S > 0) e = warp_sum64(e);
    // log psi'(s) - log psi(s), angle by angle
    double2 dl = make_double2(0.0, 0.0);
    if (PP.W) {
        for (int j = lane; j < M; j += 32) lc64(angle64(PP, s, j)).add_difference(f[j], dl);
        dl = warp_sum64(dl);
    }
    if (lane == 0) {
        if (L.eloc) L.eloc[t] = e;
        if (L.logpsi) L.logpsi[t] = lp;
        if (L.dlogpsi) L.dlogpsi[t] = dl;
    }
}

__global__ void hsd_terms64_kernel(int count, const double2* __restrict__ eloc, const double2* __restrict__ dl,
                                   int is_unitary, double2* omega, double2* pr, double2* nn) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double2 e = eloc[s];
        const double dr = dl[s].x, di = -dl[s].y;   // conj(log psi' - log psi)
        double2 om;
        double n;
        if (is_unitary) {   // source/network_functions/HilbertSpaceDistance.cu:88-94
            const double m = exp(dr);
            const double ar = m * cos(di), ai = m * sin(di);
            om = make_double2(ar * e.x - ai * e.y, ar * e.y + ai * e.x);
            n = e.x * e.x + e.y * e.y;
        } else {            // :95-101
            const double m = exp(e.x + dr);
            om = make_double2(m * cos(e.y + di), m * sin(e.y + di));
            n = exp(2.0 * e.x);
        }
        omega[s] = om;
        pr[s] = make_double2(exp(2.0 * dl[s].x), 0.0);   // :102
        nn[s] = make_double2(n, 0.0);
    }
}

// per-sample gradient coefficients w_s * B_s (see capi.cu, rbmg_hsd_gradient)
__global__ void hsd_coef_kernel(int count, const double* __restrict__ w, const double2* __restrict__ omega,
                                const double2* __restrict__ pr, double2 conj_omega_bar, double v, double u,
                                double nn_bar, int mode, double scale, double2* c) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double ws = w ? w[s] : 1.0;
        const double2 om = omega[s];
        const double2 a = cmul(conj_omega_bar, om);
        double2 r;
        if (mode == 2) {
            r = make_double2(a.y, 0.0);                                  // Im(conj(<omega>) omega_s)
        } else {
            r = make_double2(a.x * v - u * nn_bar * pr[s].x, a.y * v);   // B_s
            if (mode == 1) r.y = 0.0;                                     // Re B_s
        }
        c[s] = make_double2(scale * ws * r.x, scale * ws * r.y);
    }
}

__device__ __forceinline__ double spin_of(const uint64_t* spins, uint64_t enum_base, int enumerate, long t, int N,
                                          int i) {
    const int nw = (N + 63) / 64;
    const uint64_t word = enumerate ? ((i >> 6) == 0 ? enum_base + static_cast<uint64_t>(t) : 0ull)
                                    : spins[t * nw + (i >> 6)];
    return ((word >> (i & 63)) & 1ull) ? 1.0 : -1.0;
}

__global__ void flip_each_kernel(int count, int N, const uint64_t* spins, uint64_t enum_base, int enumerate,
                                 uint64_t* out) {
    const int nw = (N + 63) / 64;
    const long total = static_cast<long>(count) * N;
    for (long q = blockIdx.x * 256L + threadIdx.x; q < total; q += static_cast<long>(gridDim.x) * 256) {
        const long t = q / N;
        const int i = static_cast<int>(q - t * N);
        for (int k = 0; k < nw; k++) {
            uint64_t w = enumerate ? (k == 0 ? enum_base + static_cast<uint64_t>(t) : 0ull) : spins[t * nw + k];
            if ((i >> 6) == k) w ^= 1ull << (i & 63);
            out[q * nw + k] = w;
        }
    }
}

__global__ void fqa_terms_kernel(int count, int N, const uint64_t* spins, uint64_t enum_base, int enumerate,
                                 const double2* lp, const double2* lpf, const double* qa, double2* dl, double2* r) {
    for (long t = blockIdx.x * 256L + threadIdx.x; t < count; t += static_cast<long>(gridDim.x) * 256) {
        const double2 l0 = lp[t];
        double cx = 0.0, cy = 0.0;
        for (int i = 0; i < N; i++) {
            const double2 li = lpf[t * N + i];
            const double m = exp(li.x - l0.x);
            const double rx = m * cos(li.y - l0.y), ry = m * sin(li.y - l0.y);
            if (r) r[t * N + i] = make_double2(rx, ry);
            const double sg = spin_of(spins, enum_base, enumerate, t, N, i);
            const double da = qa[i], db = qa[N + i], cs = qa[2 * N + i], sn = qa[3 * N + i];
            // da s_i r_i + i db (r_i cos - s_i sin)
            cx += da * sg * rx - db * (ry * cs);
            cy += da * sg * ry + db * (rx * cs - sg * sn);
        }
        dl[t] = make_double2(dl[t].x + cx, dl[t].y + cy);
    }
}

// one block per angle k (alpha_i: k = i, beta_i: k = N + i)
__global__ void fqa_grad_kernel(int count, int N, const uint64_t* spins, uint64_t enum_base, int enumerate,
                                const double2* c, const double2* r, const double* qa, double2* out) {
    __shared__ double2 red[256];
    const int k = blockIdx.x, i = k % N;
    const bool beta = k >= N;
    double ax = 0.0, ay = 0.0;
    for (long t = threadIdx.x; t < count; t += 256) {
        const double2 rv = r[t * N + i];
        const double sg = spin_of(spins, enum_base, enumerate, t, N, i);
        double ox, oy;
        if (beta) {   // i (r cos - s sin)
            ox = -(rv.y * qa[2 * N + i]);
            oy = rv.x * qa[2 * N + i] - sg * qa[3 * N + i];
        } else {      // s r
            ox = sg * rv.x;
            oy = sg * rv.y;
        }
        const double2 cv = c[t];
        // c conj(O)
        ax += cv.x * ox + cv.y * oy;
        ay += cv.y * ox - cv.x * oy;
    }
    red[threadIdx.x] = make_double2(ax, ay);
    __syncthreads();
    for (int h = 128; h >= 1; h >>= 1) {
        if (threadIdx.x < h)
            red[threadIdx.x] = make_double2(red[threadIdx.x].x + red[threadIdx.x + h].x,
                                            red[threadIdx.x].y + red[threadIdx.x + h].y);
        __syncthreads();
    }
    if (threadIdx.x == 0) out[k] = red[0];
}

}  // namespace

cudaError_t launch_flip_each(int count, int N, const uint64_t* spins, uint64_t enum_base, int enumerate,
                             uint64_t* out, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const long total = static_cast<long>(count) * N;
    flip_each_kernel<<<static_cast<int>(std::min(4096L, (total + 255) / 256)), 256, 0, st>>>(count, N, spins, enum_base,
                                                                                           enumerate, out);
    return cudaGetLastError();
}

cudaError_t launch_fqa_terms(int count, int N, const uint64_t* spins, uint64_t enum_base, int enumerate,
                             const double2* lp, const double2* lpf, const double* qa, double2* dl, double2* r,
                             cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    fqa_terms_kernel<<<static_cast<int>(std::min(1024L, (count + 255L) / 256)), 256, 0, st>>>(
        count, N, spins, enum_base, enumerate, lp, lpf, qa, dl, r);
    return cudaGetLastError();
}

cudaError_t launch_fqa_grad(int count, int N, const uint64_t* spins, uint64_t enum_base, int enumerate,
                            const double2* c, const double2* r, const double* qa, double2* out, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    fqa_grad_kernel<<<2 * N, 256, 0, st>>>(count, N, spins, enum_base, enumerate, c, r, qa, out);
    return cudaGetLastError();
}

size_t rbm_table64_bytes(int N, int M) {
    return sizeof(double2) * static_cast<size_t>((N + kTab64Spins - 1) / kTab64Spins) * kTab64Size * M;
}

cudaError_t launch_rbm_table64(const Rbm64& P, double2* tab, cudaStream_t st) {
    const long total = static_cast<long>(rbm_table64_bytes(P.N, P.M) / sizeof(double2));
    table64_kernel<<<static_cast<int>(std::min(4096L, (total + 255) / 256)), 256, 0, st>>>(P, tab);
    return cudaGetLastError();
}

cudaError_t launch_rbm_hsd64(const Rbm64& P, const Rbm64& PP, const OpDev& op, const Hsd64Launch& L,
                             cudaStream_t st) {
    if (L.count <= 0) return cudaSuccess;
    const size_t smem = sizeof(double2) * 2 * P.M * kWarpsPerBlock;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(rbm_hsd64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    rbm_hsd64_kernel<<<(L.count + kWarpsPerBlock - 1) / kWarpsPerBlock, 32 * kWarpsPerBlock, smem, st>>>(P, PP, op, L);
    return cudaGetLastError();
}

// second order (HilbertSpaceDistance_2nd_order.cu:44-60): x = E1 + (E2 - E1^2) / 2,
// omega = exp(x + conj(log psi' - log psi)), norm = exp(2 Re x), ratio = exp(2 Re(log psi' - log psi))
__global__ void hsd2_terms64_kernel(int count, const double2* __restrict__ e1, const double2* __restrict__ e2,
                                    const double2* __restrict__ dl, double2* omega, double2* pr, double2* nn) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double2 a = e1[s], b = e2[s];
        const double xr = a.x + 0.5 * (b.x - (a.x * a.x - a.y * a.y));
        const double xi = a.y + 0.5 * (b.y - 2.0 * a.x * a.y);
        const double m = exp(xr + dl[s].x);
        const double ph = xi - dl[s].y;
        omega[s] = make_double2(m * cos(ph), m * sin(ph));
        nn[s] = make_double2(exp(2.0 * xr), 0.0);
        pr[s] = make_double2(exp(2.0 * dl[s].x), 0.0);
    }
}

cudaError_t launch_hsd2_terms64(int count, const double2* e1, const double2* e2, const double2* dl, double2* omega,
                                double2* pr, double2* nn, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const int blocks = std::min((count + 255) / 256, 4096);
    hsd2_terms64_kernel<<<blocks, 256, 0, st>>>(count, e1, e2, dl, omega, pr, nn);
    return cudaGetLastError();
}

cudaError_t launch_hsd_terms64(int count, const double2* eloc, const double2* dl, int is_unitary, double2* omega,
                               double2* pr, double2* nn, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    hsd_terms64_kernel<<<static_cast<int>(std::min(1024L, (count + 255L) / 256)), 256, 0, st>>>(
        count, eloc, dl, is_unitary, omega, pr, nn);
    return cudaGetLastError();
}

cudaError_t launch_hsd_coef(int count, const double* w, const double2* omega, const double2* pr,
                            double2 conj_omega_bar, double v, double u, double nn_bar, int mode, double scale,
                            double2* c, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    hsd_coef_kernel<<<static_cast<int>(std::min(1024L, (count + 255L) / 256)), 256, 0, st>>>(
        count, w, omega, pr, conj_omega_bar, v, u, nn_bar, mode, scale, c);
    return cudaGetLastError();
}

}  // namespace rbmg
