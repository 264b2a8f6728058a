// Deterministic reductions of per-sample quantities into the estimator sums.
//
// All sums over samples run in a fixed order: FP32 partial sums over chunks of at
// most 32 samples, accumulated in FP64, then the blocks' partials in a fixed order: those of the
// outer sums by a second kernel, split by split; those of the weighted sums of series by the block
// that arrives last, each lane its own blocks in order and the lanes by a butterfly.  No
// floating-point atomics, so results are bit-reproducible run to run.
#include <algorithm>

#include "device_math.cuh"
#include "kernels.h"
#include "reduce.h"

namespace rbmg {

namespace {

constexpr int kChunk = 32;

__device__ __forceinline__ float spin_sign(const uint64_t* spins, uint64_t enum_base, int enumerate, long s, int nw,
                                           int i) {
    uint64_t word;
    if (enumerate) {
        const uint64_t idx = enum_base + static_cast<uint64_t>(s);
        word = (i >> 6) == 0 ? idx : 0ull;
    } else {
        word = spins[s * nw + (i >> 6)];
    }
    return ((word >> (i & 63)) & 1ull) ? 1.0f : -1.0f;
}

// NC outer-product sums over the same rows A: out_q[r][j] = sum_s c_q[s] f_q(A[s][j]) g_r(s).
// Grid (ceil(M/32), row tiles, splits), block (32, T): thread (tx, ty) owns column
// j = 32 bx + tx and rows 4 (T by + ty) .. + 3 of every sum, so that a sample's row, its signs
// and its coefficients are read once for 4 NC products (one sum and two rows a thread before:
// five launches of 20 us for the sums of 4096 samples at N = 64, M = 128, together 102 us; now two of 55 and 18).  FP32 sums of
// 32 samples, added up in FP64, whose pipe they keep busy half of the time.
constexpr int kOmRows = 4, kOmMaxTy = 17;

template <int NC>
__global__ void __launch_bounds__(32 * kOmMaxTy) outer_reduce_kernel(
    int count, int N, int nw, int M, const uint64_t* __restrict__ spins, uint64_t enum_base, int enumerate,
    OuterSet set, const float2* __restrict__ A, int lda, double2* __restrict__ partial, int per_split) {
    __shared__ float2 sA[kChunk][32];
    __shared__ float2 sC[kChunk][NC];
    __shared__ __align__(16) float sSign[kChunk][kOmRows * kOmMaxTy];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int threads = 32 * blockDim.y, rows = kOmRows * blockDim.y;
    const int j = blockIdx.x * 32 + tx;
    const long s_begin = static_cast<long>(blockIdx.z) * per_split;
    const long s_end = min(static_cast<long>(count), s_begin + per_split);
    double2 acc[NC][kOmRows];
#pragma unroll
    for (int q = 0; q < NC; q++)
#pragma unroll
        for (int r = 0; r < kOmRows; r++) acc[q][r] = make_double2(0.0, 0.0);
    const int tid = ty * 32 + tx;
    for (long base = s_begin; base < s_end; base += kChunk) {
        const int n = static_cast<int>(min(static_cast<long>(kChunk), s_end - base));
        __syncthreads();
        for (int e = tid; e < kChunk * 32; e += threads) {
            const int ss = e / 32, jj = blockIdx.x * 32 + e % 32;
            sA[ss][e % 32] = ss < n && jj < M ? A[(base + ss) * lda + jj] : make_float2(0.0f, 0.0f);
        }
        for (int e = tid; e < kChunk * NC; e += threads) {
            const int ss = e / NC;
            const double2 cc = ss < n ? set.c[e % NC][base + ss] : make_double2(0.0, 0.0);
            sC[ss][e % NC] = make_float2(static_cast<float>(cc.x), static_cast<float>(cc.y));
        }
        for (int e = tid; e < kChunk * rows; e += threads) {
            const int ss = e / rows, rr = blockIdx.y * rows + e % rows;
            float sg = 0.0f;
            if (ss < n && rr <= N) sg = rr == 0 ? 1.0f : spin_sign(spins, enum_base, enumerate, base + ss, nw, rr - 1);
            sSign[ss][e % rows] = sg;
        }
        __syncthreads();
        float2 p[NC][kOmRows];
#pragma unroll
        for (int q = 0; q < NC; q++)
#pragma unroll
            for (int r = 0; r < kOmRows; r++) p[q][r] = make_float2(0.0f, 0.0f);
#pragma unroll 2
        for (int ss = 0; ss < n; ss++) {
            const float2 a = sA[ss][tx];
            const float4 g4 = *reinterpret_cast<const float4*>(&sSign[ss][kOmRows * ty]);
            const float g[kOmRows] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
            for (int q = 0; q < NC; q++) {
                const float2 cc = sC[ss][q];
                const float ay = set.conj[q] ? -a.y : a.y;
                const float vx = __fmaf_rn(cc.x, a.x, -__fmul_rn(cc.y, ay));
                const float vy = __fmaf_rn(cc.x, ay, __fmul_rn(cc.y, a.x));
#pragma unroll
                for (int r = 0; r < kOmRows; r++) {
                    p[q][r].x = fmaf(g[r], vx, p[q][r].x);
                    p[q][r].y = fmaf(g[r], vy, p[q][r].y);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NC; q++)
#pragma unroll
            for (int r = 0; r < kOmRows; r++) {
                acc[q][r].x += p[q][r].x;
                acc[q][r].y += p[q][r].y;
            }
    }
    if (j >= M) return;
    const long plane = static_cast<long>(1 + N) * M;
#pragma unroll
    for (int q = 0; q < NC; q++)
#pragma unroll
        for (int r = 0; r < kOmRows; r++) {
            const int row = blockIdx.y * rows + kOmRows * ty + r;
            if (row <= N) partial[(static_cast<long>(blockIdx.z) * NC + q) * plane + static_cast<long>(row) * M + j] = acc[q][r];
        }
}

// SplitSum, blockIdx.y the job: a block takes 32 entries, eight slices of the splits, each in z
// order with its loads in flight together, then the slices in order (one thread an entry walked
// the 64 splits of 8320 sums in 12.5 us; now 25000 take 10).  The sums of one pass go together:
// three launches of 4 us each were a sixth of the GPU's work for 4096 states of 12 spins.
struct SplitSums {
    SplitSum job[2];
};
__global__ void __launch_bounds__(256) finish_splits_kernel(SplitSums jobs, int add) {
    __shared__ double2 red[2][8][32];
    const SplitSum& J = jobs.job[blockIdx.y];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const long total = J.elems * J.nc;
    auto slice_sum = [&](const double2* partial, int splits, long stride, long e) {
        double2 a = make_double2(0.0, 0.0);
        const int per = (splits + 7) / 8, z1 = min(splits, (slice + 1) * per);
#pragma unroll 8
        for (int z = slice * per; z < z1; z++) {
            const double2 p = partial[z * stride + e];
            a.x += p.x;
            a.y += p.y;
        }
        return a;
    };
    for (long e0 = blockIdx.x * 32L; e0 < total; e0 += gridDim.x * 32L) {
        const long e = e0 + lane;
        const bool pre = J.pre && e < J.elems;
        if (e < total) red[0][slice][lane] = slice_sum(J.partial, J.splits, total, e);
        if (pre) red[1][slice][lane] = slice_sum(J.pre, J.pre_splits, J.elems, e);
        __syncthreads();
        if (slice == 0 && e < total) {
            double2* out = J.out[e / J.elems] + e % J.elems;
            double2 o = add ? *out : make_double2(0.0, 0.0);
            auto slices = [&](int k, double scale) {
                double2 a = red[k][0][lane];
                for (int q = 1; q < 8; q++) {
                    a.x += red[k][q][lane].x;
                    a.y += red[k][q][lane].y;
                }
                o.x += scale * a.x;
                o.y += scale * a.y;
            };
            if (pre) slices(1, -2.0);
            slices(0, J.scale);
            *out = o;
        }
        __syncthreads();
    }
}

// grid (ceil(M/32), N, splits), block 256 = 8 warps; warp w takes samples w, w+8, ...
__global__ void vterm_kernel(int count, int N, int nw, int M, int Mpad, const uint64_t* __restrict__ spins,
                             uint64_t enum_base, int enumerate, const double* __restrict__ w,
                             const double2* __restrict__ cw, const float2* __restrict__ X, int num_offdiag,
                             const int* __restrict__ site_ptr, const int* __restrict__ site_slots,
                             double2* __restrict__ partial, int per_split) {
    __shared__ double2 red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    const int i = blockIdx.y;
    const int sb = site_ptr[i], se = site_ptr[i + 1];
    const long s_begin = static_cast<long>(blockIdx.z) * per_split;
    const long s_end = min(static_cast<long>(count), s_begin + per_split);
    double2 acc = make_double2(0.0, 0.0);
    float2 part = make_float2(0.0f, 0.0f);
    int in_chunk = 0;
    if (se > sb && j < Mpad) {
        for (long s = s_begin + warp; s < s_end; s += 8) {
            const float g = spin_sign(spins, enum_base, enumerate, s, nw, i) * (w ? static_cast<float>(w[s]) : 1.0f);
            float2 x = make_float2(0.0f, 0.0f);
            for (int q = sb; q < se; q++) {
                const float2 v = X[(s * num_offdiag + site_slots[q]) * Mpad + j];
                x.x += v.x;
                x.y += v.y;
            }
            if (cw) {   // complex per-sample coefficient
                const float cr = static_cast<float>(cw[s].x), ci = static_cast<float>(cw[s].y);
                x = make_float2(cr * x.x - ci * x.y, cr * x.y + ci * x.x);
            }
            part.x = fmaf(g, x.x, part.x);
            part.y = fmaf(g, x.y, part.y);
            if (++in_chunk == kChunk) {
                acc.x += part.x; acc.y += part.y;
                part = make_float2(0.0f, 0.0f);
                in_chunk = 0;
            }
        }
    }
    acc.x += part.x;
    acc.y += part.y;
    red[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && j < M) {
        double2 t = make_double2(0.0, 0.0);
        for (int q = 0; q < 8; q++) { t.x += red[q][lane].x; t.y += red[q][lane].y; }
        const long plane = static_cast<long>(1 + N) * M;
        partial[blockIdx.z * plane + static_cast<long>(1 + i) * M + j] = t;
    }
    if (warp == 0 && i == 0 && j < M) {
        const long plane = static_cast<long>(1 + N) * M;
        partial[blockIdx.z * plane + j] = make_double2(0.0, 0.0);   // row 0 carries no V term
    }
}

// U and the V sums of a single-flip operator from the angles and the terms e_n (GradVectors).
// tanh(theta'') is evaluated again here instead of being stored by the pass that forms the e_n:
// per sample and string that is a second activation of every unit against 16 bytes written and
// read (268 MB a 4096-sample chunk at N = 64, M = 128).
// A unit of work is chunk c of split z of a group: warp q takes samples z per_split + q + 8 k
// (k < 32 of the chunk), its lanes 32 hidden units: vterm_kernel's FP32 sums, one by one in its
// order, added up in FP64 over the block's warps and units.  The strings go by eight in the
// operator's order, so that every U_j is the same ordered sum; a block's terms and
// signs are staged in shared memory, two samples side by side for the packed operations.  A
// thread holds eight V sums; its samples' U are in shared memory between blocks of strings.
// Bound by the FP32 pipe (57 lane operations per sample, string and unit; half of its cycles) and
// the latency of its reads of shared memory: four samples in flight and three blocks an SM walking
// the units, 2.57 ms for 81920 samples at N = 64, M = 128; eight samples and two blocks 2.85, and
// with a launch and 256 blocks per 4096 samples, which left a sixth of the SMs' places empty, 3.6;
// vterm_kernel on stored terms 7.1.
constexpr int kGvStrings = 8, kGvTile = 4, kGvWarps = 8;

// vterm_kernel's split of a group's samples, and chunks of 32 samples a warp
__host__ __device__ inline void grad_vectors_shape(int count, int max_splits, int* per_split, int* splits, int* chunks,
                                                   int* cap) {
    const int even = (count + max_splits - 1) / max_splits;
    *per_split = even > 64 ? even : 64;
    *splits = (count + *per_split - 1) / *per_split;
    const int per_warp = (*per_split + 7) / 8, two = (per_warp + 1) / 2 * 2;
    *chunks = (per_warp + 31) / 32;
    *cap = two < 32 ? two : 32;
}

// ONE: a lane of the general pass holds one hidden unit (Mpad = 32); its compiled form joins the
// other product of Im(e tanh) into an FMA than with more units, and so does this one.
template <bool ONE>
__global__ void __launch_bounds__(32 * kGvWarps, 3) grad_vectors_kernel(GradVectors g, OpDev op, int per_group,
                                                                     int units, int cap, double2* partial) {
    extern __shared__ __align__(16) unsigned char gv_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pairs = cap / 2;
    // [warp][string][pair] (ex0, ex1, ey0, ey1) and (2 s'0, 2 s'1, g0, g1)
    float4* stA = reinterpret_cast<float4*>(gv_smem) + warp * 2 * kGvStrings * pairs;
    float4* stB = stA + kGvStrings * pairs;
    float2* red = reinterpret_cast<float2*>(reinterpret_cast<float4*>(gv_smem) + kGvWarps * 2 * kGvStrings * pairs);
    pair_t* us = reinterpret_cast<pair_t*>(red + kGvStrings * kGvWarps * 32) + warp * 2 * pairs * 32 + lane;
    const int j = blockIdx.x * 32 + lane;
    const int nw = g.nw;
    double2* out = partial + static_cast<long>(blockIdx.y) * (1 + g.N) * g.M;
    for (int i = warp; i <= g.N; i += kGvWarps)   // the rows no string writes
        if (j < g.M && (i == 0 || g.site_ptr[i - 1] == g.site_ptr[i])) out[static_cast<long>(i) * g.M + j] = make_double2(0.0, 0.0);
    for (int unit = blockIdx.y; unit < units; unit += gridDim.y) {
    const int group0 = unit / per_group * g.group, in_group = min(g.group, g.count - group0);
    int per_split, splits, chunks, cap_g;
    grad_vectors_shape(in_group, g.max_splits, &per_split, &splits, &chunks, &cap_g);
    const int z = unit % per_group / chunks, c = unit % per_group - z * chunks;
    const int s_end = group0 + min(in_group, (z + 1) * per_split);
    const int s0 = group0 + z * per_split + warp + 8 * 32 * c;
    const int cnt = s0 < s_end ? min(32, (s_end - s0 + 7) / 8) : 0;   // sample k of the warp: s0 + 8 k
    for (int q = 0; q < pairs; q++) us[(2 * q) * 32] = us[(2 * q + 1) * 32] = splat2(0.0f);
    auto word = [&](int s, int k) -> uint64_t {
        if (!g.enumerate) return k < nw ? g.spins[static_cast<long>(s) * nw + k] : 0ull;
        if (k != 0) return 0ull;
        const uint64_t idx = g.enum_base + static_cast<uint64_t>(s);
        return g.N >= 64 ? idx : (idx & ((1ull << g.N) - 1ull));
    };
    auto load = [&](const float2* a, int k) {
        return k < cnt ? a[static_cast<long>(s0 + 8 * k) * g.Mpad + j] : make_float2(0.0f, 0.0f);
    };
    for (int n0 = 0; n0 < op.S;) {
        // up to eight consecutive strings of one kind
        const bool diag = op.nflip[n0] == 0;
        int nb = 1;
        while (nb < kGvStrings && n0 + nb < op.S && (op.nflip[n0 + nb] == 0) == diag) nb++;
        __syncwarp();
        for (int e = lane; e < kGvStrings * 2 * pairs; e += 32) {
            const int u = e % kGvStrings, k = e / kGvStrings, n = n0 + u;
            float2 en = make_float2(0.0f, 0.0f);
            float ts = 0.0f, gw = 0.0f;
            if (u < nb && k < cnt) {
                const int s = s0 + 8 * k;
                if (diag) {
                    // string_factor of this sample
                    int parity = 0;
                    for (int q = 0; q < nw; q++) parity += __popcll(op.zmask[n * kMaxWords + q] & ~word(s, q));
                    const float2 cf = op.coef32[n];
                    const int yp = op.ypow[n] & 3;
                    en = yp == 0 ? cf : (yp == 1 ? make_float2(cf.y, -cf.x)
                                                 : (yp == 2 ? make_float2(-cf.x, -cf.y) : make_float2(-cf.y, cf.x)));
                    if (parity & 1) en = make_float2(-en.x, -en.y);
                } else {
                    const int site = op.flip_sites[op.flip_off[n]];
                    const bool up = (word(s, site >> 6) >> (site & 63)) & 1ull;
                    en = g.en[static_cast<long>(s) * op.num_offdiag + op.offdiag_slot[n]];
                    ts = up ? -2.0f : 2.0f;
                    gw = (up ? 1.0f : -1.0f) * (g.w ? static_cast<float>(g.w[s]) : 1.0f);
                }
            }
            float* a = reinterpret_cast<float*>(stA + u * pairs + (k >> 1)) + (k & 1);
            float* b = reinterpret_cast<float*>(stB + u * pairs + (k >> 1)) + (k & 1);
            a[0] = en.x;
            a[2] = en.y;
            b[0] = ts;
            b[2] = gw;
        }
        __syncwarp();
        if (diag) {
            for (int k0 = 0; k0 < cnt; k0 += kGvTile) {
#pragma unroll
                for (int v = 0; v < kGvTile / 2; v++) {
                    const int q = (k0 >> 1) + v;
                    if (q >= pairs) break;
                    const float2 a0 = load(g.T, 2 * q), a1 = load(g.T, 2 * q + 1);
                    const pair_t tx = pk2(a0.x, a1.x), ty = pk2(a0.y, a1.y);
                    const pair_t nty = neg2(ty);
                    pair_t ur = us[(2 * q) * 32], ui = us[(2 * q + 1) * 32];
                    for (int u = 0; u < nb; u++) {
                        const float4 e = stA[u * pairs + q];
                        const pair_t ex = pk2(e.x, e.y), ey = pk2(e.z, e.w);
                        ur = add2(ur, fma2(ex, tx, mul2(ey, nty)));
                        ui = add2(ui, fma2(ex, ty, mul2(ey, tx)));
                    }
                    us[(2 * q) * 32] = ur;
                    us[(2 * q + 1) * 32] = ui;
                }
            }
        } else {
            float2 w[kGvStrings], V[kGvStrings];
#pragma unroll
            for (int u = 0; u < kGvStrings; u++) {
                w[u] = make_float2(0.0f, 0.0f);
                V[u] = make_float2(0.0f, 0.0f);
                if (u < nb)
                    w[u] = __ldg(g.W + static_cast<long>(op.flip_sites[op.flip_off[n0 + u]]) * g.Mpad + j);
            }
            for (int k0 = 0; k0 < cnt; k0 += kGvTile) {
                pair_t tr[kGvTile / 2], ti[kGvTile / 2], ur[kGvTile / 2], ui[kGvTile / 2];
#pragma unroll
                for (int v = 0; v < kGvTile / 2; v++) {
                    const int q = min((k0 >> 1) + v, pairs - 1);
                    const float2 a0 = load(g.theta, k0 + 2 * v), a1 = load(g.theta, k0 + 2 * v + 1);
                    tr[v] = pk2(a0.x, a1.x);
                    ti[v] = pk2(a0.y, a1.y);
                    ur[v] = us[(2 * q) * 32];
                    ui[v] = us[(2 * q + 1) * 32];
                }
#pragma unroll
                for (int u = 0; u < kGvStrings; u++) {
                    if (u >= nb) break;
                    const pair_t wx = splat2(w[u].x), wy = splat2(w[u].y);
#pragma unroll
                    for (int v = 0; v < kGvTile / 2; v++) {
                        const int q = min((k0 >> 1) + v, pairs - 1);
                        const float4 e = stA[u * pairs + q], b = stB[u * pairs + q];
                        const pair_t ts = pk2(b.x, b.y);
                        const Pair2 h = tanh2_approx(fma2(ts, wx, tr[v]), fma2(ts, wy, ti[v]));
                        const pair_t ex = pk2(e.x, e.y), ey = pk2(e.z, e.w);
                        const pair_t vx = fma2(ex, h.re, neg2(mul2(ey, h.im)));
                        const pair_t vy = ONE ? fma2(ex, h.im, mul2(ey, h.re)) : fma2(ey, h.re, mul2(ex, h.im));
                        ur[v] = add2(ur[v], vx);
                        ui[v] = add2(ui[v], vy);
                        if (k0 + 2 * v < cnt) {
                            float x0, x1, y0, y1;
                            up2(vx, x0, x1);
                            up2(vy, y0, y1);
                            V[u].x = fmaf(b.z, x0, V[u].x);
                            V[u].y = fmaf(b.z, y0, V[u].y);
                            V[u].x = fmaf(b.w, x1, V[u].x);
                            V[u].y = fmaf(b.w, y1, V[u].y);
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < kGvTile / 2; v++) {
                    const int q = (k0 >> 1) + v;
                    if (q < pairs) {
                        us[(2 * q) * 32] = ur[v];
                        us[(2 * q + 1) * 32] = ui[v];
                    }
                }
            }
            __syncthreads();   // the previous block's sums have been read
#pragma unroll
            for (int u = 0; u < kGvStrings; u++) red[(u * kGvWarps + warp) * 32 + lane] = V[u];
            __syncthreads();
            if (warp < nb && j < g.M) {
                double2 t = make_double2(0.0, 0.0);
                for (int q = 0; q < kGvWarps; q++) {
                    const float2 v = red[(warp * kGvWarps + q) * 32 + lane];
                    t.x += v.x;
                    t.y += v.y;
                }
                const int site = op.flip_sites[op.flip_off[n0 + warp]];
                double2* o = out + static_cast<long>(1 + site) * g.M + j;
                if (unit != blockIdx.y) {   // the block's earlier units
                    t.x += o->x;
                    t.y += o->y;
                }
                *o = t;
            }
        }
        n0 += nb;
    }
    const float shx = static_cast<float>(g.e_shift->x), shy = static_cast<float>(g.e_shift->y);
    for (int k = 0; k < cnt; k++) {
        const float2 t = load(g.T, k);
        float x[2], y[2];
        up2(us[(2 * (k >> 1)) * 32], x[0], x[1]);
        up2(us[(2 * (k >> 1) + 1) * 32], y[0], y[1]);
        float2 u = make_float2(x[k & 1], y[k & 1]);
        u.x -= __fmaf_rn(shx, t.x, -__fmul_rn(shy, t.y));
        u.y -= __fmaf_rn(shx, t.y, __fmul_rn(shy, t.x));
        g.U[static_cast<long>(s0 + 8 * k) * g.Mpad + j] = u;
    }
    }
}

// ---- weighted sums of complex series -------------------------------------
// The block's sums of n series go to block_out; the block that arrives last adds up all blocks'
// in a fixed order (warp q series q: lane l blocks l, l + 32, ..., then a butterfly) into total,
// and returns true.  A second launch of one thread per series walked 512 blocks in 26 us.
constexpr int kSumThreads = 256;
static_assert(kSumThreads / 32 >= kMaxSeries, "a warp per series");
__device__ bool block_totals(double2 (&acc)[kMaxSeries], int n, double2* block_out, double2 (&total)[kMaxSeries]) {
    __shared__ double2 red[kMaxSeries][kSumThreads / 32];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto warp_sum = [](double2 v) {
        for (int off = 16; off >= 1; off >>= 1) {
            v.x += __shfl_down_sync(0xffffffffu, v.x, off);
            v.y += __shfl_down_sync(0xffffffffu, v.y, off);
        }
        return v;
    };
#pragma unroll
    for (int q = 0; q < kMaxSeries; q++)
        if (q < n) {
            const double2 t = warp_sum(acc[q]);
            if (lane == 0) red[q][warp] = t;
        }
    __syncthreads();
    if (tid < n) {
        double2 t = make_double2(0.0, 0.0);
        for (int q = 0; q < kSumThreads / 32; q++) { t.x += red[tid][q].x; t.y += red[tid][q].y; }
        block_out[blockIdx.x * kMaxSeries + tid] = t;
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) {
        unsigned int* ticket = reinterpret_cast<unsigned int*>(block_out + kSumBlocks * kMaxSeries);
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;   // back to zero after the last block
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    if (warp < n) {
        double2 t = make_double2(0.0, 0.0);
        for (int b = lane; b < gridDim.x; b += 32) {
            const double2 v = __ldcg(block_out + b * kMaxSeries + warp);
            t.x += v.x;
            t.y += v.y;
        }
        t = warp_sum(t);
        if (lane == 0) red[warp][0] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kMaxSeries; q++) total[q] = q < n ? red[q][0] : make_double2(0.0, 0.0);
    return true;
}

// MEAN: the mean of set.v[0] (sums of w v and w); otherwise sums[q] += the sums of w v_q
template <bool MEAN>
__global__ void __launch_bounds__(kSumThreads) wsum_kernel(int count, const double* __restrict__ w, SeriesSet set,
                                                           double2* block_out, double2* sums) {
    double2 acc[kMaxSeries], total[kMaxSeries];
#pragma unroll
    for (int q = 0; q < kMaxSeries; q++) acc[q] = make_double2(0.0, 0.0);
    for (long s = blockIdx.x * long(kSumThreads) + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * kSumThreads) {
        const double ws = w ? w[s] : 1.0;
#pragma unroll
        for (int q = 0; q < kMaxSeries; q++)
            if (q < (MEAN ? 1 : set.n)) {
                const double2 v = set.v[q][s];
                acc[q].x += ws * v.x;
                acc[q].y += ws * v.y;
            }
        if (MEAN) acc[1].x += ws;
    }
    if (!block_totals(acc, MEAN ? 2 : set.n, block_out, total)) return;
    if (MEAN) {
        const double wt = total[1].x;
        if (threadIdx.x == 0)
            sums[0] = wt > 0.0 ? make_double2(total[0].x / wt, total[0].y / wt) : make_double2(0.0, 0.0);
    } else {
#pragma unroll
        for (int q = 0; q < kMaxSeries; q++)
            if (threadIdx.x == q && q < set.n) {
                sums[q].x += total[q].x;
                sums[q].y += total[q].y;
            }
    }
}

// ---- weights of exact summation: the largest 2 Re log psi, the sum over exp(2 Re log psi - m),
// the weights; on the device from end to end (a maximum and a sum taken through the host put two
// waits of 25 us each before the first weight)
__global__ void __launch_bounds__(kSumThreads) exact_max_kernel(int count, const double2* __restrict__ lp,
                                                                double2* block_out, double2* stat) {
    __shared__ double red[kSumThreads];
    __shared__ bool last;
    auto block_max = [&](double m) {
        red[threadIdx.x] = m;
        __syncthreads();
        for (int h = kSumThreads / 2; h >= 1; h >>= 1) {
            if (threadIdx.x < h) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + h]);
            __syncthreads();
        }
        return red[0];
    };
    double m = -INFINITY;
    for (long s = blockIdx.x * long(kSumThreads) + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * kSumThreads)
        m = fmax(m, 2.0 * lp[s].x);
    m = block_max(m);
    if (threadIdx.x == 0) {
        block_out[blockIdx.x].x = m;
        __threadfence();
        unsigned int* ticket = reinterpret_cast<unsigned int*>(block_out + kSumBlocks * kMaxSeries);
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    m = -INFINITY;
    for (int b = threadIdx.x; b < gridDim.x; b += kSumThreads) m = fmax(m, __ldcg(&block_out[b].x));
    m = block_max(m);
    if (threadIdx.x == 0) stat[0].x = m;
}

__global__ void __launch_bounds__(kSumThreads) exact_norm_kernel(int count, const double2* __restrict__ lp,
                                                                 double2* block_out, double2* stat) {
    double2 acc[kMaxSeries], total[kMaxSeries];
#pragma unroll
    for (int q = 0; q < kMaxSeries; q++) acc[q] = make_double2(0.0, 0.0);
    const double m = stat[0].x;
    for (long s = blockIdx.x * long(kSumThreads) + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * kSumThreads)
        acc[0].x += exp(2.0 * lp[s].x - m);
    if (!block_totals(acc, 1, block_out, total)) return;
    if (threadIdx.x == 0) {
        stat[0].y = total[0].x;
        stat[1].x = m + log(total[0].x);
    }
}

__global__ void exact_weights_kernel(int count, const double2* __restrict__ lp, const double2* __restrict__ stat,
                                     double* w) {
    const double log_z = stat[1].x;
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256)
        w[s] = exp(2.0 * lp[s].x - log_z);
}

// ---- elementwise per-sample coefficients ---------------------------------
__global__ void max_re2_kernel(int count, const double2* __restrict__ lp, double* block_max) {
    __shared__ double red[256];
    double m = -INFINITY;
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256)
        m = fmax(m, 2.0 * lp[s].x);
    red[threadIdx.x] = m;
    __syncthreads();
    for (int h = 128; h >= 1; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + h]);
        __syncthreads();
    }
    if (threadIdx.x == 0) block_max[blockIdx.x] = red[0];
}

__global__ void exp_weights_kernel(int count, const double2* __restrict__ lp, double shift, double* w) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256)
        w[s] = exp(2.0 * lp[s].x - shift);
}

__global__ void coef_kernel(int count, const double* __restrict__ w, const double2* __restrict__ v, double scale,
                            double2 shift, double2* c) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double ws = (w ? w[s] : 1.0) * scale;
        c[s] = v ? make_double2(ws * (v[s].x - shift.x), ws * (v[s].y - shift.y)) : make_double2(ws, 0.0);
    }
}

// c[s] = w[s] conj(v[s] - shift)
__global__ void coef_conj_kernel(int count, const double* __restrict__ w, const double2* __restrict__ v,
                                 double2 shift, double2* c) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double ws = w ? w[s] : 1.0;
        c[s] = make_double2(ws * (v[s].x - shift.x), -ws * (v[s].y - shift.y));
    }
}

// launch_grad_coefs: one pass over the samples (two or three launches before)
__global__ void grad_coefs_kernel(int count, const double* __restrict__ w, const double2* __restrict__ v,
                                  const double2* __restrict__ shift, double2* c1, double2* c2, double2* c3,
                                  int conj3) {
    const double2 sh = *shift;
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double ws = w ? w[s] : 1.0;
        const double x = ws * (v[s].x - sh.x), y = ws * (v[s].y - sh.y);
        c1[s] = make_double2(ws, 0.0);
        c2[s] = make_double2(x, y);
        if (c3) c3[s] = make_double2(x, conj3 ? -y : 0.0);
    }
}

// launch_grad_out.  Estimator (ExpectationValue.cu:243-253): grad = <E O*> + conj<E_k> - 2 <E> <O*>,
// from the centred sums EO' = sum w (E - E0) O*, Ek' = sum w (E_k - E0 O):
//   grad = EO' + conj(Ek') + (E0 + conj(E0) - 2 <E>) conj<O>   (all sums times the factor).
// Derivative of <E_loc>: conj(C1 - C2) and, with the sampling term, + 2 (C3 - (<Re E> - Re E0) <O>*).
// Formed here, the result is one copy; four or five copies and the host's loop were 60 to 100 us
// of a call.
__global__ void grad_out_kernel(GradOut g) {
    const long k = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < g.first) g.grad[k] = make_double2(0.0, 0.0);
    const double f = g.stat ? exp(g.norm + g.stat[1].x) : g.norm;
    const double2 E0 = *g.e0;
    const double Er = __dmul_rn(g.sums[0].x, f), Ei = __dmul_rn(g.sums[0].y, f);
    if (k == 0) {
        g.status[0] = Er;
        g.status[1] = Ei;
        g.status[2] = f;
        g.status[3] = g.stat ? g.stat[0].x : 0.0;
    }
    if (k >= g.count) return;
    auto scaled = [&](const double2* p) { return make_double2(__dmul_rn(p[k].x, f), __dmul_rn(p[k].y, f)); };
    const double2 o = scaled(g.O), a = scaled(g.A), b = scaled(g.B);
    double2 v;
    if (g.mode == 0) {
        const double sr = __dsub_rn(__dadd_rn(E0.x, E0.x), __dmul_rn(2.0, Er));
        const double si = __dsub_rn(__dsub_rn(E0.y, E0.y), __dmul_rn(2.0, Ei));
        // shift * conj(o) = (sr + i si)(o.x - i o.y)
        const double tr = __dadd_rn(__dmul_rn(sr, o.x), __dmul_rn(si, o.y));
        const double ti = __dsub_rn(__dmul_rn(si, o.x), __dmul_rn(sr, o.y));
        v = make_double2(__dadd_rn(__dadd_rn(a.x, b.x), tr), __dadd_rn(__dsub_rn(a.y, b.y), ti));
    } else {
        v = make_double2(__dsub_rn(a.x, b.x), -__dsub_rn(a.y, b.y));
        if (g.mode == 2) {
            const double2 c = scaled(g.C);
            const double dre = __dsub_rn(Er, E0.x);
            v.x = __dadd_rn(v.x, __dmul_rn(2.0, __dsub_rn(c.x, __dmul_rn(dre, o.x))));
            v.y = __dadd_rn(v.y, __dmul_rn(2.0, __dadd_rn(c.y, __dmul_rn(dre, o.y))));
        }
    }
    g.grad[g.first + k] = v;
}

// rw[s] = w[s] exp(2 (Re lp[s] - Re lpp[s])) (ExpectationValue.cu:391-395), rwc[s] = (rw[s], 0)
__global__ void ratio_weight_kernel(int count, const double* __restrict__ w, const double2* __restrict__ lp,
                                    const double2* __restrict__ lpp, double* rw, double2* rwc) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double r = (w ? w[s] : 1.0) * exp(2.0 * (lp[s].x - lpp[s].x));
        rw[s] = r;
        rwc[s] = make_double2(r, 0.0);
    }
}

// a[s] = exp(2 Im E + Re(E E - E)) (ExpectationValue.cu:106-109)
__global__ void corrected_kernel(int count, const double2* __restrict__ e, double2* a) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256) {
        const double2 v = e[s];
        a[s] = make_double2(exp(2.0 * v.y + (v.x * v.x - v.y * v.y - v.x)), 0.0);
    }
}

__global__ void abs2_kernel(int count, const double2* __restrict__ v, double2* out) {
    for (long s = blockIdx.x * 256L + threadIdx.x; s < count; s += static_cast<long>(gridDim.x) * 256)
        out[s] = make_double2(v[s].x * v[s].x + v[s].y * v[s].y, 0.0);
}

inline int grid_for(long count) { return static_cast<int>(min(1024L, max(1L, (count + 255) / 256))); }

}  // namespace

cudaError_t launch_split_sums(const SplitSum* jobs, int n, bool add, cudaStream_t st) {
    if (n < 1 || n > 2) return cudaErrorInvalidValue;
    SplitSums set{};
    long most = 0;
    for (int q = 0; q < n; q++) {
        set.job[q] = jobs[q];
        most = max(most, jobs[q].elems * jobs[q].nc);
    }
    const dim3 grid(static_cast<int>(min(4096L, (most + 31) / 32)), n);
    finish_splits_kernel<<<grid, 256, 0, st>>>(set, add ? 1 : 0);
    return cudaGetLastError();
}

static int outer_per_split(int count, int max_splits) {
    return max(kChunk, ((count + max_splits - 1) / max_splits + kChunk - 1) / kChunk * kChunk);
}
static int vterm_per_split(int count, int max_splits) { return max(64, (count + max_splits - 1) / max_splits); }
int outer_splits(int count, int max_splits) {
    const int per_split = outer_per_split(count, max_splits);
    return (count + per_split - 1) / per_split;
}
int vterm_splits(int count, int max_splits) {
    const int per_split = vterm_per_split(count, max_splits);
    return (count + per_split - 1) / per_split;
}
int outer_tiles(int N, int M) { return (M + 31) / 32 * ((N + 1 + kOmRows * kOmMaxTy - 1) / (kOmRows * kOmMaxTy)); }

cudaError_t launch_outer_reduce(int count, int N, int nw, int M, const uint64_t* spins, uint64_t enum_base,
                                int enumerate, const OuterSet& set, const float2* A, int lda, double2* partial,
                                int max_splits, cudaStream_t st, SplitSum* job) {
    if (count <= 0) return cudaSuccess;
    const int per_split = outer_per_split(count, max_splits), splits = outer_splits(count, max_splits);
    const int tiles = (N + 1 + kOmRows * kOmMaxTy - 1) / (kOmRows * kOmMaxTy);
    const int ty = (N + 1 + kOmRows * tiles - 1) / (kOmRows * tiles);
    const dim3 grid((M + 31) / 32, tiles, splits), block(32, ty);
    auto run = [&](auto kernel) {
        kernel<<<grid, block, 0, st>>>(count, N, nw, M, spins, enum_base, enumerate, set, A, lda, partial, per_split);
    };
    if (set.n == 1) run(outer_reduce_kernel<1>);
    else if (set.n == 2) run(outer_reduce_kernel<2>);
    else if (set.n == 3) run(outer_reduce_kernel<3>);
    else return cudaErrorInvalidValue;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    SplitSum own{};
    if (!job) job = &own;
    job->elems = static_cast<long>(1 + N) * M;
    job->splits = splits;
    job->nc = set.n;
    job->partial = partial;
    for (int q = 0; q < set.n; q++) job->out[q] = set.out[q];
    job->scale = 1.0;
    return job == &own ? launch_split_sums(job, 1, true, st) : cudaSuccess;
}

cudaError_t launch_vterm_reduce(int count, int N, int nw, int M, int Mpad, const uint64_t* spins, uint64_t enum_base,
                                int enumerate, const double* w, const float2* X, int num_offdiag,
                                const int* site_ptr, const int* site_slots, double2* out, double2* partial,
                                int max_splits, cudaStream_t st, const double2* cw) {
    if (count <= 0 || num_offdiag == 0) return cudaSuccess;
    const int per_split = vterm_per_split(count, max_splits), splits = vterm_splits(count, max_splits);
    const dim3 grid((M + 31) / 32, N, splits);
    vterm_kernel<<<grid, 256, 0, st>>>(count, N, nw, M, Mpad, spins, enum_base, enumerate, w, cw, X, num_offdiag,
                                       site_ptr, site_slots, partial, per_split);
    SplitSum job{};
    job.elems = static_cast<long>(1 + N) * M;
    job.splits = splits;
    job.nc = 1;
    job.partial = partial;
    job.out[0] = out;
    job.scale = -2.0;
    return launch_split_sums(&job, 1, true, st);
}

static size_t grad_vectors_smem(int cap) {
    return sizeof(float4) * kGvWarps * kGvStrings * cap + sizeof(float2) * kGvStrings * kGvWarps * 32 +
           sizeof(pair_t) * kGvWarps * 32 * cap;
}

// the blocks of a column of 32 hidden units walk its units of work, as many in all as the SMs hold at
// once: three each, or two where a group of more than 9700 samples (all states of 14 spins and more)
// takes more than a third of their shared memory; three there were a second, half empty wave (the
// gradient over all states of 16 spins, M = 128, 2.11 ms, now 2.01; 40960 samples at N = 30, M = 75
// 1.57 / 1.50)
struct GradVectorsShape {
    int per_group, units, rows, cap;   // units of a full group, of all groups; blocks a column of units
};
static GradVectorsShape grad_vectors_grid(int count, int group, int Mpad, int max_splits, int sms) {
    int per_split, splits, chunks, cap;
    grad_vectors_shape(std::min(count, group), max_splits, &per_split, &splits, &chunks, &cap);
    const int per_group = splits * chunks, units = (count + group - 1) / group * per_group;
    const int fit = std::min(3, static_cast<int>((size_t(228) << 10) / (grad_vectors_smem(cap) + 1024)));
    return {per_group, units, std::min(units, std::max(1, fit * sms / (Mpad / 32))), cap};
}

size_t grad_vectors_bytes(int count, int group, int N, int M, int Mpad, int max_splits, int sms) {
    return sizeof(double2) * static_cast<size_t>(grad_vectors_grid(count, group, Mpad, max_splits, sms).rows) * (1 + N) * M;
}

cudaError_t launch_grad_vectors(const GradVectors& g, const OpDev& op, double2* partial, int sms, cudaStream_t st,
                                SplitSum* job) {
    if (g.count <= 0) return cudaSuccess;
    const GradVectorsShape S = grad_vectors_grid(g.count, g.group, g.Mpad, g.max_splits, sms);
    const size_t sm = grad_vectors_smem(S.cap);
    const auto kernel = g.Mpad == 32 ? grad_vectors_kernel<true> : grad_vectors_kernel<false>;
    if (sm > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(sm));
        if (e != cudaSuccess) return e;
    }
    const dim3 grid(g.Mpad / 32, S.rows);
    kernel<<<grid, 32 * kGvWarps, sm, st>>>(g, op, S.per_group, S.units, S.cap, partial);
    job->pre = partial;
    job->pre_splits = S.rows;
    return cudaGetLastError();
}

cudaError_t launch_weighted_sums(int count, const double* w, const SeriesSet& set, double2* block_scratch,
                                 double2* sums, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const int blocks = min(kSumBlocks, max(1, (count + 255) / 256));
    wsum_kernel<false><<<blocks, kSumThreads, 0, st>>>(count, w, set, block_scratch, sums);
    return cudaGetLastError();
}

cudaError_t launch_weighted_mean(int count, const double* w, const double2* v, double2* block_scratch, double2* mean,
                                 cudaStream_t st) {
    if (count <= 0) return cudaErrorInvalidValue;
    SeriesSet set{};
    set.n = 1;
    set.v[0] = v;
    wsum_kernel<true><<<min(kSumBlocks, (count + 255) / 256), kSumThreads, 0, st>>>(count, w, set, block_scratch, mean);
    return cudaGetLastError();
}

cudaError_t launch_exact_weights(int count, const double2* lp, double* w, double2* block_scratch, double2* stat,
                                 cudaStream_t st) {
    const int blocks = min(kSumBlocks, max(1, (count + 255) / 256));
    exact_max_kernel<<<blocks, kSumThreads, 0, st>>>(count, lp, block_scratch, stat);
    exact_norm_kernel<<<blocks, kSumThreads, 0, st>>>(count, lp, block_scratch, stat);
    exact_weights_kernel<<<grid_for(count), 256, 0, st>>>(count, lp, stat, w);
    return cudaGetLastError();
}

cudaError_t launch_grad_coefs(int count, const double* w, const double2* v, const double2* shift, double2* c1,
                              double2* c2, double2* c3, int conj3, cudaStream_t st) {
    grad_coefs_kernel<<<grid_for(count), 256, 0, st>>>(count, w, v, shift, c1, c2, c3, conj3);
    return cudaGetLastError();
}

cudaError_t launch_grad_out(const GradOut& g, cudaStream_t st) {
    const long n = max(1L, max(g.count, static_cast<long>(g.first)));
    grad_out_kernel<<<static_cast<int>((n + 255) / 256), 256, 0, st>>>(g);
    return cudaGetLastError();
}

cudaError_t launch_max_re2(int count, const double2* lp, double* block_max, int* blocks_out, cudaStream_t st) {
    const int blocks = min(kSumBlocks, max(1, (count + 255) / 256));
    *blocks_out = blocks;
    max_re2_kernel<<<blocks, 256, 0, st>>>(count, lp, block_max);
    return cudaGetLastError();
}

cudaError_t launch_exp_weights(int count, const double2* lp, double shift, double* w, cudaStream_t st) {
    exp_weights_kernel<<<grid_for(count), 256, 0, st>>>(count, lp, shift, w);
    return cudaGetLastError();
}

cudaError_t launch_coef(int count, const double* w, const double2* v, double scale, double2* c, cudaStream_t st,
                        double2 shift) {
    coef_kernel<<<grid_for(count), 256, 0, st>>>(count, w, v, scale, shift, c);
    return cudaGetLastError();
}

cudaError_t launch_coef_conj(int count, const double* w, const double2* v, double2 shift, double2* c,
                             cudaStream_t st) {
    coef_conj_kernel<<<grid_for(count), 256, 0, st>>>(count, w, v, shift, c);
    return cudaGetLastError();
}

cudaError_t launch_ratio_weights(int count, const double* w, const double2* lp, const double2* lpp, double* rw,
                                 double2* rwc, cudaStream_t st) {
    ratio_weight_kernel<<<grid_for(count), 256, 0, st>>>(count, w, lp, lpp, rw, rwc);
    return cudaGetLastError();
}

cudaError_t launch_corrected_terms(int count, const double2* e, double2* a, cudaStream_t st) {
    corrected_kernel<<<grid_for(count), 256, 0, st>>>(count, e, a);
    return cudaGetLastError();
}

cudaError_t launch_abs2(int count, const double2* v, double2* out, cudaStream_t st) {
    abs2_kernel<<<grid_for(count), 256, 0, st>>>(count, v, out);
    return cudaGetLastError();
}

}  // namespace rbmg
