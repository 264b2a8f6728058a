// Complex-RBM kernels: Metropolis sampler and per-sample estimator pass.
//
// Layout: one warp per configuration, and per walker one warp or, where walkers fill the
// chip, a group of 16 or 8 lanes (rbm_mc_group_kernel).  Lane l of a warp owns hidden units
// j = l + 32 k, k < K (lane g of a group those of lanes g, g + G, ...), and the sampler keeps
// their angles theta_j and Re f(theta_j) in registers for the whole chain; W rows are read
// coalesced from global memory through L1/L2.  This file is included by the rbm_k*.cu
// translation units, each instantiating one K.
#pragma once
#include <type_traits>

#include "device_math.cuh"
#include "kernels.h"

namespace rbmg {

// angles from scratch: theta_j = b_j, then theta_j +/-= W_ij for i = 0..N-1 in order
// (include/quantum_state/Psi.hpp:43-53)
template <int K, int NW>
__device__ __forceinline__ void rbm_refresh(const RbmDev& P, const Spins<NW>& s, float (&tr)[K], float (&ti)[K],
                                            int lane) {
#pragma unroll
    for (int k = 0; k < K; k++) {
        const float2 b = __ldg(P.b + lane + 32 * k);
        tr[k] = b.x;
        ti[k] = b.y;
    }
    const float2* row = P.W + lane;
    for (int i = 0; i < P.N; i++, row += P.Mpad) {
        const float sg = s.up(i) ? 1.0f : -1.0f;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float2 w = __ldg(row + 32 * k);
            tr[k] = __fmaf_rn(sg, w.x, tr[k]);   // sg = +-1: the product is exact
            ti[k] = __fmaf_rn(sg, w.y, ti[k]);
        }
    }
}

template <int NW, class Rng>
__device__ __forceinline__ void draw_spins(Rng& rng, int N, Spins<NW>& s) {
#pragma unroll
    for (int k = 0; k < NW; k++) {
        const uint64_t lo = rng.next();
        const uint64_t hi = rng.next();
        s.w[k] = lo | (hi << 32);
    }
    if (N / 64 < NW) s.w[N / 64] &= (1ull << (N % 64)) - 1ull;
}

// include/random.h:60-79 with 64-bit masks (single word, N <= 64)
template <class Rng>
__device__ __forceinline__ uint64_t draw_n_over_k(Rng& rng, unsigned n, unsigned k) {
    const uint64_t mask = n >= 64 ? ~0ull : ((1ull << n) - 1ull);
    uint64_t w = rng.next();
    w |= static_cast<uint64_t>(rng.next()) << 32;
    uint64_t result = w & mask;
    int diff = static_cast<int>(k) - __popcll(result);
    while (diff != 0) {
        uint64_t w2 = rng.next();
        w2 |= static_cast<uint64_t>(rng.next()) << 32;
        unsigned pos = static_cast<unsigned>(w2 % n);
        for (unsigned guard = 0; ((result >> pos) & 1u) == static_cast<uint64_t>(diff > 0) && guard < 64; guard++)
            pos = (pos + 1) % n;
        result ^= 1ull << pos;
        diff += diff > 0 ? -1 : 1;
    }
    return result;
}

// ---------------------------------------------------------------------------
// A walker's state on packed pairs (device_math.cuh: pair_t, FP32x2):
// pair kk of a lane holds hidden units k = 2 kk and 2 kk + 1; every half is computed with
// the scalar form's operations in its order, so angles, Re f and the decision are the
// scalar ones bit for bit.  KP = ceil(K / 2); for odd K the last pair's second unit is a
// zero row (W and b padded) that enters no sum.
// ---------------------------------------------------------------------------
template <int KP, int NW>
__device__ __forceinline__ void rbm_refresh2(const RbmDev& P, const Spins<NW>& s, pair_t (&tr)[KP],
                                             pair_t (&ti)[KP], int lane) {
#pragma unroll
    for (int kk = 0; kk < KP; kk++) {
        const float4 b = __ldg(P.bq + kk * 32 + lane);
        tr[kk] = pk2(b.x, b.y);
        ti[kk] = pk2(b.z, b.w);
    }
    const float4* row = P.Wq + lane;
    for (int i = 0; i < P.N; i++, row += KP * 32) {
        const pair_t sg = splat2(s.up(i) ? 1.0f : -1.0f);
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
            const float4 w = __ldg(row + 32 * kk);
            tr[kk] = fma2(sg, pk2(w.x, w.y), tr[kk]);   // sg = +-1: the products are exact
            ti[kk] = fma2(sg, pk2(w.z, w.w), ti[kk]);
        }
    }
}

// One update of the fast sweep (MonteCarloLoop.hpp:162-171): the proposal flips the spins
// of a mask that is the AND of `tries` random configurations (each spin flips with
// probability 2^-tries; the mask is warp-uniform).  Unlike the reference, whose Psi keeps
// its angles unchanged for these moves, the proposal's angles follow every flipped site in
// increasing order (theta += 2 s'_i W_i), and the move is accepted on the change of
// Re log psi like a single flip.
template <int K, int KP, int NW, class Rng>
__device__ __forceinline__ bool rbm_fast_step2(const RbmDev& P, Spins<NW>& s, pair_t (&tr)[KP], pair_t (&ti)[KP],
                                               pair_t (&re)[KP], Rng& rng, int lane, int tries) {
    Spins<NW> mask;
    draw_spins(rng, P.N, mask);
    for (int t = 1; t < tries; t++) {
        Spins<NW> m2;
        draw_spins(rng, P.N, m2);
#pragma unroll
        for (int k = 0; k < NW; k++) mask.w[k] &= m2.w[k];
    }
    Spins<NW> s2 = s;
    pair_t nr[KP], ni[KP];
#pragma unroll
    for (int kk = 0; kk < KP; kk++) {
        nr[kk] = tr[kk];
        ni[kk] = ti[kk];
    }
#pragma unroll
    for (int k = 0; k < NW; k++) {
        uint64_t m = mask.w[k];
        while (m) {
            const int site = 64 * k + (__ffsll(static_cast<long long>(m)) - 1);
            m &= m - 1;
            s2.flip(site);
            const pair_t two_s = splat2(s2.up(site) ? 2.0f : -2.0f);
            const float4* row = P.Wq + static_cast<long>(site) * KP * 32 + lane;
#pragma unroll
            for (int kk = 0; kk < KP; kk++) {
                const float4 w = __ldg(row + 32 * kk);
                nr[kk] = fma2(two_s, pk2(w.x, w.y), nr[kk]);
                ni[kk] = fma2(two_s, pk2(w.z, w.w), ni[kk]);
            }
        }
    }
    pair_t nre[KP];
    float part = 0.0f;
#pragma unroll
    for (int kk = 0; kk < KP; kk++) {
        nre[kk] = lc_re2(nr[kk], ni[kk]);
        float d0, d1;
        up2(sub2(nre[kk], re[kk]), d0, d1);
        part = __fadd_rn(part, d0);
        if (2 * kk + 1 < K) part = __fadd_rn(part, d1);
    }
    const float delta = warp_sum_xor(part);
    bool accept = delta > 0.0f;
    if (!accept) accept = rng.uniform() <= expf_det(__fmul_rn(2.0f, delta));
    if (accept) {
        s = s2;
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
            tr[kk] = nr[kk];
            ti[kk] = ni[kk];
            re[kk] = nre[kk];
        }
    }
    return accept;
}

// sign * (-i)^ypow * coef of string n for the current (original) spins, in FP32: the
// local-energy sums run in FP32 with compensated (Kahan) accumulation, since GB300's
// FP64 rate is 1/64 of its FP32 rate and every lane of the warp executes the sum
template <int NW>
__device__ __forceinline__ float2 string_factor(const OpDev& op, int n, const Spins<NW>& s) {
    int parity = 0;
#pragma unroll
    for (int k = 0; k < NW; k++) parity += __popcll(op.zmask[n * kMaxWords + k] & ~s.w[k]);
    const float2 c = op.coef32[n];
    const int yp = op.ypow[n] & 3;
    float2 r;
    if (yp == 0) r = c;
    else if (yp == 1) r = make_float2(c.y, -c.x);
    else if (yp == 2) r = make_float2(-c.x, -c.y);
    else r = make_float2(-c.y, c.x);
    return (parity & 1) ? make_float2(-r.x, -r.y) : r;
}

// compensated FP32 sum (Kahan 1965): the represented value is s - c
struct KahanC {
    float sr = 0.0f, si = 0.0f, cr = 0.0f, ci = 0.0f;
    __device__ __forceinline__ void add(float x, float y) {
        const float yr = __fsub_rn(x, cr), yi = __fsub_rn(y, ci);
        const float tr = __fadd_rn(sr, yr), ti = __fadd_rn(si, yi);
        cr = __fsub_rn(__fsub_rn(tr, sr), yr);
        ci = __fsub_rn(__fsub_rn(ti, si), yi);
        sr = tr;
        si = ti;
    }
    __device__ __forceinline__ double2 value() const {
        return make_double2(static_cast<double>(sr) - static_cast<double>(cr),
                            static_cast<double>(si) - static_cast<double>(ci));
    }
};

// coef * exp(d) for the complex log-ratio d
__device__ __forceinline__ float2 string_term(float2 cf, float2 d) {
    float sn, cs;
    sincosf(d.y, &sn, &cs);
    const float mag = expf(d.x);
    const float xr = mag * cs, xi = mag * sn;
    return make_float2(fmaf(cf.x, xr, -cf.y * xi), fmaf(cf.x, xi, cf.y * xr));
}

// Local energy E_loc(s) = sum_n coef_n phase_n exp(log psi(s'_n) - log psi(s))
// (include/operator/Operator.hpp:90-115).  Diagonal strings contribute coef * phase
// exactly.  With GRAD, also accumulates U_j = sum_n e_n tanh(theta'_nj) (the E_k term,
// Operator.hpp:145-179) and stores X[slot][j] = e_n tanh(theta'_nj) per off-diagonal string.
template <bool GRAD, int K, int NW>
__device__ __forceinline__ double2 rbm_local_energy(const RbmDev& P, const OpDev& op, const Spins<NW>& s,
                                                    const float (&tr)[K], const float (&ti)[K],
                                                    const float2 (&f)[K], const float2 (&T)[K], float2 (&U)[K],
                                                    float2* X, int lane) {
    KahanC acc;
    if (GRAD) {
#pragma unroll
        for (int k = 0; k < K; k++) U[k] = make_float2(0.0f, 0.0f);
    }
    for (int n = 0; n < op.S; n++) {
        const float2 cf = string_factor(op, n, s);
        const int nf = op.nflip[n];
        if (nf == 0) {
            acc.add(cf.x, cf.y);
            if (GRAD) {
                const float ex = cf.x, ey = cf.y;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    U[k].x += ex * T[k].x - ey * T[k].y;
                    U[k].y += ex * T[k].y + ey * T[k].x;
                }
            }
            continue;
        }
        float nr[K], ni[K];
#pragma unroll
        for (int k = 0; k < K; k++) { nr[k] = tr[k]; ni[k] = ti[k]; }
        const int off = op.flip_off[n];
        for (int q = 0; q < nf; q++) {
            const int site = op.flip_sites[off + q];
            const float two_s = s.up(site) ? -2.0f : 2.0f;   // new spin = -old
            const float2* row = P.W + static_cast<long>(site) * P.Mpad + lane;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float2 w = __ldg(row + 32 * k);
                nr[k] = fmaf(two_s, w.x, nr[k]);
                ni[k] = fmaf(two_s, w.y, ni[k]);
            }
        }
        float2 part = make_float2(0.0f, 0.0f);
        float2 th[GRAD ? K : 1];
#pragma unroll
        for (int k = 0; k < K; k++) {
            float2 g;
            if (GRAD) {
                // f and tanh of the flipped angle from one denominator (lc_tanh_approx)
                lc_tanh_approx(nr[k], ni[k], g, th[k]);
            } else {
                g = lc_c(nr[k], ni[k]);
            }
            part.x += g.x - f[k].x;
            part.y += g.y - f[k].y;
        }
        const float2 e = string_term(cf, warp_sum_xor2(part));
        acc.add(e.x, e.y);
        if (GRAD) {
            const float ex = e.x, ey = e.y;
            float2* xrow = X + static_cast<long>(op.offdiag_slot[n]) * P.Mpad + lane;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float2 t2 = th[k];
                const float2 v = make_float2(ex * t2.x - ey * t2.y, ex * t2.y + ey * t2.x);
                U[k].x += v.x;
                U[k].y += v.y;
                xrow[32 * k] = v;
            }
        }
    }
    return acc.value();
}

template <int K>
__device__ __forceinline__ double2 warp_log_psi(const float2 (&f)[K]) {
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < K; k++) { acc.x += f[k].x; acc.y += f[k].y; }
    acc = warp_sum_xor2(acc);
    return make_double2(acc.x, acc.y);
}

// ---------------------------------------------------------------------------
// Metropolis sampler (include/spin_ensembles/MonteCarloLoop.hpp:55-138).  The angles are
// recomputed from the spins at the start of every sweep.  Measurements (local energies, log psi)
// are a separate pass over the recorded configurations, which keeps the registers to the
// walkers' state.
//
// G lanes share a walker, each with PP pairs of hidden units.  G = 32, one walker per warp, where
// walkers are few: a proposal is a chain of dependent steps, and half the units a lane make it
// shorter.  G = 16 (8 at K = 1), two to four walkers per warp, where they fill the chip: what a
// proposal does once per walker -- the random words, the site, the last steps of the lane sum, the
// exponential, the test -- was 65 % of the warp's instructions at K = 4 (273 a proposal, 96 of them
// activations) and serves 32 / G walkers.  Lane g of a group holds what lanes g, g + G, g + 2 G, ...
// of a whole warp hold: their partial sums stay apart until they meet in the order of its
// butterfly (offsets 16, 8, ... down to G within the lane, the rest by shuffles), so angles, sums
// and decisions are the same bit for bit.
// Bound by the FP32 pipe with many walkers (16384: its floor is half of the time) and by one
// proposal's latency with few; the next site is found while a proposal is evaluated, both ways
// the test's number may or may not be used.  rbm_grouped has the times of both; K = 18 has no groups
// (N = 140, 512 / 4096 / 16384 walkers 139, 551, 1996 us a sweep, in groups 252, 652, 2250).
// Blocks of one, two or four warps and keeping the proposed angles measured alike; G = 8 at K = 2
// and 4 was slower up to 4096 walkers.  Five blocks an SM where the registers allow it gained 3 %
// at 16384 walkers and lost 8 % at 512.
//
// total_z: the partner of a flip is the first of a stream of draws whose spin fits; the group's
// lanes test G of them at once (one at a time took two to four rounds of dependent steps: N = 36,
// M = 75, 2048 walkers 44 -> 29 us a sweep with its energies, and 90 -> 32 in a nearly full sector).
// ---------------------------------------------------------------------------
template <int K, int G, int NW, bool SZ>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, K >= 13 ? 3 : 4) rbm_mc_group_kernel(RbmDev P, McLaunch L) {
    constexpr bool WARP = G == 32;   // one walker: a lane's units pair up as in Wq
    constexpr int H = WARP ? 1 : 16 / G, PP = WARP ? (K + 1) / 2 : K * H, PW = 32 / G;   // PW walkers per warp
    const float4* __restrict__ Wp = WARP ? P.Wq : P.Wg;
    const float4* __restrict__ bp = WARP ? P.bq : P.bg;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, g = lane % G;
    const int w0 = (blockIdx.x * kWarpsPerBlock + wib) * PW;
    if (w0 >= L.B) return;
    const int w = min(w0 + lane / G, L.B - 1);
    const bool live = w0 + lane / G < L.B;   // a group past the end repeats the last walker, unwritten
    __shared__ uint4 words_sm[kWarpsPerBlock][32];
    GroupRng<G> rng;
    const uint64_t nmagic = fastmod_magic(static_cast<uint32_t>(P.N));
    Spins<NW> s;
    {
        uint64_t start = L.rng_index[w];
        if (L.init) {
            WalkerRng r;   // the lanes of a group draw the same words, groups go their own way
            r.init(L.seed, L.walker_base + static_cast<uint32_t>(w), start);
#pragma unroll
            for (int k = 0; k < NW; k++) s.w[k] = 0;
            if (SZ) s.w[0] = draw_n_over_k(r, P.N, static_cast<unsigned>((L.sector + P.N) / 2));
            else draw_spins(r, P.N, s);
            start = r.index;
        } else {
#pragma unroll
            for (int k = 0; k < NW; k++) s.w[k] = L.spins[static_cast<long>(w) * NW + k];
        }
        __syncwarp();
        rng.init(L.seed, L.walker_base + static_cast<uint32_t>(w), start, words_sm[wib] + (lane - g), g);
    }
    // the next proposal's site, should the words up to it be used: found while the last one is
    // evaluated, off the chain of dependent steps that one walker's proposals are
    rng.ensure(3, g);
    int next = static_cast<int>(fastmod(rng.peek(), nmagic, static_cast<uint32_t>(P.N)));
    pair_t tr[PP], ti[PP], re[PP];
    unsigned long long acc = 0, props = 0;
    const int total_sweeps = L.n_therm + L.n_samples * L.sweeps_per_sample;
    int sample = 0;
    for (int sw = 0; sw < total_sweeps; sw++) {
        // angles from the spins
#pragma unroll
        for (int p = 0; p < PP; p++) {
            const float4 b = __ldg(bp + p * G + g);
            tr[p] = pk2(b.x, b.y);
            ti[p] = pk2(b.z, b.w);
        }
        const float4* row = Wp + g;
        for (int i = 0; i < P.N; i++, row += PP * G) {
            const pair_t sg = splat2(s.up(i) ? 1.0f : -1.0f);
#pragma unroll
            for (int p = 0; p < PP; p++) {
                const float4 v = __ldg(row + p * G);
                tr[p] = fma2(sg, pk2(v.x, v.y), tr[p]);   // sg = +-1: the products are exact
                ti[p] = fma2(sg, pk2(v.z, v.w), ti[p]);
            }
        }
#pragma unroll
        for (int p = 0; p < PP; p++) re[p] = lc_re2(tr[p], ti[p]);
        for (int prop = 0; prop < P.N; prop++) {
            // words: the site, the partner's candidates, the test's number and the next site
            rng.ensure(SZ ? G + 3 : 3, g);
            const int site = next;
            rng.pos++;
            Spins<NW> s2 = s;
            s2.flip(site);
            const bool first_new = s2.up(site);
            const pair_t t0 = splat2(first_new ? 2.0f : -2.0f);
            const float4* row0 = Wp + static_cast<long>(site) * PP * G + g;
            pair_t t1 = t0;
            const float4* row1 = row0;
            if (SZ) {
                // the partner: drawn until its spin equals the first site's new one; the group's
                // lanes test G draws at once and the first that fits is taken
                int sec = site;
                bool found = false;
                for (int guard = 0; guard < (1 << 20) / G; guard++) {
                    const int c = static_cast<int>(fastmod(rng.words[rng.pos + g], nmagic, static_cast<uint32_t>(P.N)));
                    const bool fits = (c == site ? first_new : s.up(c)) == first_new;
                    const unsigned int fit = (__ballot_sync(0xffffffffu, fits) >> (lane - g)) & (0xffffffffu >> (32 - G));
                    const int taken = __ffs(static_cast<int>(fit)) - 1;
                    const int c2 = __shfl_sync(0xffffffffu, c, (lane - g) + max(taken, 0));
                    if (!found) {
                        if (fit) sec = c2;
                        rng.pos += fit ? taken + 1 : G;
                        found = fit != 0;
                    }
                    if (!__any_sync(0xffffffffu, !found)) break;
                    rng.ensure(G + 2, g);
                }
                s2.flip(sec);
                t1 = splat2(s2.up(sec) ? 2.0f : -2.0f);
                row1 = Wp + static_cast<long>(sec) * PP * G + g;
            }
            const int next0 = static_cast<int>(fastmod(rng.peek(), nmagic, static_cast<uint32_t>(P.N)));
            const int next1 = static_cast<int>(fastmod(rng.words[rng.pos + 1], nmagic, static_cast<uint32_t>(P.N)));
            pair_t part[H], fnew[PP];
            float delta = 0.0f;
#pragma unroll
            for (int h = 0; h < H; h++) part[h] = splat2(0.0f);
#pragma unroll
            for (int p = 0; p < PP; p++) {
                const float4 v = __ldg(row0 + p * G);
                pair_t nr = fma2(t0, pk2(v.x, v.y), tr[p]), ni = fma2(t0, pk2(v.z, v.w), ti[p]);
                if (SZ) {
                    const float4 u = __ldg(row1 + p * G);
                    nr = fma2(t1, pk2(u.x, u.y), nr);
                    ni = fma2(t1, pk2(u.z, u.w), ni);
                }
                fnew[p] = lc_re2(nr, ni);
                const pair_t d = sub2(fnew[p], re[p]);
                if (WARP) {
                    float d0, d1;
                    up2(d, d0, d1);
                    delta = __fadd_rn(delta, d0);
                    if (2 * p + 1 < K) delta = __fadd_rn(delta, d1);
                } else {
                    part[p % H] = add2(part[p % H], d);
                }
            }
            // the butterfly of the one-walker kernel: lanes l and l ^ off, off = 16, 8, 4, 2, 1
            if (!WARP) {
#pragma unroll
                for (int half = H / 2; half >= 1; half >>= 1)
#pragma unroll
                    for (int h = 0; h < half; h++) part[h] = add2(part[h], part[h + half]);
                float d0, d1;
                up2(part[0], d0, d1);
                delta = __fadd_rn(d0, d1);
            }
#pragma unroll
            for (int off = G / 2; off >= 1; off >>= 1)
                delta = __fadd_rn(delta, __shfl_xor_sync(0xffffffffu, delta, off));
            bool accept = delta > 0.0f;
            next = accept ? next0 : next1;
            if (!accept) {
                const float u = __fmul_rn(static_cast<float>((rng.peek() >> 8) + 1u), 5.9604644775390625e-8f);
                rng.pos++;
                accept = u <= expf_det(__fmul_rn(2.0f, delta));
            }
            if (accept) {
                s = s2;
                acc++;
#pragma unroll
                for (int p = 0; p < PP; p++) {
                    const float4 v = __ldg(row0 + p * G);
                    tr[p] = fma2(t0, pk2(v.x, v.y), tr[p]);
                    ti[p] = fma2(t0, pk2(v.z, v.w), ti[p]);
                    if (SZ) {
                        const float4 u = __ldg(row1 + p * G);
                        tr[p] = fma2(t1, pk2(u.x, u.y), tr[p]);
                        ti[p] = fma2(t1, pk2(u.z, u.w), ti[p]);
                    }
                    re[p] = fnew[p];
                }
            }
            __syncwarp();
        }
        props += P.N;
        const int done = sw + 1 - L.n_therm;
        if (done > 0 && done % L.sweeps_per_sample == 0) {
            const long out = static_cast<long>(L.sample_base + sample) * L.B + w;
            if (L.sample_spins && g == 0 && live) {
#pragma unroll
                for (int k = 0; k < NW; k++) L.sample_spins[out * NW + k] = s.w[k];
            }
            sample++;
        }
    }
    if (g == 0 && live) {
#pragma unroll
        for (int k = 0; k < NW; k++) L.spins[static_cast<long>(w) * NW + k] = s.w[k];
        L.rng_index[w] = rng.index();
        L.accepts[w] += acc;
        L.proposals[w] += props;
    }
}

// Fast-sweep sampler (MonteCarloLoop::set_fast_sweep, MonteCarloLoop.hpp:108-113, 139-151,
// 162-171): a thermalisation sweep is N mask updates, a sampling sweep one.  The angles are
// recomputed from the spins every N updates of the thermalisation and at the start of every
// sample's updates (and every N updates within them).
template <int K, int NW>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, K > 13 ? 3 : 4) rbm_mc_fast_kernel(RbmDev P, McLaunch L) {
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (w >= L.B) return;
    WarpRng rng;
    rng.init(L.seed, L.walker_base + static_cast<uint32_t>(w), L.rng_index[w], lane);
    Spins<NW> s;
    if (L.init) {
#pragma unroll
        for (int k = 0; k < NW; k++) s.w[k] = 0;
        draw_spins(rng, P.N, s);
    } else {
#pragma unroll
        for (int k = 0; k < NW; k++) s.w[k] = L.spins[static_cast<long>(w) * NW + k];
    }
    constexpr int KP = (K + 1) / 2;
    pair_t tr[KP], ti[KP], re[KP];
    unsigned long long acc = 0, props = 0;
    auto refresh = [&]() {
        rbm_refresh2(P, s, tr, ti, lane);
#pragma unroll
        for (int kk = 0; kk < KP; kk++) re[kk] = lc_re2(tr[kk], ti[kk]);
    };
    for (int sw = 0; sw < L.n_therm; sw++) {
        refresh();
        for (int p = 0; p < P.N; p++) acc += rbm_fast_step2<K>(P, s, tr, ti, re, rng, lane, L.fast_tries);
        props += P.N;
    }
    for (int sample = 0; sample < L.n_samples; sample++) {
        for (int u = 0; u < L.sweeps_per_sample; u++) {
            if (u % P.N == 0) refresh();
            acc += rbm_fast_step2<K>(P, s, tr, ti, re, rng, lane, L.fast_tries);
        }
        props += L.sweeps_per_sample;
        const long row = static_cast<long>(L.sample_base + sample) * L.B + w;
        if (L.sample_spins && lane == 0) {
#pragma unroll
            for (int k = 0; k < NW; k++) L.sample_spins[row * NW + k] = s.w[k];
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NW; k++) L.spins[static_cast<long>(w) * NW + k] = s.w[k];
        L.rng_index[w] = rng.index;
        L.accepts[w] += acc;
        L.proposals[w] += props;
    }
}

// ---------------------------------------------------------------------------
// Estimator pass over given configurations (one warp each): local energy, log psi,
// the O_k vectors T = tanh(theta), the E_k vectors U and X, and psi' quantities for
// the Hilbert-space distance.
// ---------------------------------------------------------------------------
template <int K, int NW>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) rbm_est_kernel(RbmDev P, OpDev op, int has_op, RbmDev PP,
                                                                       EstLaunch L) {
    const int lane = threadIdx.x & 31;
    const long t = static_cast<long>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
    if (t >= L.count) return;
    Spins<NW> s;
    if (L.flags & EST_ENUMERATE) {
        const uint64_t idx = L.enum_base + static_cast<uint64_t>(t);
        s.w[0] = P.N >= 64 ? idx : (idx & ((1ull << P.N) - 1ull));
#pragma unroll
        for (int k = 1; k < NW; k++) s.w[k] = 0;
    } else {
#pragma unroll
        for (int k = 0; k < NW; k++) s.w[k] = L.spins[t * NW + k];
    }
    if (L.flags & (EST_ELOC | EST_LOGPSI | EST_GRADVEC)) {
        float tr[K], ti[K];
        rbm_refresh(P, s, tr, ti, lane);
        float2 f[K], T[K], U[K];
        const bool grad = (L.flags & EST_GRADVEC) != 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            // with the O_k vectors: f and tanh from one denominator, the same evaluation as
            // the flipped angles' in rbm_local_energy<true> (so that unchanged units cancel)
            if (grad) lc_tanh_approx(tr[k], ti[k], f[k], T[k]);
            else f[k] = lc_c(tr[k], ti[k]);
        }
        if (L.flags & EST_LOGPSI) {
            const double2 lp = warp_log_psi(f);
            if (lane == 0) L.logpsi[t] = lp;
        }
        if (grad) {
#pragma unroll
            for (int k = 0; k < K; k++) L.T[t * P.Mpad + lane + 32 * k] = T[k];
            const double2 e = rbm_local_energy<true>(P, op, s, tr, ti, f, T, U,
                                                     L.X + t * op.num_offdiag * P.Mpad, lane);
            const float shx = static_cast<float>(L.e_shift->x), shy = static_cast<float>(L.e_shift->y);
#pragma unroll
            for (int k = 0; k < K; k++) {
                U[k].x -= shx * T[k].x - shy * T[k].y;
                U[k].y -= shx * T[k].y + shy * T[k].x;
                L.U[t * P.Mpad + lane + 32 * k] = U[k];
            }
            if (lane == 0 && L.eloc) L.eloc[t] = e;
        } else if ((L.flags & EST_ELOC) && has_op) {
            const double2 e = rbm_local_energy<false>(P, op, s, tr, ti, f, T, U, nullptr, lane);
            if (lane == 0) L.eloc[t] = e;
        }
    }
    if (L.flags & EST_PRIME) {
        float pr[K], pi[K];
        rbm_refresh(PP, s, pr, pi, lane);
        float2 fp[K];
#pragma unroll
        for (int k = 0; k < K; k++) fp[k] = lc_c(pr[k], pi[k]);
        const double2 lp = warp_log_psi(fp);
        if (lane == 0) L.logpsi_prime[t] = lp;
        if (L.Tp) {
#pragma unroll
            for (int k = 0; k < K; k++) L.Tp[t * PP.Mpad + lane + 32 * k] = tanh_c(pr[k], pi[k]);
        }
    }
}

// ---------------------------------------------------------------------------
// The gradient's per-sample pass for an operator whose off-diagonal strings flip one site each
// (EstLaunch::en): T = tanh(theta), the angles, every string's term e_n and the local energy.
// One warp per configuration, lanes over the hidden units, as rbm_est_kernel; bound by the FP32
// pipe.  Eight strings at a time, two of them in the halves of each packed operation, and their
// lane sums folded in one butterfly; the exponentials of 32 strings run in the 32 lanes at once
// (they took as long as a unit's activation in every lane before).  Each string's arithmetic
// and the order of the energy's sum are rbm_est_kernel's, so the values are the same.
// N = 64, M = 128, 64 + 128 strings, 4096 samples: 70 us, and 178 us for launch_grad_vectors,
// against 263 us of rbm_est_kernel and 354 us of the sums over its stored terms.
// ---------------------------------------------------------------------------
template <int K, int NW>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) rbm_grad_terms_kernel(RbmDev P, OpDev op, EstLaunch L) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long t = static_cast<long>(blockIdx.x) * kWarpsPerBlock + wib;
    __shared__ float2 terms_sm[kWarpsPerBlock][32];
    if (t >= L.count) return;
    float2* terms = terms_sm[wib];
    Spins<NW> s;
    if (L.flags & EST_ENUMERATE) {
        const uint64_t idx = L.enum_base + static_cast<uint64_t>(t);
        s.w[0] = P.N >= 64 ? idx : (idx & ((1ull << P.N) - 1ull));
#pragma unroll
        for (int k = 1; k < NW; k++) s.w[k] = 0;
    } else {
#pragma unroll
        for (int k = 0; k < NW; k++) s.w[k] = L.spins[t * NW + k];
    }
    float tr[K], ti[K];
    float2 f[K];
    rbm_refresh(P, s, tr, ti, lane);
    const long row = t * P.Mpad + lane;
#pragma unroll
    for (int k = 0; k < K; k++) {
        float2 th;
        lc_tanh_approx(tr[k], ti[k], f[k], th);
        L.T[row + 32 * k] = th;
        L.theta[row + 32 * k] = make_float2(tr[k], ti[k]);
    }
    // lanes 0 and 1: the compensated sums of the terms' real and imaginary parts (KahanC)
    float ks = 0.0f, kc = 0.0f;
    for (int n0 = 0; n0 < op.S; n0 += 32) {
        const int n = n0 + lane;
        const bool live = n < op.S;
        const float2 cf = live ? string_factor(op, n, s) : make_float2(0.0f, 0.0f);
        const bool flips = live && op.nflip[n] != 0;
        const unsigned off = __ballot_sync(0xffffffffu, flips);
        const int rank = __popc(off & ((1u << lane) - 1u));
        float2 d = make_float2(0.0f, 0.0f);
        unsigned m = off;
        for (int b = 0; m; b++) {
            const float2* wrow[8];
            float two_s[8];
            int site = 0;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (m) {
                    site = op.flip_sites[op.flip_off[n0 + __ffs(m) - 1]];
                    m &= m - 1;
                }
                two_s[u] = s.up(site) ? -2.0f : 2.0f;
                wrow[u] = P.W + static_cast<long>(site) * P.Mpad + lane;
            }
            pair_t pr[4], pi[4];
#pragma unroll
            for (int v = 0; v < 4; v++) pr[v] = pi[v] = splat2(0.0f);
#pragma unroll
            for (int k = 0; k < K; k++) {
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const float2 wa = __ldg(wrow[2 * v] + 32 * k), wb = __ldg(wrow[2 * v + 1] + 32 * k);
                    const pair_t ts = pk2(two_s[2 * v], two_s[2 * v + 1]);
                    const Pair2 g = lc_c2_approx(fma2(ts, pk2(wa.x, wb.x), splat2(tr[k])),
                                                 fma2(ts, pk2(wa.y, wb.y), splat2(ti[k])));
                    pr[v] = add2(pr[v], sub2(g.re, splat2(f[k].x)));
                    pi[v] = add2(pi[v], sub2(g.im, splat2(f[k].y)));
                }
            }
            float2 part[8];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                up2(pr[v], part[2 * v].x, part[2 * v + 1].x);
                up2(pi[v], part[2 * v].y, part[2 * v + 1].y);
            }
            const float2 sum = warp_fold8(part, lane);
            const float dx = __shfl_sync(0xffffffffu, sum.x, 4 * (rank & 7));
            const float dy = __shfl_sync(0xffffffffu, sum.y, 4 * (rank & 7));
            if (rank >> 3 == b) d = make_float2(dx, dy);
        }
        float2 e = cf;
        if (flips) {
            e = string_term(cf, d);
            L.en[t * op.num_offdiag + op.offdiag_slot[n]] = e;
        }
        terms[lane] = e;
        __syncwarp();
        const int cnt = min(32, op.S - n0);
        if (lane < 2) {
            const float* v = reinterpret_cast<const float*>(terms) + lane;
            for (int i = 0; i < cnt; i++) {
                const float y = __fsub_rn(v[2 * i], kc), z = __fadd_rn(ks, y);
                kc = __fsub_rn(__fsub_rn(z, ks), y);
                ks = z;
            }
        }
        __syncwarp();
    }
    if (lane < 2) reinterpret_cast<double*>(L.eloc + t)[lane] = static_cast<double>(ks) - static_cast<double>(kc);
}

// ---------------------------------------------------------------------------
// Local energies only (the measurement of a chain step, Operator.hpp:90-115), the lanes
// over the strings: one warp per configuration; its angles
// and f(theta) sit in the warp's shared-memory slice, and every lane evaluates the whole
// log-ratio of its own (off-diagonal string, quarter of the hidden units) item: units
// j = q, q + 4, ... two at a time on FP32x2 pairs (j and j + 4), the flipped angles from the
// transposed W (the lanes of a round read neighbouring spins of the same unit rows), the
// differences f(theta'') - f(theta) summed in pairs (104 units a lane at M = 400; the
// reciprocal of the activation's denominator is the hardware's approximation, within an
// ulp).  Two shuffles join a
// string's quarters; one warp reduction per configuration joins the strings.  No
// per-string reduction sits on the critical path, and each lane's loop over units is
// independent work.
// Bound by shared-memory reads of theta and f and the latency of W's loads beside the FP32 pipe
// (62 to 70 %).  TWO (OpDev::in_pairs): a lane takes two items per round, which halve those reads,
// and four units in flight at large K, where W exceeds the L1.  16384 energies of a transverse field,
// one item a round / two: N = 64, M = 128 238 / 209 us; N = 75, M = 150 366 / 324; N = 100, M = 400 1061 /
// 1002; N = 140, M = 576 2057 / 1867; 512 of them 37 / 25, 76 / 37, 154 / 80, 264 / 127.  Two
// configurations a warp, sharing the loads of W instead, took 225, 336, 1129 and 2330, and half as long
// again at 512.  Strings of two flips (a Heisenberg chain) gain as much: 16384 energies at N = 64, M = 128
// 1.23 times, 500 1.8 times.  One item a round, and the registers for ten blocks an SM instead of
// seven, serves operators of few strings (eight: the second item is no one's), of three flips and more,
// whose sites are looked up unit by unit (5000 energies, N = 64, M = 256, three flips: 356 us, two items 498),
// and of kinds that alternate.  Between 4256 and 5500 configurations, a wave of ten blocks and two of
// seven, strings of two flips lose up to 13 % by it at N = 64 and 256 and gain up to a third elsewhere.
// ---------------------------------------------------------------------------
template <int K, int NW, bool TWO>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, TWO ? (K >= 18 ? 4 : (K >= 13 ? 5 : 7)) : 0) rbm_eloc_t_kernel(RbmDev P, OpDev op, EstLaunch L) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long t = static_cast<long>(blockIdx.x) * kWarpsPerBlock + wib;
    if (t >= L.count) return;
    Spins<NW> s;
    if (L.flags & EST_ENUMERATE) {
        const uint64_t idx = L.enum_base + static_cast<uint64_t>(t);
        s.w[0] = P.N >= 64 ? idx : (idx & ((1ull << P.N) - 1ull));
#pragma unroll
        for (int k = 1; k < NW; k++) s.w[k] = 0;
    } else {
#pragma unroll
        for (int k = 0; k < NW; k++) s.w[k] = L.spins[t * NW + k];
    }
    constexpr int KP = (K + 1) / 2;
    constexpr int MP = 32 * K;
    // the angles and f of every unit in the warp's slice, units j and j + 4 side by side
    // (the pairs the loops below evaluate): pair p = 4 (j / 8) + j % 4 holds
    // tA[p] = (theta.re_j, theta.re_j+4, theta.im_j, theta.im_j+4) and
    // tB[p] = (f.re_j, f.re_j+4, f.im_j, f.im_j+4)
    __shared__ float4 tf_sm[kWarpsPerBlock][MP];
    float4* tA = tf_sm[wib];
    float4* tB = tA + MP / 2;
    {
        // a lane's pair kk holds units lane + 64 kk and lane + 64 kk + 32
        pair_t tr[KP], ti[KP];
        rbm_refresh2(P, s, tr, ti, lane);
        float* fa = reinterpret_cast<float*>(tA);
        float* fb = reinterpret_cast<float*>(tB);
        auto put = [&](int j, float a, float b, float r, float i) {
            const int p = 4 * (j >> 3) + (j & 3), h = (j >> 2) & 1;
            fa[4 * p + h] = a;
            fa[4 * p + 2 + h] = b;
            fb[4 * p + h] = r;
            fb[4 * p + 2 + h] = i;
        };
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
            // f(theta) with the same approximate reciprocal as f(theta'') below
            const Pair2 v = lc_c2_approx(tr[kk], ti[kk]);
            float a0, a1, b0, b1, r0, r1, i0, i1;
            up2(tr[kk], a0, a1);
            up2(ti[kk], b0, b1);
            up2(v.re, r0, r1);
            up2(v.im, i0, i1);
            const int j0 = lane + 64 * kk;
            put(j0, a0, b0, r0, i0);
            if (2 * kk + 1 < K) put(j0 + 32, a1, b1, r1, i1);
        }
    }
    __syncwarp();
    KahanC acc;
    // diagonal strings: the lanes over the strings
    for (int n = lane; n < op.S; n += 32) {
        if (op.nflip[n] == 0) {
            const float2 cf = string_factor(op, n, s);
            acc.add(cf.x, cf.y);
        }
    }
    const int items = 4 * op.num_offdiag;
    const int N = P.N;
    // an item a lane and round
    auto item = [&](int nf, int off, int q, pair_t& sr, pair_t& si) {
        auto unit = [&](float4 f, pair_t xr, pair_t xi) {
            const Pair2 g = lc_c2_approx(xr, xi);
            sr = add2(sr, sub2(g.re, pk2(f.x, f.y)));
            si = add2(si, sub2(g.im, pk2(f.z, f.w)));
        };
        // pairs p = q, q + 4, ...: units (j, j + 4), j = q, q + 8, ...
        if (nf == 1) {
            const int site = op.flip_sites[off];
            const pair_t two_s = splat2(s.up(site) ? -2.0f : 2.0f);
            const float4* wcol = P.Wt4 + site;
#pragma unroll 2
            for (int p = q; p < MP / 2; p += 4) {
                const float4 w = __ldg(wcol + static_cast<long>(p) * N);
                const float4 a = tA[p], f = tB[p];
                unit(f, fma2(two_s, pk2(w.x, w.y), pk2(a.x, a.y)), fma2(two_s, pk2(w.z, w.w), pk2(a.z, a.w)));
            }
        } else {
            for (int p = q; p < MP / 2; p += 4) {
                const float4 a = tA[p], f = tB[p];
                pair_t xr = pk2(a.x, a.y), xi = pk2(a.z, a.w);
                for (int u = 0; u < nf; u++) {
                    const int site = op.flip_sites[off + u];
                    const pair_t two_s = splat2(s.up(site) ? -2.0f : 2.0f);
                    const float4 w = __ldg(P.Wt4 + static_cast<long>(p) * N + site);
                    xr = fma2(two_s, pk2(w.x, w.y), xr);
                    xi = fma2(two_s, pk2(w.z, w.w), xi);
                }
                unit(f, xr, xi);
            }
        }
    };
    for (int it0 = 0; !TWO && it0 < items; it0 += 32) {
        const int it = it0 + lane, q = it & 3;
        const bool live = it < items;
        const int n = live ? op.offdiag[it >> 2] : 0;
        pair_t sr = splat2(0.0f), si = sr;
        if (live) item(op.nflip[n], op.flip_off[n], q, sr, si);
        float r0, r1, i0, i1;
        up2(sr, r0, r1);
        up2(si, i0, i1);
        float dx = r0 + r1, dy = i0 + i1;
        // the four quarters of a string are lanes 4m .. 4m + 3
        dx += __shfl_xor_sync(0xffffffffu, dx, 1);
        dy += __shfl_xor_sync(0xffffffffu, dy, 1);
        dx += __shfl_xor_sync(0xffffffffu, dx, 2);
        dy += __shfl_xor_sync(0xffffffffu, dy, 2);
        if (live && q == 0) {
            const float2 e = string_term(string_factor(op, n, s), make_float2(dx, dy));
            acc.add(e.x, e.y);
        }
    }
    // rounds of 64 items, a lane's two 32 apart: they share the loads of theta and f
    for (int it0 = 0; TWO && it0 < items; it0 += 64) {
        const int q = lane & 3;
        const bool two = it0 + 32 < items;   // for the whole warp
        bool live[2];
        int n[2], nf[2], off[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int it = it0 + 32 * h + lane;
            live[h] = it < items;
            n[h] = op.offdiag[min(it >> 2, op.num_offdiag - 1)];   // of no item: a string of this round's kind
            nf[h] = op.nflip[n[h]];
            off[h] = op.flip_off[n[h]];
        }
        // sums of the real and imaginary differences on pairs (units j, j + 4)
        pair_t sr[2], si[2];
#pragma unroll
        for (int h = 0; h < 2; h++) sr[h] = si[h] = splat2(0.0f);
        auto unit = [&](int h, float4 f, pair_t xr, pair_t xi) {
            const Pair2 g = lc_c2_approx(xr, xi);
            sr[h] = add2(sr[h], sub2(g.re, pk2(f.x, f.y)));
            si[h] = add2(si[h], sub2(g.im, pk2(f.z, f.w)));
        };
        // pairs p = q, q + 4, ...: units (j, j + 4), j = q, q + 8, ...
        // both items, strings of F flips each
        auto both = [&](auto flips) {
            constexpr int F = decltype(flips)::value;
            const float4* w[2][F];
            pair_t ts[2][F];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int u = 0; u < F; u++) {
                    const int site = op.flip_sites[off[h] + u];
                    ts[h][u] = splat2(s.up(site) ? -2.0f : 2.0f);
                    w[h][u] = P.Wt4 + site;
                }
#pragma unroll (K >= 13 && F == 1 ? 4 : 2)
            for (int p = q; p < MP / 2; p += 4) {
                float4 wv[2][F];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int u = 0; u < F; u++) wv[h][u] = __ldg(w[h][u] + static_cast<long>(p) * N);
                const float4 a = tA[p], f = tB[p];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    pair_t xr = pk2(a.x, a.y), xi = pk2(a.z, a.w);
#pragma unroll
                    for (int u = 0; u < F; u++) {
                        xr = fma2(ts[h][u], pk2(wv[h][u].x, wv[h][u].y), xr);
                        xi = fma2(ts[h][u], pk2(wv[h][u].z, wv[h][u].w), xi);
                    }
                    unit(h, f, xr, xi);
                }
            }
        };
        if (two && __all_sync(0xffffffffu, nf[0] == 1 && nf[1] == 1)) {
            both(std::integral_constant<int, 1>());
        } else if (two && __all_sync(0xffffffffu, nf[0] == 2 && nf[1] == 2)) {
            both(std::integral_constant<int, 2>());
        } else {
            // an item at a time, live ones only
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (live[h]) item(nf[h], off[h], q, sr[h], si[h]);
        }
        // the four quarters of a string are lanes 4m .. 4m + 3, of which lane 4m + h forms the
        // term of item h
        float2 d = make_float2(0.0f, 0.0f);
        int mine = n[0];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (h && !two) break;
            float r0, r1, i0, i1;
            up2(sr[h], r0, r1);
            up2(si[h], i0, i1);
            float dx = r0 + r1, dy = i0 + i1;
            dx += __shfl_xor_sync(0xffffffffu, dx, 1);
            dy += __shfl_xor_sync(0xffffffffu, dy, 1);
            dx += __shfl_xor_sync(0xffffffffu, dx, 2);
            dy += __shfl_xor_sync(0xffffffffu, dy, 2);
            if (h == 0 || q == 1) {
                d = make_float2(dx, dy);
                mine = n[h];
            }
        }
        float2 e = make_float2(0.0f, 0.0f);
        if (q < 2) e = string_term(string_factor(op, mine, s), d);
        const float ex = __shfl_down_sync(0xffffffffu, e.x, 1), ey = __shfl_down_sync(0xffffffffu, e.y, 1);
        if (q == 0) {
            if (live[0]) acc.add(e.x, e.y);
            if (live[1]) acc.add(ex, ey);
        }
    }
    double2 v = acc.value();
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if (lane == 0) L.eloc[t] = v;
}

// ---------------------------------------------------------------------------
// launchers for this K (instantiated by rbm_k<K>.cu)
// ---------------------------------------------------------------------------
// One walker per warp or a group of lanes each (rbm_mc_group_kernel).  A sweep takes as long as the
// blocks that the fullest SM has, with whole warps ceil(walkers / 4 SMs).  Up to one (K = 3, whose whole
// warps leave a quarter of their pairs empty), two (K = 1) or three of them the shorter chain of a whole
// warp's proposal wins.  From there on half as many blocks of the groups, each slower, do the same
// work: below K = 8 they are faster at once, above, where one costs 1.9 to 2 of the others, only where
// they are exactly half as many, or so many that the odd one is lost.  K = 10 and 18 have no groups.
// Microseconds a sweep at N = 96, 152 SMs, whole warps / groups of lanes, walkers 1216, 1536, 2048, 3072,
// 4096, 6144, 16384: K = 1: 31/33 38/33 47/33 70/43 78/43 119/59 275/124; K = 2: 32/31 40/40 49/40 74/53
// 83/67 126/102 292/222; K = 3: 38/36 50/49 62/50 92/66 106/85 163/127 385/281; K = 4: 40/43 51/60
// 64/60 96/81 110/103 169/154 400/339; K = 5: 47/48 63/70 80/70 117/95 134/121 209/180 494/399; K = 6:
// 50/60 65/80 82/80 122/111 140/142 216/210 512/468; K = 8: 59/74 78/100 100/100 147/140 169/180 262/264
// 620/594; K = 10: 71/111 93/138 119/138 173/182 200/232 308/336 732/754; K = 13: 91/128 122/162 165/162
// 231/222 270/310 414/430 985/967.
constexpr bool rbm_grouped(int K, int walkers, int sms) {
    if (rbm_group(K) == 32) return false;
    const int blocks = (walkers + 4 * sms - 1) / (4 * sms);
    if (blocks <= (K == 3 ? 1 : (K == 1 ? 2 : 3))) return false;
    return K < 8 || blocks % 2 == 0 || blocks > 14;
}

template <int K>
cudaError_t rbm_mc_launch_k(const RbmDev& P, const OpDev* op, const McLaunch& L, cudaStream_t st) {
    const int nw = (P.N + 63) / 64;
    const dim3 grid((L.B + kWarpsPerBlock - 1) / kWarpsPerBlock), block(32 * kWarpsPerBlock);
    (void)op;
    if (L.fast_tries > 0) {
        if (L.total_z) return cudaErrorInvalidValue;
        switch (nw) {
            case 1: rbm_mc_fast_kernel<K, 1><<<grid, block, 0, st>>>(P, L); break;
            case 2: rbm_mc_fast_kernel<K, 2><<<grid, block, 0, st>>>(P, L); break;
            case 3: rbm_mc_fast_kernel<K, 3><<<grid, block, 0, st>>>(P, L); break;
            case 4: rbm_mc_fast_kernel<K, 4><<<grid, block, 0, st>>>(P, L); break;
            default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
    auto sampler = [&](auto group) {
        constexpr int G = decltype(group)::value, per_block = kWarpsPerBlock * 32 / G;
        const dim3 blocks((L.B + per_block - 1) / per_block);
        if (L.total_z && nw != 1) return cudaErrorInvalidValue;
        if (L.total_z) rbm_mc_group_kernel<K, G, 1, true><<<blocks, block, 0, st>>>(P, L);
        else if (nw == 1) rbm_mc_group_kernel<K, G, 1, false><<<blocks, block, 0, st>>>(P, L);
        else if (nw == 2) rbm_mc_group_kernel<K, G, 2, false><<<blocks, block, 0, st>>>(P, L);
        else if (nw == 3) rbm_mc_group_kernel<K, G, 3, false><<<blocks, block, 0, st>>>(P, L);
        else if (nw == 4) rbm_mc_group_kernel<K, G, 4, false><<<blocks, block, 0, st>>>(P, L);
        else return cudaErrorInvalidValue;
        return cudaGetLastError();
    };
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (rbm_grouped(K, L.B, sms)) return sampler(std::integral_constant<int, rbm_group(K)>());
    return sampler(std::integral_constant<int, 32>());
}

template <int K>
cudaError_t rbm_est_launch_k(const RbmDev& P, const OpDev* op, const RbmDev* PP, const EstLaunch& L,
                             cudaStream_t st) {
    const int nw = (P.N + 63) / 64;
    const dim3 grid((L.count + kWarpsPerBlock - 1) / kWarpsPerBlock), block(32 * kWarpsPerBlock);
    OpDev o = op ? *op : OpDev{};
    const int has = op != nullptr;
    RbmDev pp = PP ? *PP : P;
    if (has && (L.flags & ~(EST_ELOC | EST_ENUMERATE)) == 0) {
        auto energies = [&](auto two) {
            constexpr bool TWO = decltype(two)::value;
            switch (nw) {
                case 1: rbm_eloc_t_kernel<K, 1, TWO><<<grid, block, 0, st>>>(P, o, L); break;
                case 2: rbm_eloc_t_kernel<K, 2, TWO><<<grid, block, 0, st>>>(P, o, L); break;
                case 3: rbm_eloc_t_kernel<K, 3, TWO><<<grid, block, 0, st>>>(P, o, L); break;
                case 4: rbm_eloc_t_kernel<K, 4, TWO><<<grid, block, 0, st>>>(P, o, L); break;
                default: return cudaErrorInvalidValue;
            }
            return cudaGetLastError();
        };
        return o.in_pairs ? energies(std::true_type()) : energies(std::false_type());
    }
    if (L.en) {
        switch (nw) {
            case 1: rbm_grad_terms_kernel<K, 1><<<grid, block, 0, st>>>(P, o, L); break;
            case 2: rbm_grad_terms_kernel<K, 2><<<grid, block, 0, st>>>(P, o, L); break;
            case 3: rbm_grad_terms_kernel<K, 3><<<grid, block, 0, st>>>(P, o, L); break;
            case 4: rbm_grad_terms_kernel<K, 4><<<grid, block, 0, st>>>(P, o, L); break;
            default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
    switch (nw) {
        case 1: rbm_est_kernel<K, 1><<<grid, block, 0, st>>>(P, o, has, pp, L); break;
        case 2: rbm_est_kernel<K, 2><<<grid, block, 0, st>>>(P, o, has, pp, L); break;
        case 3: rbm_est_kernel<K, 3><<<grid, block, 0, st>>>(P, o, has, pp, L); break;
        case 4: rbm_est_kernel<K, 4><<<grid, block, 0, st>>>(P, o, has, pp, L); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace rbmg
