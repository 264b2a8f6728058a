// Batched serving of many independent complex RBMs of uneven N and M (extension: the
// reference runs one network per call, include/spin_ensembles/MonteCarloLoop.hpp:294-339).
//
// One persistent launch serves the whole batch.  Its warps take tasks from a global
// queue (one atomic counter): first the walker tasks of every instance, longest first
// (sweeps of single-flip Metropolis, then at the final configuration the local energy,
// tanh(theta), the angles, U_j = sum_n e_n tanh(theta''_nj) over every string and the
// terms e_n of the off-diagonal strings), then the reduction tasks, each a tile of rows by
// a chunk of walkers of one instance's sums, which start once that instance's walkers are
// all done (a per-instance counter; the wait is bounded by a wall-clock limit after which
// the kernel raises an error flag and returns).  Each tile writes its chunk's partial sums;
// a second kernel of the graph adds the chunks in a fixed order and forms the gradient, so
// every replay gives the same bits.  The walker tasks are compiled for each hidden-unit
// count per lane (rbm_lanes_k: M <= 576) as separate functions of the one kernel.  The
// launch (counter resets + both kernels) is captured once in a CUDA graph and replayed; the
// warps per block, the reduction tile height and a register cap come from an autotuner that
// times the candidates on the batch itself.
//
// Per instance and replay the result is <E_loc> over its walkers and the reference's O_k
// gradient <E O*> + conj<E_k> - 2 <E> <O*> (source/network_functions/ExpectationValue.cu:
// 243-253), with E_k(s) = sum_n e_n O_k(s'_n) (include/operator/Operator.hpp:145-179): for
// W_ij, s_i (U_j - 2 V_ij) with V_ij = sum of e_n tanh(theta''_nj) over the strings n
// flipping site i, recomputed in the tiles from the stored angles (storing these terms
// per walker and string would move O(N^2 M) bytes per walker through HBM).
//
// All parts are bound by FP32 arithmetic and, at the 8 to 16 warps per SM that the walker
// tasks' registers leave, by latency: of a proposal's dependent steps (the next site is found
// ahead, the random words wait in shared memory) and of the L2 loads beside the arithmetic
// (the measurement and the tiles take two strings, or two rows, per packed operation, and the
// tiles fetch a walker ahead).  64 instances of 16 to 144 spins, a replay: 30.7 ms at first,
// 26.2 with packed measurement and tiles, 24.0 with hidden-unit counts between 2 and 13 and
// signs off the FP32 pipe, 22.2 with the shorter proposals.
//
// The sums run centred on the instance's mean energy E (the same value in every tile):
//   gO = sum conj(O),  gE = sum (E_w - E) conj(O),  gK = sum conj(E_k) - conj(E) conj(O),
//   gradient = (gE + gK) / W + (conj(E) - E) gO / W.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <memory>
#include <vector>

#include "host.h"
#include "rbm_impl.cuh"

namespace rbmg {
namespace {

constexpr int kSK = 18;   // hidden units per lane at most (Mpad <= 576)
constexpr int kSW = 3;    // spin words at most (N <= 192)

struct SInst {
    int N, M, Mpad, K, nw;
    const float2* W;
    const float2* b;
    const float4* Wq;     // W and b with a lane's hidden units k and k + 1 side by side (kernels.h)
    const float4* bq;
    OpDev op;
    int walkers;
    uint64_t seed;
    double2* eloc;        // [walkers]
    float2* T;            // [walkers][Mpad] tanh(theta)
    float2* U;            // [walkers][Mpad] sum over every string of e_n tanh(theta''_n)
    float2* theta;        // [walkers][Mpad] the angles of the final configuration
    float2* en;           // [walkers][num_offdiag] e_n of the off-diagonal strings
    const int* site_ptr;  // [N + 1] off-diagonal slots flipping each site (CSR)
    const int* site_slots;
    uint64_t* spins;      // [walkers][nw]
    uint64_t* rng_index;  // [walkers]
    int chunks;           // walker chunks of kReduceWalkers
    float2* part;         // [chunks][3][N + 1][Mpad] a chunk's gO, gE, gK (row N: the biases)
    double2* grad;        // [2 N + M + N M] the gradient, the reference's layout (alpha, beta: 0)
    double2* emean;       // [1] the mean local energy the sums are centred on
    unsigned int* done;   // walkers finished in this replay
};

struct STask {
    int kind;    // 0 walker, 1 reduction tile
    int inst;
    int index;   // walker within the instance, or first row of the tile
    int w0;      // reduction tile: first walker of its walker chunk
    int general; // reduction tile: 1 if a row's site is not flipped by exactly one string
                 // that flips that site alone
};

constexpr int kReduceWalkers = 256;   // walkers per reduction tile

struct SLaunch {
    const SInst* inst;
    const STask* tasks;
    int ntasks;
    unsigned int* next;
    int therm, sweeps;    // sweeps before this replay's measurement: therm (first replay) + sweeps
    int first;            // 1: draw the walkers' start spins
    int* error;           // 1: a reduction task gave up waiting
    unsigned long long* accepts;   // [1]
    unsigned long long wait_ns;    // wall-clock limit of a reduction task's wait
    unsigned int wait_extra;       // walkers a reduction task waits for beyond the instance's
                                   // (0; a test sets it so that the wait runs out)
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <int K, int NW>
__device__ __forceinline__ void s_refresh(const SInst& I, const Spins<NW>& s, float (&tr)[K], float (&ti)[K],
                                          int lane) {
#pragma unroll
    for (int k = 0; k < K; k++) {
        const float2 b = __ldg(I.b + lane + 32 * k);
        tr[k] = b.x;
        ti[k] = b.y;
    }
    const float2* row = I.W + lane;
    for (int i = 0; i < I.N; i++, row += I.Mpad) {
        const float sg = s.up(i) ? 1.0f : -1.0f;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float2 w = __ldg(row + 32 * k);
            tr[k] = __fmaf_rn(sg, w.x, tr[k]);   // sg = +-1: the product is exact
            ti[k] = __fmaf_rn(sg, w.y, ti[k]);
        }
    }
}

// the sweeps on packed pairs (rbm_mc_group_kernel of a single network with 32 lanes a walker, the
// same arithmetic and draw order)
template <int KP, int NW>
__device__ __forceinline__ void s_refresh2(const SInst& I, const Spins<NW>& s, pair_t (&tr)[KP], pair_t (&ti)[KP],
                                           int lane) {
#pragma unroll
    for (int kk = 0; kk < KP; kk++) {
        const float4 b = __ldg(I.bq + kk * 32 + lane);
        tr[kk] = pk2(b.x, b.y);
        ti[kk] = pk2(b.z, b.w);
    }
    const float4* row = I.Wq + lane;
    for (int i = 0; i < I.N; i++, row += KP * 32) {
        const pair_t sg = splat2(s.up(i) ? 1.0f : -1.0f);
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
            const float4 w = __ldg(row + 32 * kk);
            tr[kk] = fma2(sg, pk2(w.x, w.y), tr[kk]);
            ti[kk] = fma2(sg, pk2(w.z, w.w), ti[kk]);
        }
    }
}

template <int K, int KP, int NW>
__device__ __forceinline__ bool s_mh_step2(const SInst& I, Spins<NW>& s, pair_t (&tr)[KP], pair_t (&ti)[KP],
                                           pair_t (&re)[KP], GroupRng<32>& rng, int& next, int lane,
                                           uint64_t nmagic) {
    // words: the site, the test's number and the next site, found ahead for both ways the test's
    // number may or may not be used
    rng.ensure(3, lane);
    const int site = next;
    rng.pos++;
    const int next0 = static_cast<int>(fastmod(rng.peek(), nmagic, static_cast<uint32_t>(I.N)));
    const int next1 = static_cast<int>(fastmod(rng.words[rng.pos + 1], nmagic, static_cast<uint32_t>(I.N)));
    Spins<NW> s2 = s;
    s2.flip(site);
    const pair_t two_s = splat2(s2.up(site) ? 2.0f : -2.0f);
    const float4* row = I.Wq + static_cast<long>(site) * KP * 32 + lane;
    float4 w[KP];
#pragma unroll
    for (int kk = 0; kk < KP; kk++) w[kk] = __ldg(row + 32 * kk);
    float part = 0.0f;
    pair_t fnew[KP];   // Re f of the proposed angles
#pragma unroll
    for (int kk = 0; kk < KP; kk++) {
        const pair_t nr = fma2(two_s, pk2(w[kk].x, w[kk].y), tr[kk]);
        const pair_t ni = fma2(two_s, pk2(w[kk].z, w[kk].w), ti[kk]);
        fnew[kk] = lc_re2(nr, ni);
        float d0, d1;
        up2(sub2(fnew[kk], re[kk]), d0, d1);
        part = __fadd_rn(part, d0);
        if (2 * kk + 1 < K) part = __fadd_rn(part, d1);
    }
    const float delta = warp_sum_xor(part);
    bool accept = delta > 0.0f;
    next = accept ? next0 : next1;
    if (!accept) {
        const float u = __fmul_rn(static_cast<float>((rng.peek() >> 8) + 1u), 5.9604644775390625e-8f);
        rng.pos++;
        accept = u <= expf_det(__fmul_rn(2.0f, delta));
    }
    if (accept) {
        s = s2;
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
            const float4 ww = __ldg(row + 32 * kk);
            tr[kk] = fma2(two_s, pk2(ww.x, ww.y), tr[kk]);
            ti[kk] = fma2(two_s, pk2(ww.z, ww.w), ti[kk]);
            // lc_re2 of the new angles: kept from the proposal where the registers allow
            re[kk] = K <= 8 ? fnew[kk] : lc_re2(tr[kk], ti[kk]);
        }
    }
    return accept;
}

// each task kind is a separate (not inlined) function, so that the register allocation of
// one does not constrain the others
template <int K>
__device__ __noinline__ void walker_task(const SLaunch& L, const SInst& Ig, int w, int lane) {
    constexpr int NW = kSW;
    const SInst I = Ig;   // the descriptor in registers / local memory, not re-read from global
    // the random words sit in this warp's slice of shared memory, which the measurement uses later
    extern __shared__ float2 s_f[];
    GroupRng<32> rng;
    rng.init(I.seed, static_cast<uint32_t>(w), I.rng_index[w],
             reinterpret_cast<uint4*>(s_f + (threadIdx.x >> 5) * 3 * kSK * 32), lane);
    const uint64_t nmagic = fastmod_magic(static_cast<uint32_t>(I.N));
    Spins<NW> s;
#pragma unroll
    for (int k = 0; k < NW; k++) s.w[k] = 0;
    if (L.first) {
        // the draws of draw_spins for this instance's word count (low then high half)
#pragma unroll
        for (int k = 0; k < NW; k++)
            if (k < I.nw) {
                rng.ensure(2, lane);
                const uint64_t lo = rng.peek(), hi = rng.words[rng.pos + 1];
                rng.pos += 2;
                s.w[k] = lo | (hi << 32);
            }
#pragma unroll
        for (int k = 0; k < NW; k++)
            if (k == I.N / 64 && k < I.nw) s.w[k] &= (1ull << (I.N % 64)) - 1ull;
    } else {
#pragma unroll
        for (int k = 0; k < NW; k++)
            if (k < I.nw) s.w[k] = I.spins[static_cast<long>(w) * I.nw + k];
    }
    unsigned long long acc = 0;
    {
        constexpr int KP = (K + 1) / 2;
        pair_t tp[KP], tq[KP], rp[KP];
        const int total = (L.first ? L.therm : 0) + L.sweeps;
        rng.ensure(3, lane);
        int next = static_cast<int>(fastmod(rng.peek(), nmagic, static_cast<uint32_t>(I.N)));
        for (int sw = 0; sw < total; sw++) {
            s_refresh2(I, s, tp, tq, lane);
#pragma unroll
            for (int kk = 0; kk < KP; kk++) rp[kk] = lc_re2(tp[kk], tq[kk]);
            for (int p = 0; p < I.N; p++) acc += s_mh_step2<K>(I, s, tp, tq, rp, rng, next, lane, nmagic);
        }
    }
    // measurement at the final configuration: the local energy, tanh(theta), and for the
    // E_k term the angles, U_j = sum_n e_n tanh(theta''_nj) and the e_n.  Two consecutive
    // off-diagonal strings at a time, in the halves of the packed operations: their four lane
    // sums fold into one butterfly and their terms' exponentials run in the two halves of the
    // warp (12 shuffles and one exponential for 40 and two).  f and tanh of an angle come from
    // one evaluation with the approximate reciprocal (the local-energy differences, as
    // rbm_eloc_t_kernel takes them).  f(theta), U and, between the two uses, tanh(theta'') are in
    // registers up to K = 8; above, f, U and the real parts of tanh in this warp's shared-memory
    // slices [3][kSK][32].
    constexpr bool REGS = K <= 8;
    float tr[K], ti[K];
    s_refresh(I, s, tr, ti, lane);
    __syncwarp();   // the random words have been read
    float2* myf = s_f + (threadIdx.x >> 5) * 3 * kSK * 32 + lane;
    float2* myt = myf + kSK * 32;
    float2* myu = myt + kSK * 32;
    float2 freg[REGS ? K : 1], ureg[REGS ? K : 1];
    const long row_w = static_cast<long>(w) * I.Mpad + lane;
#pragma unroll
    for (int k = 0; k < K; k++) {
        float2 f, t;
        lc_tanh_approx(tr[k], ti[k], f, t);
        if (REGS) {
            freg[REGS ? k : 0] = f;
            ureg[REGS ? k : 0] = make_float2(0.0f, 0.0f);
        } else {
            myf[32 * k] = f;
            myu[32 * k] = make_float2(0.0f, 0.0f);
        }
        I.T[row_w + 32 * k] = t;
        I.theta[row_w + 32 * k] = make_float2(tr[k], ti[k]);
    }
    float2 dsum = make_float2(0.0f, 0.0f);   // the diagonal strings' summed coefficient
    KahanC e;
    for (int n = 0; n < I.op.S;) {
        if (I.op.nflip[n] == 0) {
            const float2 cf = string_factor(I.op, n, s);
            e.add(cf.x, cf.y);
            dsum.x += cf.x;
            dsum.y += cf.y;
            n++;
            continue;
        }
        // strings n and, if it is off-diagonal, n + 1 (else n twice, used once)
        const bool two = n + 1 < I.op.S && I.op.nflip[n + 1] != 0;
        const int n1 = two ? n + 1 : n;
        pair_t pr = splat2(0.0f), pi = pr;
        pair_t hr[REGS ? K : 1], hi[K];
        auto unit = [&](int k, pair_t x, pair_t y) {
            Pair2 g, h;
            lc_tanh2_approx(x, y, g, h);
            const float2 f0 = REGS ? freg[REGS ? k : 0] : myf[32 * k];
            pr = add2(pr, sub2(g.re, splat2(f0.x)));
            pi = add2(pi, sub2(g.im, splat2(f0.y)));
            if (REGS) hr[REGS ? k : 0] = h.re;
            else up2(h.re, myt[32 * k].x, myt[32 * k].y);
            hi[k] = h.im;
        };
        if (I.op.nflip[n] == 1 && I.op.nflip[n1] == 1) {
            const int s0 = I.op.flip_sites[I.op.flip_off[n]], s1 = I.op.flip_sites[I.op.flip_off[n1]];
            const pair_t ts = pk2(s.up(s0) ? -2.0f : 2.0f, s.up(s1) ? -2.0f : 2.0f);
            const float2* r0 = I.W + static_cast<long>(s0) * I.Mpad + lane;
            const float2* r1 = I.W + static_cast<long>(s1) * I.Mpad + lane;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float2 wa = __ldg(r0 + 32 * k), wb = __ldg(r1 + 32 * k);
                unit(k, fma2(ts, pk2(wa.x, wb.x), splat2(tr[k])), fma2(ts, pk2(wa.y, wb.y), splat2(ti[k])));
            }
        } else {
#pragma unroll
            for (int k = 0; k < K; k++) {
                float x[2], y[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int m = h == 0 ? n : n1;
                    float nr = tr[k], ni = ti[k];
                    for (int q = 0; q < I.op.nflip[m]; q++) {
                        const int site = I.op.flip_sites[I.op.flip_off[m] + q];
                        const float two_s = s.up(site) ? -2.0f : 2.0f;
                        const float2 wv = __ldg(I.W + static_cast<long>(site) * I.Mpad + lane + 32 * k);
                        nr = fmaf(two_s, wv.x, nr);
                        ni = fmaf(two_s, wv.y, ni);
                    }
                    x[h] = nr;
                    y[h] = ni;
                }
                unit(k, pk2(x[0], x[1]), pk2(y[0], y[1]));
            }
        }
        // lanes 8 v .. 8 v + 7 end with the sum of value v of (Re 0, Im 0, Re 1, Im 1), added in
        // warp_sum_xor2's order
        float v[4];
        up2(pr, v[0], v[2]);
        up2(pi, v[1], v[3]);
#pragma unroll
        for (int half = 2, off = 16; half >= 1; half >>= 1, off >>= 1) {
            const bool up = (lane & off) != 0;
#pragma unroll
            for (int q = 0; q < half; q++) {
                const float send = up ? v[q] : v[q + half], keep = up ? v[q + half] : v[q];
                v[q] = keep + __shfl_xor_sync(0xffffffffu, send, off);
            }
        }
#pragma unroll
        for (int off = 4; off >= 1; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
        // the lower half of the warp forms string n's term, the upper string n1's
        const int half0 = lane & 16, mine = half0 ? n1 : n;
        const float dx = __shfl_sync(0xffffffffu, v[0], half0), dy = __shfl_sync(0xffffffffu, v[0], half0 + 8);
        const float2 t = string_term(string_factor(I.op, mine, s), make_float2(dx, dy));
        if ((lane & 15) == 0 && (two || lane == 0))
            I.en[static_cast<long>(w) * I.op.num_offdiag + I.op.offdiag_slot[mine]] = t;
        const float2 t0 = make_float2(__shfl_sync(0xffffffffu, t.x, 0), __shfl_sync(0xffffffffu, t.y, 0));
        const float2 t1 = make_float2(__shfl_sync(0xffffffffu, t.x, 16), __shfl_sync(0xffffffffu, t.y, 16));
        e.add(t0.x, t0.y);
        if (two) e.add(t1.x, t1.y);
        const pair_t tx = pk2(t0.x, t1.x), ty = pk2(t0.y, t1.y);
#pragma unroll
        for (int k = 0; k < K; k++) {
            const pair_t a = REGS ? hr[REGS ? k : 0] : pk2(myt[32 * k].x, myt[32 * k].y), b = hi[k];
            const pair_t xr = fma2(tx, a, neg2(mul2(ty, b)));
            const pair_t xi = fma2(ty, a, mul2(tx, b));
            float x0, x1, y0, y1;
            up2(xr, x0, x1);
            up2(xi, y0, y1);
            float2 u = REGS ? ureg[REGS ? k : 0] : myu[32 * k];
            u.x += x0;
            u.y += y0;
            if (two) {
                u.x += x1;
                u.y += y1;
            }
            if (REGS) ureg[REGS ? k : 0] = u;
            else myu[32 * k] = u;
        }
        n = n1 + 1;
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        const float2 h = I.T[row_w + 32 * k];
        float2 u = REGS ? ureg[REGS ? k : 0] : myu[32 * k];
        u.x += __fmaf_rn(dsum.x, h.x, -__fmul_rn(dsum.y, h.y));
        u.y += __fmaf_rn(dsum.x, h.y, __fmul_rn(dsum.y, h.x));
        I.U[row_w + 32 * k] = u;
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NW; k++)
            if (k < I.nw) I.spins[static_cast<long>(w) * I.nw + k] = s.w[k];
        I.rng_index[w] = rng.index();
        I.eloc[w] = e.value();
        atomicAdd(L.accepts, acc);
    }
    __syncwarp();
    __threadfence();
    if (lane == 0) atomicAdd(I.done, 1u);
}

// rows [r0, r0 + R) of the instance's sums (row N: the biases), every column, over the
// walkers of chunk [w0, w0 + kReduceWalkers): the chunk's partial sums of gO, gE and gK
// (every partial is written by exactly one tile; serve_finish_kernel adds the chunks)
template <int R, bool GENERAL>
__device__ __noinline__ void reduce_task(const SLaunch& L, const SInst& Ig, int r0, int w0, int lane) {
    const SInst I = Ig;   // the descriptor in registers: loop-invariant, not re-read per walker
    // wait for the instance's walkers (bounded by L.wait_ns of wall clock; a wait that gives
    // up raises the error flag, and every other waiter leaves as soon as it sees the flag)
    if (lane == 0) {
        const unsigned long long t0 = global_ns();
        const unsigned int need = static_cast<unsigned int>(I.walkers) + L.wait_extra;
        while (atomicAdd(I.done, 0u) < need) {
            if (*reinterpret_cast<volatile int*>(L.error)) break;
            if (global_ns() - t0 > L.wait_ns) {
                atomicExch(L.error, 1);
                break;
            }
            __nanosleep(1000);
        }
    }
    __syncwarp();
    if (*reinterpret_cast<volatile int*>(L.error)) return;
    __threadfence();
    // the instance's mean local energy, in a fixed order (the same value in every tile)
    double mx = 0.0, my = 0.0;
    for (int w = lane; w < I.walkers; w += 32) {
        const double2 ed = __ldcg(I.eloc + w);
        mx += ed.x;
        my += ed.y;
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        mx += __shfl_xor_sync(0xffffffffu, mx, off);
        my += __shfl_xor_sync(0xffffffffu, my, off);
    }
    mx /= I.walkers;
    my /= I.walkers;
    if (r0 == 0 && w0 == 0 && lane == 0) *I.emean = make_double2(mx, my);
    const float Er = static_cast<float>(mx), Ei = static_cast<float>(my);
    const int chunk = w0 / kReduceWalkers;
    const long plane = static_cast<long>(I.N + 1) * I.Mpad;
    float2* part = I.part + static_cast<long>(chunk) * 3 * plane;
    const int w1 = min(I.walkers, w0 + kReduceWalkers);
    // per row, fetched once: the off-diagonal slots flipping its site; in the common case
    // of one slot whose string flips that one site, the slot and the site
    int sb[R], se[R], fslot[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = r0 + r;
        sb[r] = i < I.N ? I.site_ptr[i] : 0;
        se[r] = i < I.N ? I.site_ptr[i + 1] : 0;
        fslot[r] = -1;
        if (se[r] - sb[r] == 1) {
            const int slot = I.site_slots[sb[r]];
            const int n = I.op.offdiag[slot];
            if (I.op.nflip[n] == 1) fslot[r] = slot;
        }
    }
    // rows r0 + 2 q and r0 + 2 q + 1 in the halves of the packed operations.  A block of 32
    // walkers' e_n (Re, Re', Im, Im') and spins (+-1, +-1') of each row pair, [R / 2][32], are in
    // this warp's shared-memory slice
    extern __shared__ float2 s_f[];
    float4* sen = reinterpret_cast<float4*>(s_f + (threadIdx.x >> 5) * 3 * kSK * 32);
    float2* ssg = reinterpret_cast<float2*>(sen + R / 2 * 32);
    const long estride = I.op.num_offdiag;
    const uint64_t* spins = reinterpret_cast<const uint64_t*>(I.spins);
    for (int kc = 0; kc < I.K; kc++) {
        pair_t aOx[R / 2], aOy[R / 2], aEx[R / 2], aEy[R / 2], aKx[R / 2], aKy[R / 2];
#pragma unroll
        for (int q = 0; q < R / 2; q++) aOx[q] = aOy[q] = aEx[q] = aEy[q] = aKx[q] = aKy[q] = splat2(0.0f);
        const int j = lane + 32 * kc;
        pair_t wx[R / 2], wy[R / 2];   // -2 W[i][j] of each row pair's sites (the single-flip case)
#pragma unroll
        for (int q = 0; q < R / 2; q++) {
            float2 a = make_float2(0.0f, 0.0f), b = a;
            const float2* wp = I.W + static_cast<long>(r0 + 2 * q) * I.Mpad + j;
            if (r0 + 2 * q < I.N) a = __ldg(wp);
            if (r0 + 2 * q + 1 < I.N) b = __ldg(wp + I.Mpad);
            wx[q] = pk2(-2.0f * a.x, -2.0f * b.x);
            wy[q] = pk2(-2.0f * a.y, -2.0f * b.y);
        }
        for (int wb = w0; wb < w1; wb += 32) {
            // a block of 32 walkers: lane b fetches walker wb + b's centred energy, the spins
            // of the tile's rows (bit r: row r0 + r up) and the e_n of the rows' single-flip
            // strings, all at once; the walker loop below takes them by shuffles.  L2 loads
            // (__ldcg): the walkers' results were written by other SMs
            const int nb = min(32, w1 - wb);
            float sdx = 0.0f, sdy = 0.0f;
            __syncwarp();   // the previous block's reads of the slice are done
            if (lane < nb) {
                const int ws = wb + lane;
                const double2 ed = __ldcg(I.eloc + ws);
                sdx = static_cast<float>(ed.x - mx);
                sdy = static_cast<float>(ed.y - my);
                // rows r0 .. r0 + R - 1 (R <= 64) lie in at most two spin words
                const int q0 = min(r0, I.N - 1) >> 6, q1 = min(r0 + R - 1, I.N - 1) >> 6;
                const uint64_t lo = __ldcg(spins + static_cast<long>(ws) * I.nw + q0);
                const uint64_t hi = q1 != q0 ? __ldcg(spins + static_cast<long>(ws) * I.nw + q1) : lo;
#pragma unroll
                for (int q = 0; q < R / 2; q++) {
                    float sg[2] = {1.0f, 1.0f};   // the bias row's factor
                    float2 en[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int i = r0 + 2 * q + h;
                        if (i >= I.N) continue;
                        const uint64_t wd = (i >> 6) == q0 ? lo : hi;
                        sg[h] = (wd >> (i & 63)) & 1ull ? 1.0f : -1.0f;
                        if (fslot[2 * q + h] >= 0) en[h] = __ldcg(I.en + ws * estride + fslot[2 * q + h]);
                    }
                    sen[q * 32 + lane] = make_float4(en[0].x, en[1].x, en[0].y, en[1].y);
                    ssg[q * 32 + lane] = make_float2(sg[0], sg[1]);
                }
            }
            __syncwarp();
            // the next walker's column is fetched while this one's rows are formed
            long o = static_cast<long>(wb) * I.Mpad + j;
            float2 tn = __ldcg(I.T + o), un = __ldcg(I.U + o), thn = __ldcg(I.theta + o);
            for (int bw = 0; bw < nb; bw++) {
                const int w = wb + bw;
                const float2 t = tn, u = un, th = thn;
                if (bw + 1 < nb) {
                    o += I.Mpad;
                    tn = __ldcg(I.T + o);
                    un = __ldcg(I.U + o);
                    thn = __ldcg(I.theta + o);
                }
                const float dx = __shfl_sync(0xffffffffu, sdx, bw);
                const float dy = __shfl_sync(0xffffffffu, sdy, bw);
                // conj(t), (E - <E>) conj(t), and U - <E> t (E_k of the biases, centred)
                const float cx = t.x, cy = -t.y;
                const float ex = __fmaf_rn(dx, cx, -__fmul_rn(dy, cy)), ey = __fmaf_rn(dy, cx, __fmul_rn(dx, cy));
                const float kx = __fsub_rn(u.x, __fmaf_rn(Er, t.x, -__fmul_rn(Ei, t.y)));
                const float ky = __fsub_rn(u.y, __fmaf_rn(Er, t.y, __fmul_rn(Ei, t.x)));
                uint64_t sw[kSW];
#pragma unroll
                for (int q = 0; q < kSW; q++)
                    sw[q] = GENERAL && q < I.nw ? __ldcg(spins + static_cast<long>(w) * I.nw + q) : 0ull;
                auto up = [&](int site) {
                    uint64_t wd = sw[0];
#pragma unroll
                    for (int q = 1; q < kSW; q++)
                        if ((site >> 6) == q) wd = sw[q];
                    return ((wd >> (site & 63)) & 1ull) != 0ull;
                };
#pragma unroll
                for (int q = 0; q < R / 2; q++) {
                    if (r0 + 2 * q > I.N) continue;
                    const float2 sgf = ssg[q * 32 + bw];
                    const pair_t sg = pk2(sgf.x, sgf.y);
                    // V_ij = sum over the strings n flipping site i of e_n tanh(theta''_nj),
                    // the angles theta'' formed as the walker task formed them
                    pair_t vx = splat2(0.0f), vy = vx;
                    if (!GENERAL || fslot[2 * q] >= 0 || fslot[2 * q + 1] >= 0) {
                        const Pair2 h = tanh2_approx(fma2(sg, wx[q], splat2(th.x)), fma2(sg, wy[q], splat2(th.y)));
                        const float4 en = sen[q * 32 + bw];
                        const pair_t enx = pk2(en.x, en.y), eny = pk2(en.z, en.w);
                        vx = fma2(enx, h.re, neg2(mul2(eny, h.im)));
                        vy = fma2(enx, h.im, mul2(eny, h.re));
                    }
                    if (GENERAL) {
                        float v0[2], v1[2];
                        up2(vx, v0[0], v0[1]);
                        up2(vy, v1[0], v1[1]);
#pragma unroll
                        for (int hf = 0; hf < 2; hf++) {
                            const int r = 2 * q + hf;
                            if (fslot[r] >= 0 || r0 + r >= I.N) continue;
                            float vrx = 0.0f, vry = 0.0f;
                            const float2* enw = I.en + w * estride;
                            for (int p = sb[r]; p < se[r]; p++) {
                                const int slot = I.site_slots[p];
                                const int n = I.op.offdiag[slot];
                                const int nf = I.op.nflip[n], fo = I.op.flip_off[n];
                                float nr = th.x, ni = th.y;
                                for (int f = 0; f < nf; f++) {
                                    const int site = I.op.flip_sites[fo + f];
                                    const float ts = up(site) ? -2.0f : 2.0f;
                                    const float2 wv = __ldg(I.W + static_cast<long>(site) * I.Mpad + j);
                                    nr = fmaf(ts, wv.x, nr);
                                    ni = fmaf(ts, wv.y, ni);
                                }
                                float2 g, h;
                                lc_tanh_approx(nr, ni, g, h);
                                const float2 en = __ldcg(enw + slot);
                                vrx += en.x * h.x - en.y * h.y;
                                vry += en.x * h.y + en.y * h.x;
                            }
                            v0[hf] = vrx;
                            v1[hf] = vry;
                        }
                        vx = pk2(v0[0], v0[1]);
                        vy = pk2(v1[0], v1[1]);
                    }
                    aOx[q] = fma2(sg, splat2(cx), aOx[q]);   // sg = +-1: the products are exact
                    aOy[q] = fma2(sg, splat2(cy), aOy[q]);
                    aEx[q] = fma2(sg, splat2(ex), aEx[q]);
                    aEy[q] = fma2(sg, splat2(ey), aEy[q]);
                    // conj(s_i (U - 2 V) - <E> O) = sg conj(U - <E> t - 2 V); aKy holds its negative
                    aKx[q] = fma2(sg, fma2(splat2(-2.0f), vx, splat2(kx)), aKx[q]);
                    aKy[q] = fma2(sg, fma2(splat2(-2.0f), vy, splat2(ky)), aKy[q]);
                }
            }
        }
        auto put = [&](pair_t x, pair_t y, float sy, float2* out, int q) {
            float x0, x1, y0, y1;
            up2(x, x0, x1);
            up2(y, y0, y1);
            const long e = static_cast<long>(r0 + 2 * q) * I.Mpad + j;
            if (r0 + 2 * q <= I.N) out[e] = make_float2(x0, sy * y0);
            if (r0 + 2 * q + 1 <= I.N) out[e + I.Mpad] = make_float2(x1, sy * y1);
        };
#pragma unroll
        for (int q = 0; q < R / 2; q++) {
            put(aOx[q], aOy[q], 1.0f, part, q);
            put(aEx[q], aEy[q], 1.0f, part + plane, q);
            put(aKx[q], aKy[q], -1.0f, part + 2 * plane, q);
        }
    }
}

// the sums over the walker chunks, in chunk order, and from them the gradient in the
// reference's parameter layout (FP64): blockIdx.y is the instance, e a row and column of its
// sums.  Formed here, a result is one copy of 16 bytes per parameter; three sums per padded
// entry and the combination on the host took 8.6 ms for 64 instances of up to 144 spins, 30 ms
// of kernel.
__global__ void serve_finish_kernel(const SInst* inst) {
    const SInst& I = inst[blockIdx.y];
    const long plane = static_cast<long>(I.N + 1) * I.Mpad, n = 3 * plane;
    const double inv = 1.0 / I.walkers;
    const double shift = -2.0 * I.emean->y;   // conj(E) - E = i shift
    for (long e = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; e < plane;
         e += static_cast<long>(gridDim.x) * blockDim.x) {
        const int row = static_cast<int>(e / I.Mpad), j = static_cast<int>(e - static_cast<long>(row) * I.Mpad);
        if (j >= I.M) continue;
        double ox = 0.0, oy = 0.0, ex = 0.0, ey = 0.0, kx = 0.0, ky = 0.0;
        for (int c = 0; c < I.chunks; c++) {
            const float2 o = I.part[c * n + e], v = I.part[c * n + plane + e], k = I.part[c * n + 2 * plane + e];
            ox += o.x;
            oy += o.y;
            ex += v.x;
            ey += v.y;
            kx += k.x;
            ky += k.y;
        }
        // the biases (row N) come before the weights
        const long at = 2L * I.N + j + (row == I.N ? 0L : I.M + static_cast<long>(row) * I.M);
        I.grad[at] = make_double2((ex + kx - shift * oy) * inv, (ey + ky + shift * ox) * inv);
    }
}

// REGS caps the registers per thread (the largest walker task sets the kernel's count, so
// a cap trades its spills against more resident warps for every task); the autotuner picks
template <int R, int REGS>
__global__ void __maxnreg__(REGS) serve_kernel(SLaunch L) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int t = 0;
        if (lane == 0) t = static_cast<int>(atomicAdd(L.next, 1u));
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= L.ntasks) return;
        const STask task = L.tasks[t];
        const SInst& I = L.inst[task.inst];
        if (task.kind == 0) {
            switch (I.K) {   // the hidden-unit counts per lane of rbm_lanes_k
                case 1: walker_task<1>(L, I, task.index, lane); break;
                case 2: walker_task<2>(L, I, task.index, lane); break;
                case 3: walker_task<3>(L, I, task.index, lane); break;
                case 4: walker_task<4>(L, I, task.index, lane); break;
                case 5: walker_task<5>(L, I, task.index, lane); break;
                case 6: walker_task<6>(L, I, task.index, lane); break;
                case 8: walker_task<8>(L, I, task.index, lane); break;
                case 10: walker_task<10>(L, I, task.index, lane); break;
                case 13: walker_task<13>(L, I, task.index, lane); break;
                default: walker_task<18>(L, I, task.index, lane); break;
            }
        } else {
            // rows whose sites are all flipped by one single-flip string each take the
            // specialised tile (task.general: some row is not)
            if (task.general) reduce_task<R, true>(L, I, task.index, task.w0, lane);
            else reduce_task<R, false>(L, I, task.index, task.w0, lane);
        }
    }
}

}  // namespace
}  // namespace rbmg

using namespace rbmg;

struct rbmg_batch {
    int n = 0;
    std::vector<const rbmg_psi*> psis;
    std::vector<const rbmg_operator*> ops;
    std::vector<SInst> host_inst;
    std::vector<std::vector<char>> single_flip;   // [instance][site]: the single-flip tile serves the site
    std::vector<uint32_t> walkers;
    DevBuf d_inst, d_tasks, d_next, d_done, d_accepts;
    DevBuf d_status;            // [n] mean energies, then the error flag: one copy per replay
    std::vector<double2> status;   // the last replay's
    int* d_error() const { return reinterpret_cast<int*>(d_status.as<double2>() + n); }
    int max_elems = 0;          // largest instance's (N + 1) Mpad (the finish kernel's grid)
    std::vector<std::unique_ptr<DevBuf>> bufs;
    int ntasks_walk = 0, ntasks = 0;
    int rows = 16;              // reduction tile height
    int warps_per_block = 4;
    int regs = 255;             // register cap per thread: 255, 128 or 96
    int blocks = 0;
    bool first = true;
    int therm = 0, sweeps = 1;  // graph parameters
    unsigned long long wait_ns = 20000000000ull;
    unsigned int wait_extra = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_rows = 0, graph_wpb = 0, graph_regs = 0, graph_first = -1, graph_therm = -1, graph_sweeps = -1;
    unsigned long long graph_wait_ns = 0;
    unsigned int graph_wait_extra = 0;
    double tuned_ms = 0.0;
    ~rbmg_batch() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

namespace {

int batch_tasks(rbmg_batch* b) {
    // walker tasks, longest first (cost ~ N * Mpad per sweep), then reduction tiles
    std::vector<int> order(b->n);
    for (int i = 0; i < b->n; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int c) {
        return static_cast<long>(b->host_inst[a].N) * b->host_inst[a].Mpad >
               static_cast<long>(b->host_inst[c].N) * b->host_inst[c].Mpad;
    });
    std::vector<STask> tasks;
    for (int i : order)
        for (int w = 0; w < b->host_inst[i].walkers; w++) tasks.push_back(STask{0, i, w, 0, 0});
    b->ntasks_walk = static_cast<int>(tasks.size());
    for (int i : order) {
        const int N = b->host_inst[i].N;
        for (int r0 = 0; r0 <= N; r0 += b->rows) {
            int general = 0;
            for (int r = r0; r < std::min(N, r0 + b->rows); r++) general |= !b->single_flip[i][r];
            for (int w0 = 0; w0 < b->host_inst[i].walkers; w0 += kReduceWalkers)
                tasks.push_back(STask{1, i, r0, w0, general});
        }
    }
    b->ntasks = static_cast<int>(tasks.size());
    RBMG_CK(b->d_tasks.ensure(sizeof(STask) * tasks.size()));
    RBMG_CK(cudaMemcpy(b->d_tasks.p, tasks.data(), sizeof(STask) * tasks.size(), cudaMemcpyHostToDevice));
    return RBMG_OK;
}

size_t serve_smem(int warps_per_block) { return sizeof(float2) * 3 * kSK * 32 * warps_per_block; }

// calls f with the kernel instantiation of (reduction rows, register cap)
template <class F>
void with_serve_kernel(int rows, int regs, F f) {
    if (rows == 8) {
        if (regs == 128) f(serve_kernel<8, 128>);
        else if (regs == 96) f(serve_kernel<8, 96>);
        else f(serve_kernel<8, 255>);
    } else {
        if (regs == 128) f(serve_kernel<16, 128>);
        else if (regs == 96) f(serve_kernel<16, 96>);
        else f(serve_kernel<16, 255>);
    }
}

// the kernel instantiation's dynamic shared-memory limit (above the 48 KB default for 4 and
// 8 warps per block); the attribute belongs to the current device's context
cudaError_t serve_smem_attr(int rows, int regs, size_t sm) {
    cudaError_t e = cudaSuccess;
    with_serve_kernel(rows, regs, [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sm));
    });
    return e;
}

cudaError_t launch_serve(rbmg_batch* b, cudaStream_t st) {
    SLaunch L{};
    L.inst = b->d_inst.as<SInst>();
    L.tasks = b->d_tasks.as<STask>();
    L.ntasks = b->ntasks;
    L.next = b->d_next.as<unsigned int>();
    L.therm = b->therm;
    L.sweeps = b->sweeps;
    L.first = b->first ? 1 : 0;
    L.error = b->d_error();
    L.accepts = b->d_accepts.as<unsigned long long>();
    L.wait_ns = b->wait_ns;
    L.wait_extra = b->wait_extra;
    const int threads = 32 * b->warps_per_block;
    const size_t sm = serve_smem(b->warps_per_block);
    const cudaError_t e = serve_smem_attr(b->rows, b->regs, sm);
    if (e != cudaSuccess) return e;
    with_serve_kernel(b->rows, b->regs, [&](auto kern) { kern<<<b->blocks, threads, sm, st>>>(L); });
    return cudaGetLastError();
}

// (re)captures the replay: counter resets and the persistent launch
int batch_capture(rbmg_batch* b) {
    if (b->exec && b->graph_rows == b->rows && b->graph_wpb == b->warps_per_block && b->graph_regs == b->regs &&
        b->graph_first == static_cast<int>(b->first) && b->graph_therm == b->therm && b->graph_sweeps == b->sweeps &&
        b->graph_wait_ns == b->wait_ns && b->graph_wait_extra == b->wait_extra)
        return RBMG_OK;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    int dev = 0, sms = 0, per_sm = 0;
    RBMG_CK(cudaGetDevice(&dev));
    RBMG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int threads = 32 * b->warps_per_block;
    const size_t sm = serve_smem(b->warps_per_block);
    RBMG_CK(serve_smem_attr(b->rows, b->regs, sm));
    cudaError_t oe = cudaSuccess;
    with_serve_kernel(b->rows, b->regs,
                      [&](auto kern) { oe = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, sm); });
    RBMG_CK(oe);
    b->blocks = std::max(1, sms * std::max(1, per_sm));
    cudaStream_t st = stream();
    RBMG_CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(b->d_next.p, 0, sizeof(unsigned int), st);
    cudaMemsetAsync(b->d_done.p, 0, sizeof(unsigned int) * b->n, st);
    cudaMemsetAsync(b->d_accepts.p, 0, sizeof(unsigned long long), st);
    cudaError_t le = launch_serve(b, st);
    if (le == cudaSuccess) {
        const dim3 grid(std::min(64, (b->max_elems + 255) / 256), b->n);
        serve_finish_kernel<<<grid, 256, 0, st>>>(b->d_inst.as<SInst>());
        le = cudaGetLastError();
    }
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(st, &g);
    RBMG_CK(le);
    RBMG_CK(ce);
    b->graph = g;
    RBMG_CK(cudaGraphInstantiate(&b->exec, b->graph, 0));
    b->graph_rows = b->rows;
    b->graph_wpb = b->warps_per_block;
    b->graph_regs = b->regs;
    b->graph_first = static_cast<int>(b->first);
    b->graph_therm = b->therm;
    b->graph_sweeps = b->sweeps;
    b->graph_wait_ns = b->wait_ns;
    b->graph_wait_extra = b->wait_extra;
    return RBMG_OK;
}

// waits for the replays and takes the mean energies and the error flag
cudaError_t batch_status(rbmg_batch* b, int* err) {
    cudaError_t e = cudaMemcpyAsync(b->status.data(), b->d_status.p, sizeof(double2) * (b->n + 1), cudaMemcpyDeviceToHost,
                                    stream());
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
    std::memcpy(err, &b->status[b->n], sizeof(int));
    return e;
}

int batch_replay(rbmg_batch* b) {
    int r = batch_capture(b);
    if (r != RBMG_OK) return r;
    RBMG_CK(cudaGraphLaunch(b->exec, stream()));
    int err = 0;
    RBMG_CK(batch_status(b, &err));
    if (err) {
        RBMG_CK(cudaMemset(b->d_error(), 0, sizeof(int)));
        return fail(RBMG_ETIMEOUT, "batch: a reduction task timed out waiting for its walkers");
    }
    b->first = false;
    return RBMG_OK;
}

}  // namespace

extern "C" int rbmg_batch_create(int n, const rbmg_psi* const* psis, const rbmg_operator* const* ops,
                                 const uint32_t* walkers, const uint64_t* seeds, rbmg_batch** out) {
    if (n <= 0 || !psis || !ops || !walkers || !seeds || !out) return fail(RBMG_EINVAL, "batch: bad arguments");
    auto b = std::make_unique<rbmg_batch>();
    b->n = n;
    b->status.resize(n + 1);
    RBMG_CK(b->d_status.ensure(sizeof(double2) * (n + 1)));
    RBMG_CK(cudaMemset(b->d_status.p, 0, sizeof(double2) * (n + 1)));
    for (int i = 0; i < n; i++) {
        const rbmg_psi* p = psis[i];
        const rbmg_operator* o = ops[i];
        if (!p || !o || walkers[i] == 0) return fail(RBMG_EINVAL, "batch: null instance or no walkers");
        if (p->kind != 0) return fail(RBMG_EUNSUPPORTED, "batch: complex RBM (Psi) instances only");
        if (p->Mpad / 32 > kSK) return fail(RBMG_EUNSUPPORTED, "batch: M <= 576");
        if (p->Mpad != 32 * rbm_lanes_k(p->M)) return fail(RBMG_EINVAL, "batch: unexpected hidden-unit padding");
        if (p->N > 64 * kSW) return fail(RBMG_EUNSUPPORTED, "batch: N <= 192");
        if (o->max_site >= p->N) return fail(RBMG_EINVAL, "batch: operator acts on a site >= N");
        for (int q = 0; q < i; q++)
            if (ops[q] == o && psis[q]->N != p->N)
                return fail(RBMG_EINVAL, "batch: an operator shared by instances of different N");
        {
            const int r = op_site_lists(const_cast<rbmg_operator*>(o), p->N);
            if (r != RBMG_OK) return r;
        }
        const int nw = nwords_of(p->N);
        SInst I{};
        I.N = p->N;
        I.M = p->M;
        I.Mpad = p->Mpad;
        I.K = p->Mpad / 32;
        I.nw = nw;
        const RbmDev d = p->rbm_dev();
        I.W = d.W;
        I.b = d.b;
        I.Wq = d.Wq;
        I.bq = d.bq;
        I.op = o->dev();
        I.walkers = static_cast<int>(walkers[i]);
        I.seed = seeds[i];
        auto alloc = [&](size_t bytes) -> void* {
            b->bufs.push_back(std::make_unique<DevBuf>());
            if (b->bufs.back()->ensure(std::max<size_t>(bytes, 16)) != cudaSuccess) return nullptr;
            return b->bufs.back()->p;
        };
        const size_t B = walkers[i];
        I.eloc = static_cast<double2*>(alloc(sizeof(double2) * B));
        I.T = static_cast<float2*>(alloc(sizeof(float2) * B * p->Mpad));
        I.U = static_cast<float2*>(alloc(sizeof(float2) * B * p->Mpad));
        I.theta = static_cast<float2*>(alloc(sizeof(float2) * B * p->Mpad));
        I.en = static_cast<float2*>(alloc(sizeof(float2) * B * std::max(1, o->num_offdiag)));
        I.spins = static_cast<uint64_t*>(alloc(sizeof(uint64_t) * B * nw));
        I.rng_index = static_cast<uint64_t*>(alloc(sizeof(uint64_t) * B));
        I.chunks = static_cast<int>((B + kReduceWalkers - 1) / kReduceWalkers);
        const size_t elems = static_cast<size_t>(p->N + 1) * p->Mpad;
        const size_t params = 2 * static_cast<size_t>(p->N) + p->M + static_cast<size_t>(p->N) * p->M;
        I.part = static_cast<float2*>(alloc(sizeof(float2) * 3 * I.chunks * elems));
        I.grad = static_cast<double2*>(alloc(sizeof(double2) * params));
        I.emean = b->d_status.as<double2>() + i;
        // the batch's own copy of the site lists (the operator's are rebuilt when it is used
        // with another N), and per site whether the single-flip tile serves it: exactly one
        // off-diagonal string flips the site and flips it alone (reduce_task's test)
        int* site_ptr = static_cast<int*>(alloc(sizeof(int) * o->site_ptr.size()));
        int* site_slots = static_cast<int*>(alloc(sizeof(int) * o->site_slots.size()));
        if (!site_ptr || !site_slots) return fail(RBMG_ENOMEM, "batch: device allocation failed");
        RBMG_CK(cudaMemcpy(site_ptr, o->site_ptr.data(), sizeof(int) * o->site_ptr.size(), cudaMemcpyHostToDevice));
        RBMG_CK(cudaMemcpy(site_slots, o->site_slots.data(), sizeof(int) * o->site_slots.size(),
                           cudaMemcpyHostToDevice));
        I.site_ptr = site_ptr;
        I.site_slots = site_slots;
        {
            std::vector<int> string_of(std::max(1, o->num_offdiag), 0);
            for (int n = 0; n < o->S; n++)
                if (o->offdiag_slot[n] >= 0) string_of[o->offdiag_slot[n]] = n;
            std::vector<char> single(p->N);
            for (int site = 0; site < p->N; site++) {
                const int sb = o->site_ptr[site], se = o->site_ptr[site + 1];
                single[site] = se - sb == 1 && o->nflip[string_of[o->site_slots[sb]]] == 1;
            }
            b->single_flip.push_back(std::move(single));
        }
        b->max_elems = std::max(b->max_elems, static_cast<int>(elems));
        if (!I.eloc || !I.T || !I.U || !I.theta || !I.en || !I.spins || !I.rng_index || !I.part || !I.grad)
            return fail(RBMG_ENOMEM, "batch: device allocation failed");
        RBMG_CK(cudaMemset(I.rng_index, 0, sizeof(uint64_t) * B));
        RBMG_CK(cudaMemset(I.grad, 0, sizeof(double2) * 2 * p->N));   // alpha and beta
        b->psis.push_back(p);
        b->ops.push_back(o);
        b->walkers.push_back(walkers[i]);
        b->host_inst.push_back(I);
    }
    RBMG_CK(b->d_done.ensure(sizeof(unsigned int) * n));
    for (int i = 0; i < n; i++) b->host_inst[i].done = b->d_done.as<unsigned int>() + i;
    RBMG_CK(b->d_inst.ensure(sizeof(SInst) * n));
    RBMG_CK(cudaMemcpy(b->d_inst.p, b->host_inst.data(), sizeof(SInst) * n, cudaMemcpyHostToDevice));
    RBMG_CK(b->d_next.ensure(sizeof(unsigned int)));
    RBMG_CK(b->d_accepts.ensure(sizeof(unsigned long long)));
    const int r = batch_tasks(b.get());
    if (r != RBMG_OK) return r;
    *out = b.release();
    return RBMG_OK;
}

extern "C" int rbmg_batch_destroy(rbmg_batch* b) {
    delete b;
    return RBMG_OK;
}

extern "C" int rbmg_batch_set_shape(rbmg_batch* b, int warps_per_block, int rows) {
    if (!b || (warps_per_block != 2 && warps_per_block != 4 && warps_per_block != 8) || (rows != 8 && rows != 16))
        return fail(RBMG_EINVAL, "batch: warps per block in {2, 4, 8}, tile rows in {8, 16}");
    if (rows != b->rows) {
        b->rows = rows;
        const int r = batch_tasks(b);
        if (r != RBMG_OK) return r;
    }
    b->warps_per_block = warps_per_block;
    return RBMG_OK;
}

extern "C" int rbmg_batch_set_wait(rbmg_batch* b, double seconds, uint32_t extra_walkers) {
    if (!b || !(seconds > 0.0) || seconds > 60.0) return fail(RBMG_EINVAL, "batch: wait limit in (0, 60] s");
    b->wait_ns = static_cast<unsigned long long>(seconds * 1e9);
    b->wait_extra = extra_walkers;
    return RBMG_OK;
}

extern "C" int rbmg_batch_set_register_cap(rbmg_batch* b, int regs) {
    if (!b || (regs != 255 && regs != 128 && regs != 96))
        return fail(RBMG_EINVAL, "batch: register cap in {255, 128, 96}");
    b->regs = regs;
    return RBMG_OK;
}

extern "C" int rbmg_batch_get_register_cap(const rbmg_batch* b, int* regs) {
    if (!b || !regs) return fail(RBMG_EINVAL, "batch: null");
    *regs = b->regs;
    return RBMG_OK;
}

extern "C" int rbmg_batch_get_shape(const rbmg_batch* b, int* warps_per_block, int* rows, int* blocks) {
    if (!b) return fail(RBMG_EINVAL, "batch: null");
    if (warps_per_block) *warps_per_block = b->warps_per_block;
    if (rows) *rows = b->rows;
    if (blocks) *blocks = b->blocks;
    return RBMG_OK;
}

extern "C" int rbmg_batch_run(rbmg_batch* b, int therm, int sweeps) {
    if (!b || therm < 0 || sweeps < 0) return fail(RBMG_EINVAL, "batch run: bad arguments");
    b->therm = therm;
    b->sweeps = sweeps;
    return batch_replay(b);
}

// Times every candidate shape on `reps` replays of `sweeps` sweeps (the chains advance),
// keeps the fastest; ms_out [18] receives the candidates' mean milliseconds per replay,
// register caps 255, 128, 96 in turn, each in the order (2,8) (2,16) (4,8) (4,16) (8,8) (8,16).
extern "C" int rbmg_batch_autotune(rbmg_batch* b, int sweeps, int reps, double* ms_out) {
    if (!b || sweeps < 0 || reps <= 0) return fail(RBMG_EINVAL, "batch autotune: bad arguments");
    if (b->first) {   // start the chains outside the timing
        const int r = rbmg_batch_run(b, 0, 0);
        if (r != RBMG_OK) return r;
    }
    const int wpbs[3] = {2, 4, 8}, rowss[2] = {8, 16}, capss[3] = {255, 128, 96};
    double best = 1e300;
    int bw = 4, brows = 16, bregs = 255, c = 0;
    for (int regs : capss)
    for (int wpb : wpbs)
        for (int rows : rowss) {
            int r = rbmg_batch_set_shape(b, wpb, rows);
            if (r == RBMG_OK) r = rbmg_batch_set_register_cap(b, regs);
            if (r != RBMG_OK) return r;
            b->therm = 0;
            b->sweeps = sweeps;
            r = batch_replay(b);   // capture + warm-up
            if (r != RBMG_OK) return r;
            cudaEvent_t e0, e1;
            RBMG_CK(cudaEventCreate(&e0));
            RBMG_CK(cudaEventCreate(&e1));
            RBMG_CK(cudaEventRecord(e0, stream()));
            for (int k = 0; k < reps; k++) RBMG_CK(cudaGraphLaunch(b->exec, stream()));
            RBMG_CK(cudaEventRecord(e1, stream()));
            RBMG_CK(cudaEventSynchronize(e1));
            float ms = 0.0f;
            RBMG_CK(cudaEventElapsedTime(&ms, e0, e1));
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            int err = 0;
            RBMG_CK(batch_status(b, &err));
            if (err) return fail(RBMG_ETIMEOUT, "batch autotune: a reduction task timed out");
            const double per = ms / reps;
            if (ms_out) ms_out[c] = per;
            c++;
            if (per < best) {
                best = per;
                bw = wpb;
                brows = rows;
                bregs = regs;
            }
        }
    b->tuned_ms = best;
    const int r = rbmg_batch_set_shape(b, bw, brows);
    return r != RBMG_OK ? r : rbmg_batch_set_register_cap(b, bregs);
}

// results of the last replay for instance i: <E_loc> over its walkers, the reference's O_k
// gradient <E O*> + conj<E_k> - 2 <E> <O*> in the reference's parameter layout [2P] (alpha
// and beta entries 0), optionally the walkers' local energies [2 walkers]
extern "C" int rbmg_batch_result(const rbmg_batch* b, int i, double* energy, double* grad, double* eloc) {
    if (!b || i < 0 || i >= b->n || !energy) return fail(RBMG_EINVAL, "batch result: bad arguments");
    const SInst& I = b->host_inst[i];
    energy[0] = b->status[i].x;
    energy[1] = b->status[i].y;
    if (eloc) {
        prefault(eloc, sizeof(double2) * I.walkers);
        RBMG_CK(cudaMemcpy(eloc, I.eloc, sizeof(double2) * I.walkers, cudaMemcpyDeviceToHost));
    }
    if (grad) {
        const size_t params = 2 * static_cast<size_t>(I.N) + I.M + static_cast<size_t>(I.N) * I.M;
        prefault(grad, sizeof(double2) * params);
        RBMG_CK(cudaMemcpy(grad, I.grad, sizeof(double2) * params, cudaMemcpyDeviceToHost));
    }
    return RBMG_OK;
}

// the walkers' configurations of instance i after the last replay [walkers][ceil(N/64)]
extern "C" int rbmg_batch_spins(const rbmg_batch* b, int i, uint64_t* spins) {
    if (!b || i < 0 || i >= b->n || !spins) return fail(RBMG_EINVAL, "batch spins: bad arguments");
    const SInst& I = b->host_inst[i];
    RBMG_CK(cudaMemcpy(spins, I.spins, sizeof(uint64_t) * I.walkers * I.nw, cudaMemcpyDeviceToHost));
    return RBMG_OK;
}

extern "C" int rbmg_batch_info(const rbmg_batch* b, int* num_instances, uint64_t* accepts, double* tuned_ms) {
    if (!b) return fail(RBMG_EINVAL, "batch: null");
    if (num_instances) *num_instances = b->n;
    if (accepts) RBMG_CK(cudaMemcpy(accepts, b->d_accepts.p, sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    if (tuned_ms) *tuned_ms = b->tuned_ms;
    return RBMG_OK;
}
