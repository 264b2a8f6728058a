// PsiDeep / PsiPair kernels (include/quantum_state/PsiDeep.hpp:89-293, PsiPair.hpp:36-119).
//
// The general form has one CTA per configuration, thread j owning unit j of the layer being
// evaluated; complex nets without translation sums take several walkers or neighbours of a sample
// per CTA (deep_mc_pairs_kernel, deep_adjoint_pairs_kernel, deep_local64_kernel);
// the estimator kernels (local energies, O_k and E_k rows) run in FP64 -- for these
// nets log psi(s') - log psi(s) is the difference of two full forward passes, so FP32
// would cost ~1e-7 |log psi| per local-energy term -- while the Metropolis sampler runs
// in FP32;
// the layer's inputs, angles and activations live in shared memory; weights are read
// coalesced over j ([connectivity][size] layout, as the reference stores them).
// The backward pass gathers over the rhs connection lists compiled on the host in
// the reference's order (source/quantum_state/PsiDeep.cu:85-117).
#include <cstdlib>
#include <algorithm>
#include <functional>
#include <memory>
#include <type_traits>

#include "device_math.cuh"
#include "host.h"
#include "math64.cuh"
#include "reduce.h"

namespace rbmg {

namespace {

// ---------------------------------------------------------------- complex helpers
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename V> __device__ __forceinline__ V czero();
template <> __device__ __forceinline__ float2 czero<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ double2 czero<double2>() { return make_double2(0.0, 0.0); }
template <typename V> __device__ __forceinline__ V creal(double x);
template <> __device__ __forceinline__ float2 creal<float2>(double x) { return make_float2(float(x), 0.f); }
template <> __device__ __forceinline__ double2 creal<double2>(double x) { return make_double2(x, 0.0); }

// the activation in the reference's order of operations (math64.cuh has the faster form)
__device__ __forceinline__ double2 lc64_plain(double2 z) {
    const double s = z.x > 0.0 ? 1.0 : -1.0;
    double2 t = make_double2(s * 3.746646023906276 + z.x, z.y);
    t = cmul(z, t); t.x += 7.771429504240965;
    t = cmul(z, t); t.x += s * 10.2180213465;
    t = cmul(z, t); t.x += 9.19376335670885;
    const double2 num = make_double2(5.49914721954 - s * 2.16564366435 * z.x, -s * 2.16564366435 * z.y);
    const double den = t.x * t.x + t.y * t.y;
    return make_double2(s * 0.9003320053750442 * z.x + (num.x * t.x + num.y * t.y) / den - 0.598139,
                        s * 0.9003320053750442 * z.y + (num.y * t.x - num.x * t.y) / den);
}

// activation: the reference's rational log-cosh for complex nets, ReLU for the real
// nets of a PsiPair (include/quantum_state/psi_functions.hpp:118-125)
template <bool REAL> __device__ __forceinline__ float2 act(float2 a) {
    return REAL ? make_float2(a.x > 0.f ? a.x : 0.f, 0.f) : lc_c(a.x, a.y);
}
template <bool REAL> __device__ __forceinline__ double2 act(double2 a) {
    return REAL ? make_double2(a.x > 0.0 ? a.x : 0.0, 0.0) : lc64_plain(a);
}
// derivative: my_tanh for complex nets, 1 for the real nets (psi_functions.hpp:127-136)
template <bool REAL> __device__ __forceinline__ float2 dact(float2 a) {
    return REAL ? make_float2(1.f, 0.f) : tanh_c(a.x, a.y);
}
// my_tanh in FP64 (psi_functions.hpp:97-114)
__device__ __forceinline__ double2 tanh64(double2 z) {
    const double s = z.x > 0.0 ? 1.0 : -1.0;
    const double2 u = make_double2(s * z.x, s * z.y);
    double2 d = make_double2(u.x + 3.746646023906276, u.y);
    d = cmul(u, d); d.x += 7.771429504240965;
    d = cmul(u, d); d.x += 10.218021346543315;
    d = cmul(u, d); d.x += 9.19376335670885;
    double2 q = make_double2(6.746450656267947 + 0.9003320053750442 * u.x, 0.9003320053750442 * u.y);
    q = cmul(u, q); q.x += 26.632014683761202;
    q = cmul(u, q); q.x += 70.82878897882324;
    q = cmul(u, q); q.x += 146.36284300074402;
    q = cmul(u, q); q.x += 199.24474920889975;
    q = cmul(u, q); q.x += 177.6769746361748;
    q = cmul(u, q); q.x += 83.68563506532087;
    q = cmul(u, q);
    const double2 d2 = cmul(d, d);
    const double den = d2.x * d2.x + d2.y * d2.y;
    const double2 h = make_double2((q.x * d2.x + q.y * d2.y) / den, (q.y * d2.x - q.x * d2.y) / den);
    return make_double2(s * h.x, s * h.y);
}
template <bool REAL> __device__ __forceinline__ double2 dact(double2 a) {
    return REAL ? make_double2(1.0, 0.0) : tanh64(a);
}

template <typename V> struct W_of;
template <> struct W_of<float2> {
    static __device__ __forceinline__ const float2* w(const DeepNetDev& n, int l) { return n.w[l]; }
    static __device__ __forceinline__ const float2* b(const DeepNetDev& n, int l) { return n.b[l]; }
    static __device__ __forceinline__ const float2* fw(const DeepNetDev& n) { return n.fw; }
};
template <> struct W_of<double2> {
    static __device__ __forceinline__ const double2* w(const DeepNetDev& n, int l) { return n.w64[l]; }
    static __device__ __forceinline__ const double2* b(const DeepNetDev& n, int l) { return n.b64[l]; }
    static __device__ __forceinline__ const double2* fw(const DeepNetDev& n) { return n.fw64; }
};

// deterministic block sum of one complex value per thread; all threads receive it
template <typename V>
__device__ __forceinline__ V block_sum(V v, V* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
    }
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    V t = czero<V>();
    for (int q = 0; q < nwarps; q++) t = cadd(t, red[q]);
    return t;
}

__device__ __forceinline__ bool bit_up(const uint64_t* s, int i) { return (s[i >> 6] >> (i & 63)) & 1ull; }

// shared-memory layout of one configuration's evaluation
template <typename V>
struct Work {
    V* in;        // [width]
    V* out;       // [width]
    V* angles;    // [units] or null
    V* acts;      // [units] or null
    V* red;       // [32]
    uint64_t* s;  // [kMaxWords] spins being evaluated
};

// forward pass (PsiDeep.hpp:89-133) of one net on the spins in w.s; returns
// sum_j act_j * final_w_j; with STORE keeps every angle and activation
template <typename V, bool REAL, bool STORE>
__device__ V forward_once(const DeepNetDev& net, const uint64_t* s, Work<V>& w) {
    const int t = threadIdx.x;
    if (t < net.N) w.in[t] = creal<V>(bit_up(s, t) ? 1.0 : -1.0);
    __syncthreads();
    V* in = w.in;
    V* out = w.out;
    for (int l = 0; l < net.L; l++) {
        const int size = net.size[l], conn = net.conn[l];
        if (t < size) {
            const V* wl = W_of<V>::w(net, l);
            const int* ci = net.cidx[l];
            V a = czero<V>();
            for (int c = 0; c < conn; c++) a = cadd(a, cmul(wl[c * size + t], in[ci[c * size + t]]));
            a = cadd(a, W_of<V>::b(net, l)[t]);
            const V y = act<REAL>(a);
            if (STORE) {
                w.angles[net.begin_angle[l] + t] = a;
                w.acts[net.begin_angle[l] + t] = y;
            }
            out[t] = y;
        }
        __syncthreads();
        V* tmp = in;
        in = out;
        out = tmp;
    }
    const int last = net.size[net.L - 1];
    V term = czero<V>();
    if (t < last) term = cmul(in[t], W_of<V>::fw(net)[t]);
    return block_sum(term, w.red);
}

// layer 0's pre-activations of the spins s (the order of forward_once's layer 0)
__device__ void layer0_pre(const DeepNetDev& net, const uint64_t* s, float2* z0) {
    const int size = net.size[0], conn = net.conn[0];
    for (int u = threadIdx.x; u < size; u += blockDim.x) {
        const float2* wl = net.w[0];
        const int* ci = net.cidx[0];
        float2 a = czero<float2>();
        for (int c = 0; c < conn; c++)
            a = cadd(a, cmul(wl[c * size + u], creal<float2>(bit_up(s, ci[c * size + u]) ? 1.0 : -1.0)));
        z0[u] = cadd(a, net.b[0][u]);
    }
}

// forward pass of a complex net from its layer-0 pre-activations z0 (the rest as
// forward_once; with STORE keeps every angle and activation)
template <bool STORE = false>
__device__ float2 forward_from_z0(const DeepNetDev& net, const float2* z0, Work<float2>& w) {
    const int t = threadIdx.x;
    const int size0 = net.size[0];
    for (int u = t; u < size0; u += blockDim.x) {
        const float2 y = act<false>(z0[u]);
        if (STORE) {
            w.angles[net.begin_angle[0] + u] = z0[u];
            w.acts[net.begin_angle[0] + u] = y;
        }
        w.in[u] = y;
    }
    __syncthreads();
    float2* in = w.in;
    float2* out = w.out;
    for (int l = 1; l < net.L; l++) {
        const int size = net.size[l], conn = net.conn[l];
        if (t < size) {
            const float2* wl = net.w[l];
            const int* ci = net.cidx[l];
            float2 a = czero<float2>();
            for (int c = 0; c < conn; c++) a = cadd(a, cmul(wl[c * size + t], in[ci[c * size + t]]));
            a = cadd(a, net.b[l][t]);
            const float2 y = act<false>(a);
            if (STORE) {
                w.angles[net.begin_angle[l] + t] = a;
                w.acts[net.begin_angle[l] + t] = y;
            }
            out[t] = y;
        }
        __syncthreads();
        float2* tmp = in;
        in = out;
        out = tmp;
    }
    const int last = net.size[net.L - 1];
    float2 term = czero<float2>();
    if (t < last) term = cmul(in[t], net.fw[t]);
    return block_sum(term, w.red);
}

// log psi of one net with optional translational averaging (PsiDeep.hpp:135-169)
template <typename V, bool REAL>
__device__ V net_log_psi(const DeepNetDev& net, const uint64_t* s, Work<V>& w, uint64_t* shifted) {
    if (!net.ti) return forward_once<V, REAL, false>(net, s, w);
    V r = czero<V>();
    for (int shift = 0; shift < net.N; shift++) {
        __syncthreads();
        if (threadIdx.x == 0) {   // Spins_t<1>::rotate_left (include/Spins.h:280-285)
            const uint64_t x = s[0];
            uint64_t y = shift == 0 ? x : ((x << shift) | (x >> (net.N - shift)));
            if (net.N < 64) y &= (1ull << net.N) - 1ull;
            shifted[0] = y;
        }
        __syncthreads();
        r = cadd(r, forward_once<V, REAL, false>(net, shifted, w));
    }
    const double inv = 1.0 / net.N;
    r.x *= inv;
    r.y *= inv;
    return r;
}

// log psi of the state: one complex net, or (Re, Im) from the two real nets of a PsiPair
template <typename V>
__device__ V state_log_psi(const DeepNetDev& n0, const DeepNetDev& n1, int pair, const uint64_t* s, Work<V>& w,
                           uint64_t* shifted) {
    if (!pair) return net_log_psi<V, false>(n0, s, w, shifted);
    const V re = net_log_psi<V, true>(n0, s, w, shifted);
    const V im = net_log_psi<V, true>(n1, s, w, shifted);
    V r;
    r.x = re.x;
    r.y = im.x;
    return r;
}

// reverse pass (PsiDeep.hpp:214-293) after forward_once<STORE>; emit(k, value) with k
// counted from the first O_k entry (parameter index - 2N)
template <typename V, bool REAL, typename Emit>
__device__ void backward(const DeepNetDev& net, const uint64_t* s, Work<V>& w, V log_psi, Emit emit) {
    const int t = threadIdx.x;
    const int L = net.L;
    V* cur = w.in;
    V* nxt = w.out;
    for (int l = L - 1; l >= 0; l--) {
        const int size = net.size[l];
        V d = czero<V>();
        if (t < size) {
            const V ang = w.angles[net.begin_angle[l] + t];
            if (l == L - 1) {
                d = cmul(W_of<V>::fw(net)[t], dact<REAL>(ang));
            } else {
                const int nsize = net.size[l + 1];
                V acc = czero<V>();
                const V* wn = W_of<V>::w(net, l + 1);
                for (int e = net.rptr[l][t]; e < net.rptr[l][t + 1]; e++) {
                    const int q = net.rq[l][e];
                    acc = cadd(acc, cmul(wn[q], nxt[q % nsize]));
                }
                d = cmul(acc, dact<REAL>(ang));
            }
        }
        __syncthreads();
        if (t < size) {
            cur[t] = d;
            const int base = net.begin_params[l];
            emit(base + t, d);
            const int conn = net.conn[l];
            for (int c = 0; c < conn; c++) {
                const int src = net.cidx[l][c * size + t];
                const V in = l == 0 ? creal<V>(bit_up(s, src) ? 1.0 : -1.0) : w.acts[net.begin_angle[l - 1] + src];
                emit(base + size + c * size + t, cmul(d, in));
            }
        }
        __syncthreads();
        V* tmp = cur;
        cur = nxt;
        nxt = tmp;
    }
    // final weights: log psi * activation of the last layer (PsiDeep.hpp:285-292)
    const int last = net.size[L - 1];
    if (t < last) emit(net.P - 2 * net.N - last + t, cmul(log_psi, w.acts[net.begin_angle[L - 1] + t]));
    __syncthreads();
}

template <typename V>
__device__ Work<V> carve(void* base, const DeepNetDev& net, bool store) {
    Work<V> w;
    V* p = static_cast<V*>(base);
    const int width = net.width;
    w.red = p;
    p += 32;
    w.in = p;
    p += width;
    w.out = p;
    p += width;
    w.angles = store ? p : nullptr;
    if (store) p += net.units;
    w.acts = store ? p : nullptr;
    if (store) p += net.units;
    w.s = reinterpret_cast<uint64_t*>(p);
    return w;
}

__device__ __forceinline__ void load_config(const uint64_t* spins, uint64_t enum_base, int enumerate, long t, int N,
                                            uint64_t* s) {
    const int nw = (N + 63) / 64;
    if (threadIdx.x < kMaxWords) {
        uint64_t v = 0;
        if (enumerate) {
            if (threadIdx.x == 0) {
                v = enum_base + static_cast<uint64_t>(t);
                if (N < 64) v &= (1ull << N) - 1ull;
            }
        } else if (static_cast<int>(threadIdx.x) < nw) {
            v = spins[t * nw + threadIdx.x];
        }
        s[threadIdx.x] = v;
    }
    __syncthreads();
}

// string n applied to s: flipped configuration into sp, returns coef * phase (Operator.hpp:45-88)
__device__ double2 apply_string(const OpDev& op, int n, const uint64_t* s, uint64_t* sp) {
    int parity = 0;
    for (int k = 0; k < kMaxWords; k++) parity += __popcll(op.zmask[n * kMaxWords + k] & ~s[k]);
    const double sg = (parity & 1) ? -1.0 : 1.0;
    const double2 c = op.coef[n];
    const int yp = op.ypow[n] & 3;
    double2 r = yp == 0 ? c : (yp == 1 ? make_double2(c.y, -c.x) : (yp == 2 ? make_double2(-c.x, -c.y)
                                                                            : make_double2(-c.y, c.x)));
    __syncthreads();
    if (threadIdx.x < kMaxWords) {
        uint64_t v = s[threadIdx.x];
        for (int q = 0; q < op.nflip[n]; q++) {
            const int site = op.flip_sites[op.flip_off[n] + q];
            if ((site >> 6) == static_cast<int>(threadIdx.x)) v ^= 1ull << (site & 63);
        }
        sp[threadIdx.x] = v;
    }
    __syncthreads();
    return make_double2(sg * r.x, sg * r.y);
}

// ---------------------------------------------------------------- kernels
template <typename V>
__global__ void deep_logpsi_kernel(DeepNetDev n0, DeepNetDev n1, int pair, int count, const uint64_t* spins,
                                   uint64_t enum_base, int enumerate, double2* out) {
    extern __shared__ __align__(16) unsigned char smem[];
    Work<V> w = carve<V>(smem, n0, false);
    uint64_t* shifted = w.s + kMaxWords;
    const long t = blockIdx.x;
    if (t >= count) return;
    load_config(spins, enum_base, enumerate, t, n0.N, w.s);
    const V lp = state_log_psi<V>(n0, n1, pair, w.s, w, shifted);
    if (threadIdx.x == 0) out[t] = make_double2(lp.x, lp.y);
}

// local energy (Operator.hpp:90-115); FP32 or FP64 evaluation; with PRIME also
// log psi'(s) - log psi(s) for the Hilbert-space distance
template <typename V, bool PRIME>
__global__ void deep_eloc_kernel(DeepNetDev n0, DeepNetDev n1, int pair, DeepNetDev p0, DeepNetDev p1, OpDev op,
                                 int count, const uint64_t* spins, uint64_t enum_base, int enumerate, double2* eloc,
                                 double2* dlp) {
    extern __shared__ __align__(16) unsigned char smem[];
    Work<V> w = carve<V>(smem, n0.width >= p0.width ? n0 : p0, false);
    uint64_t* sp = w.s + kMaxWords;
    uint64_t* shifted = sp + kMaxWords;
    const long t = blockIdx.x;
    if (t >= count) return;
    load_config(spins, enum_base, enumerate, t, n0.N, w.s);
    const V lp = state_log_psi<V>(n0, n1, pair, w.s, w, shifted);
    double er = 0.0, ei = 0.0;
    for (int n = 0; n < op.S; n++) {
        const double2 cf = apply_string(op, n, w.s, sp);
        if (op.nflip[n] == 0) {
            er += cf.x;
            ei += cf.y;
            continue;
        }
        const V lq = state_log_psi<V>(n0, n1, pair, sp, w, shifted);
        if (threadIdx.x >= 32) continue;   // thread 0 writes the sum: the FP64 exponentials of one warp
        const double dr = static_cast<double>(lq.x) - static_cast<double>(lp.x);
        const double di = static_cast<double>(lq.y) - static_cast<double>(lp.y);
        const double m = exp(dr);
        const double xr = m * cos(di), xi = m * sin(di);
        er += cf.x * xr - cf.y * xi;
        ei += cf.x * xi + cf.y * xr;
    }
    double2 d = make_double2(0.0, 0.0);
    if (PRIME) {
        const V lq = state_log_psi<V>(p0, p1, pair, w.s, w, shifted);
        d = make_double2(static_cast<double>(lq.x) - static_cast<double>(lp.x),
                         static_cast<double>(lq.y) - static_cast<double>(lp.y));
    }
    if (threadIdx.x == 0) {
        if (eloc) eloc[t] = make_double2(er, ei);
        if (PRIME) dlp[t] = d;
    }
}

// O_k rows [count][P - 2N] of one net (complex, or a real PsiPair net stored as (x, 0))
template <bool REAL>
__global__ void deep_ok_kernel(DeepNetDev net, int count, const uint64_t* spins, uint64_t enum_base, int enumerate,
                               double2* rows, long ld) {
    extern __shared__ __align__(16) unsigned char smem[];
    Work<double2> w = carve<double2>(smem, net, true);
    const long t = blockIdx.x;
    if (t >= count) return;
    load_config(spins, enum_base, enumerate, t, net.N, w.s);
    const double2 lp = forward_once<double2, REAL, true>(net, w.s, w);
    double2* row = rows + t * ld;
    backward<double2, REAL>(net, w.s, w, lp, [&](int k, double2 v) { row[k] = v; });
}

// FP64 local energy of a complex net (no translation sums) and, with GRAD, per sample the O_k
// row and the centred E_k row
//   Ek[s] = (E_diag - E0) O(s) + sum_{off-diagonal n} e_n O(s'_n)
// (Operator.hpp:145-179 with the shift of the gradient estimator); with prime, also
// log psi'(s) - log psi(s).  One block per sample.
//
// Bound by the FP64 pipe, whose instructions take 16 cycles of the SM whatever the number of
// active lanes, so the work is counted and packed: `nb` neighbours at a time, their units side
// by side in the threads; a neighbour's layer 0 is the sample's moved by the flipped spins; an
// activation and its derivative come from one D(u) (math64.cuh); exp, cos and sin run one
// neighbour a lane (in every thread of a block before); the reverse pass carries e_n delta and
// a parameter's entries are summed over the neighbours of a batch before its one read and write
// of the row (one per neighbour before, and ten FP64 operations per entry instead of four).
// 512 samples of the 20-40-20-10 net, 20 strings: gradient pass 2066 -> 489 us, energies 750 ->
// 171 us.  128 threads a block up to 128 units, 512 above, whose batches are small and which wait for
// the rows and the weights: 256 samples, N = 32, ms of the gradient pass with one neighbour at a time /
// 128 threads / 512: 200-100-50 22.8 / 10.7 / 8.6, 256-256 55.9 / 37.3 / 27.7, 400-400 139 / 166 / 72,
// 512-512 320 / 568 / 205; energies and log psi' of 1024 samples of 72-30 3.21 / 0.99 / 1.09.
size_t deep_local64_smem(const DeepNetDev& n, int nb, bool grad) {
    return sizeof(double2) * ((grad ? 2 : 1) * static_cast<size_t>(nb) * n.units + n.size[0] + 2 * nb) +
           sizeof(uint64_t) * (1 + nb) * kMaxWords;
}

template <bool GRAD, int T>
__global__ void __launch_bounds__(T, 1024 / T) deep_local64_kernel(DeepNetDev net, OpDev op, int count,
                                                                  const uint64_t* spins, uint64_t enum_base,
                                                                  int enumerate, int nbatch, DeepNetDev prime,
                                                                  double2* dlp, double2 e_shift, double2* eloc,
                                                                  double2* Orows, double2* Ekrows, long ld) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int units = net.units, size0 = net.size[0], L = net.L;
    double2* A = reinterpret_cast<double2*>(smem);           // [nb][units] activations
    double2* H = A + nbatch * units;                         // GRAD: [nb][units] derivatives, then e_n delta
    double2* z0s = GRAD ? H + nbatch * units : H;            // [size0] the sample's layer 0
    double2* lq = z0s + size0;                               // [nb] log psi
    double2* en = lq + nbatch;                               // [nb] terms e_n
    uint64_t* s = reinterpret_cast<uint64_t*>(en + nbatch);  // [kMaxWords] the sample
    uint64_t* sp = s + kMaxWords;                            // [nb][kMaxWords] the neighbours
    const long t = blockIdx.x;
    if (t >= count) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    load_config(spins, enum_base, enumerate, t, net.N, s);
    for (int u = tid; u < size0; u += T) {
        double2 a = net.b64[0][u];
        for (int c = 0; c < net.conn[0]; c++) {
            const double2 w = net.w64[0][c * size0 + u];
            const double sg = bit_up(s, net.cidx[0][c * size0 + u]) ? 1.0 : -1.0;
            a.x = fma(sg, w.x, a.x);
            a.y = fma(sg, w.y, a.y);
        }
        z0s[u] = a;
    }
    __syncthreads();
    // activations (and derivatives) of nb configurations whose layer 0 is z0of(k, u); log psi to lq
    auto forward = [&](auto z0of, int nb) {
        const DeepNetDev& n = net;
        auto unit = [&](int k, int at, double2 z) {
            const Lc64 f = lc64(z);
            A[k * units + at] = f.value();
            if (GRAD) H[k * units + at] = f.tanh();
        };
        for (int e = tid; e < nb * n.size[0]; e += T) {
            const int k = e / n.size[0], u = e - k * n.size[0];
            unit(k, u, z0of(k, u));
        }
        __syncthreads();
        for (int l = 1; l < L; l++) {
            const int size = n.size[l], conn = n.conn[l], at = n.begin_angle[l], below = n.begin_angle[l - 1];
            const int* ci = n.cidx[l];
            const double2* w = n.w64[l];
            for (int e = tid; e < nb * size; e += T) {
                const int k = e / size, u = e - k * size;
                const double2* in = A + k * units + below;
                double2 a = n.b64[l][u], b = make_double2(0.0, 0.0);
                for (int c = 0; c < conn; c++) {
                    const double2 wv = w[c * size + u], x = in[ci[c * size + u]];
                    a.x = fma(wv.x, x.x, a.x);
                    b.x = fma(-wv.y, x.y, b.x);
                    a.y = fma(wv.x, x.y, a.y);
                    b.y = fma(wv.y, x.x, b.y);
                }
                unit(k, at + u, cadd(a, b));
            }
            __syncthreads();
        }
        const int last = n.size[L - 1];
        for (int k = warp; k < nb; k += T / 32) {
            double2 v = make_double2(0.0, 0.0);
            for (int u = lane; u < last; u += 32) v = cadd(v, cmul(A[k * units + n.begin_angle[L - 1] + u], n.fw64[u]));
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
                v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
                v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
            }
            if (lane == 0) lq[k] = v;
        }
        __syncthreads();
    };
    // H: en[k] delta_l of nb configurations
    auto backward = [&](int nb) {
        for (int l = L - 1; l >= 0; l--) {
            const int size = net.size[l], at = net.begin_angle[l];
            for (int e = tid; e < nb * size; e += T) {
                const int k = e / size, u = e - k * size;
                double2 a = make_double2(0.0, 0.0);
                if (l == L - 1) {
                    a = cmul(en[k], net.fw64[u]);
                } else {
                    const int above = net.size[l + 1];
                    const double2* d = H + k * units + net.begin_angle[l + 1];
                    const double2* w = net.w64[l + 1];
                    for (int q = net.rptr[l][u]; q < net.rptr[l][u + 1]; q++) {
                        const int i = net.rq[l][q];
                        const double2 wv = w[i], x = d[i % above];
                        a.x = fma(wv.x, x.x, fma(-wv.y, x.y, a.x));
                        a.y = fma(wv.x, x.y, fma(wv.y, x.x, a.y));
                    }
                }
                H[k * units + at + u] = cmul(a, H[k * units + at + u]);
            }
            __syncthreads();
        }
    };
    // parameter k (counted from the first O_k entry): emit(k, sum over the nb configurations)
    auto parameters = [&](int nb, const uint64_t* cfg, auto emit) {
        for (int l = 0; l < L; l++) {
            const int size = net.size[l], total = size + net.conn[l] * size, at = net.begin_angle[l];
            for (int e = tid; e < total; e += T) {
                double2 v = make_double2(0.0, 0.0);
                if (e < size) {
                    for (int k = 0; k < nb; k++) v = cadd(v, H[k * units + at + e]);
                } else {
                    const int u = (e - size) % size, src = net.cidx[l][e - size];
                    for (int k = 0; k < nb; k++) {
                        const double2 d = H[k * units + at + u];
                        if (l == 0) {
                            const double sg = bit_up(cfg + k * kMaxWords, src) ? 1.0 : -1.0;
                            v.x = fma(sg, d.x, v.x);
                            v.y = fma(sg, d.y, v.y);
                        } else {
                            const double2 a = A[k * units + net.begin_angle[l - 1] + src];
                            v.x = fma(d.x, a.x, fma(-d.y, a.y, v.x));
                            v.y = fma(d.x, a.y, fma(d.y, a.x, v.y));
                        }
                    }
                }
                emit(net.begin_params[l] + e, v);
            }
        }
        // final weights: log psi * activation of the last layer (PsiDeep.hpp:285-292)
        const int last = net.size[L - 1];
        for (int u = tid; u < last; u += T) {
            double2 v = make_double2(0.0, 0.0);
            for (int k = 0; k < nb; k++)
                v = cadd(v, cmul(cmul(en[k], lq[k]), A[k * units + net.begin_angle[L - 1] + u]));
            emit(net.P - 2 * net.N - last + u, v);
        }
    };
    auto factor = [&](int n) {
        int parity = 0;
        for (int k = 0; k < kMaxWords; k++) parity += __popcll(op.zmask[n * kMaxWords + k] & ~s[k]);
        const double2 c = op.coef[n];
        const int yp = op.ypow[n] & 3;
        const double2 r = yp == 0 ? c : (yp == 1 ? make_double2(c.y, -c.x)
                                                 : (yp == 2 ? make_double2(-c.x, -c.y) : make_double2(-c.y, c.x)));
        return (parity & 1) ? make_double2(-r.x, -r.y) : r;
    };
    auto warp_sum = [&](double2 v) {
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
        }
        return v;
    };
    forward([&](int, int u) { return z0s[u]; }, 1);
    const double2 lp = lq[0];
    double2* orow = Orows + t * ld;
    double2* erow = Ekrows + t * ld;
    // the diagonal strings (every warp: the E_k row needs their sum)
    double2 diag = make_double2(0.0, 0.0);
    for (int n = lane; n < op.S; n += 32)
        if (op.nflip[n] == 0) diag = cadd(diag, factor(n));
    diag = warp_sum(diag);
    if (GRAD) {
        if (tid == 0) en[0] = make_double2(1.0, 0.0);
        __syncthreads();
        backward(1);
        const double2 c = make_double2(diag.x - e_shift.x, diag.y - e_shift.y);
        parameters(1, s, [&](int k, double2 v) {
            orow[k] = v;
            erow[k] = cmul(c, v);
        });
        __syncthreads();
    }
    double2 E = make_double2(0.0, 0.0);   // warp 0: the neighbours' terms, a lane's own
    for (int q = 0; q < op.num_offdiag; q += nbatch) {
        const int nb = min(nbatch, op.num_offdiag - q);
        for (int i = tid; i < nb * kMaxWords; i += T) {
            const int k = i / kMaxWords, word = i - k * kMaxWords, n = op.offdiag[q + k];
            uint64_t v = s[word];
            for (int f = 0; f < op.nflip[n]; f++) {
                const int site = op.flip_sites[op.flip_off[n] + f];
                if ((site >> 6) == word) v ^= 1ull << (site & 63);
            }
            sp[i] = v;
        }
        forward([&](int k, int u) {
            double2 z = z0s[u];
            const int n = op.offdiag[q + k];
            for (int f = 0; f < op.nflip[n]; f++) {
                const int site = op.flip_sites[op.flip_off[n] + f];
                const double ts = bit_up(s, site) ? -2.0 : 2.0;
                for (int d = 0; d < net.w0n; d++) {
                    const double2 w = net.w064[(static_cast<long>(d) * net.N + site) * size0 + u];
                    z.x = fma(ts, w.x, z.x);
                    z.y = fma(ts, w.y, z.y);
                }
            }
            return z;
        }, nb);
        if (warp == 0 && lane < nb) {
            const double2 cf = factor(op.offdiag[q + lane]);
            const double m = exp(lq[lane].x - lp.x);
            double sn, cs;
            sincos(lq[lane].y - lp.y, &sn, &cs);
            const double2 e = cmul(cf, make_double2(m * cs, m * sn));
            en[lane] = e;
            E = cadd(E, e);
        }
        __syncthreads();
        if (GRAD) {
            backward(nb);
            parameters(nb, sp, [&](int k, double2 v) { erow[k] = cadd(erow[k], v); });
            __syncthreads();
        }
    }
    if (warp == 0) {
        E = warp_sum(E);
        if (lane == 0 && eloc) eloc[t] = cadd(diag, E);
    }
    if (dlp) {
        // log psi'(s) - log psi(s) by forward_once's operations in its order: the distance is a
        // difference of nearly equal sums, down to the last bits of these two
        auto plain = [&](const DeepNetDev& n) {
            for (int l = 0; l < L; l++) {
                const int size = n.size[l], conn = n.conn[l];
                for (int u = tid; u < size; u += T) {
                    double2 a = make_double2(0.0, 0.0);
                    for (int c = 0; c < conn; c++) {
                        const int i = n.cidx[l][c * size + u];
                        const double2 x = l == 0 ? make_double2(bit_up(s, i) ? 1.0 : -1.0, 0.0)
                                                 : A[n.begin_angle[l - 1] + i];
                        a = cadd(a, cmul(n.w64[l][c * size + u], x));
                    }
                    A[n.begin_angle[l] + u] = lc64_plain(cadd(a, n.b64[l][u]));
                }
                __syncthreads();
            }
            const int last = n.size[L - 1];
            double2 r = make_double2(0.0, 0.0);
            for (int q = 0; q < last; q += 32)
                r = cadd(r, warp_sum(q + lane < last ? cmul(A[n.begin_angle[L - 1] + q + lane], n.fw64[q + lane])
                                                     : make_double2(0.0, 0.0)));
            __syncthreads();
            return r;
        };
        const double2 l0 = plain(net), l1 = plain(prime);
        if (tid == 0) dlp[t] = make_double2(l1.x - l0.x, l1.y - l0.y);
    }
}

// sums over the samples of the O_k and E_k rows (FP64), one pass over both:
//   0: c1 O, 1: c2 conj(O), 2: c1 Ek, 3 (c3): c3 Ek;  partial [split][4][P]
__global__ void __launch_bounds__(128) row_sums_kernel(int count, int P, const double2* __restrict__ c1,
                                                       const double2* __restrict__ c2, const double2* __restrict__ c3,
                                                       const double2* __restrict__ O, const double2* __restrict__ Ek,
                                                       long ld, double2* __restrict__ partial, int per_split) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const long s0 = static_cast<long>(blockIdx.y) * per_split;
    const long s1 = min(static_cast<long>(count), s0 + per_split);
    if (k >= P) return;
    double2 a[4] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
#pragma unroll 2
    for (long s = s0; s < s1; s++) {
        const double2 o = O[s * ld + k], e = Ek[s * ld + k], u = c1[s], v = c2[s];
        a[0] = cadd(a[0], cmul(u, o));
        a[1] = cadd(a[1], cmul(v, make_double2(o.x, -o.y)));
        a[2] = cadd(a[2], cmul(u, e));
        if (c3) a[3] = cadd(a[3], cmul(c3[s], e));
    }
#pragma unroll
    for (int q = 0; q < 4; q++) partial[(static_cast<long>(blockIdx.y) * 4 + q) * P + k] = a[q];
}

struct RowSums {
    double2* out[4];
};
__global__ void __launch_bounds__(128) row_sums_finish_kernel(int P, int splits, const double2* __restrict__ partial,
                                                              RowSums sums) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
    if (k >= P || !sums.out[q]) return;
    double2 a = make_double2(0.0, 0.0);
#pragma unroll 8
    for (int z = 0; z < splits; z++) a = cadd(a, partial[(static_cast<long>(z) * 4 + q) * P + k]);
    sums.out[q][k] = cadd(sums.out[q][k], a);
}

// out[k] += sum_s c[s] f(A[s][k]) over count samples, f = conj if conj_a (FP64)
__global__ void col_reduce_kernel(int count, int P, const double2* __restrict__ c, const double2* __restrict__ A,
                                  long ld, int conj_a, double2* __restrict__ partial, int per_split) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const long s0 = static_cast<long>(blockIdx.y) * per_split;
    const long s1 = min(static_cast<long>(count), s0 + per_split);
    if (k >= P) return;
    double2 acc = make_double2(0.0, 0.0);
    for (long s = s0; s < s1; s++) {
        double2 a = A[s * ld + k];
        if (conj_a) a.y = -a.y;
        acc = cadd(acc, cmul(c[s], a));
    }
    partial[static_cast<long>(blockIdx.y) * P + k] = acc;
}

__global__ void col_finish_kernel(int P, int splits, const double2* __restrict__ partial, double2* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P) return;
    double2 a = make_double2(0.0, 0.0);
    for (int z = 0; z < splits; z++) {
        a.x += partial[static_cast<long>(z) * P + k].x;
        a.y += partial[static_cast<long>(z) * P + k].y;
    }
    out[k].x += a.x;
    out[k].y += a.y;
}

// Metropolis for PsiDeep / PsiPair: one CTA per walker, full forward pass per proposal
// (PsiDeep.hpp:191-194: angles are not updated incrementally; single flips of a complex
// net move layer 0 incrementally here, and run several walkers per CTA in
// deep_mc_pairs_kernel).  Fast sweep
// (MonteCarloLoop.hpp:162-171): the proposal flips the AND of fast_tries random
// configurations, N such updates per thermalisation sweep and one per sampling sweep.
__global__ void deep_mc_kernel(DeepNetDev n0, DeepNetDev n1, int pair, McLaunch L) {
    extern __shared__ __align__(16) unsigned char smem[];
    Work<float2> w = carve<float2>(smem, n0, false);
    uint64_t* sp = w.s + kMaxWords;
    uint64_t* shifted = sp + kMaxWords;
    const int walker = blockIdx.x;
    if (walker >= L.B) return;
    const int N = n0.N, nw = (N + 63) / 64;
    WalkerRng rng;
    rng.init(L.seed, L.walker_base + static_cast<uint32_t>(walker), L.rng_index[walker]);
    // every thread draws the same words, so all threads agree without a broadcast
    uint64_t s[kMaxWords] = {0, 0, 0, 0};
    if (L.init) {
        for (int k = 0; k < nw; k++) {
            const uint64_t lo = rng.next();
            const uint64_t hi = rng.next();
            s[k] = lo | (hi << 32);
        }
        if (N / 64 < nw) s[N / 64] &= (1ull << (N % 64)) - 1ull;
    } else {
        for (int k = 0; k < nw; k++) s[k] = L.spins[static_cast<long>(walker) * nw + k];
    }
    if (threadIdx.x < kMaxWords) w.s[threadIdx.x] = s[threadIdx.x];
    __syncthreads();
    float lpr = state_log_psi<float2>(n0, n1, pair, w.s, w, shifted).x;
    // single-flip proposals of a complex net move layer 0's pre-activations by the flipped
    // spin's connections (z0' = z0 - 2 s_i W0[i, :]) and evaluate the later layers only;
    // z0 and log psi are recomputed from the spins at the start of every sweep
    const bool incr = L.fast_tries == 0 && !pair && !n0.ti;
    float2* z0 = reinterpret_cast<float2*>(shifted + kMaxWords);   // [size[0]] the state's
    float2* z0p = z0 + n0.size[0];                                   // [size[0]] a proposal's
    unsigned long long acc = 0, props = 0;
    const int total = L.n_therm + L.n_samples * L.sweeps_per_sample;
    int sample = 0;
    for (int sw = 0; sw < total; sw++) {
        const int updates = (L.fast_tries > 0 && sw >= L.n_therm) ? 1 : N;
        if (incr) {
            __syncthreads();
            layer0_pre(n0, w.s, z0);
            __syncthreads();
            lpr = forward_from_z0(n0, z0, w).x;
        }
        for (int p = 0; p < updates; p++) {
            int site = -1;
            if (L.fast_tries > 0) {
                // every thread draws the same mask words
                uint64_t m[kMaxWords] = {0, 0, 0, 0};
                for (int t = 0; t < L.fast_tries; t++) {
                    for (int k = 0; k < nw; k++) {
                        const uint64_t lo = rng.next();
                        const uint64_t hi = rng.next();
                        const uint64_t v = lo | (hi << 32);
                        m[k] = t == 0 ? v : (m[k] & v);
                    }
                }
                if (N / 64 < nw) m[N / 64] &= (1ull << (N % 64)) - 1ull;
                __syncthreads();
                if (threadIdx.x < kMaxWords) {
                    uint64_t v = w.s[threadIdx.x];
                    for (int k = 0; k < kMaxWords; k++)
                        if (k == static_cast<int>(threadIdx.x)) v ^= m[k];
                    sp[threadIdx.x] = v;
                }
            } else {
                site = static_cast<int>(rng.next() % static_cast<uint32_t>(N));
                __syncthreads();
                if (threadIdx.x < kMaxWords) {
                    uint64_t v = w.s[threadIdx.x];
                    if ((site >> 6) == static_cast<int>(threadIdx.x)) v ^= 1ull << (site & 63);
                    sp[threadIdx.x] = v;
                }
                if (incr)
                    for (int u = threadIdx.x; u < n0.size[0]; u += blockDim.x) z0p[u] = z0[u];
            }
            __syncthreads();
            float nl;
            if (incr && site >= 0) {
                const float two_s = bit_up(w.s, site) ? -2.0f : 2.0f;
                const int size0 = n0.size[0];
                for (int q = n0.sptr[site] + threadIdx.x; q < n0.sptr[site + 1]; q += blockDim.x) {
                    const int e = n0.sq[q];
                    const float2 wv = n0.w[0][e];
                    float2* z = z0p + e % size0;
                    atomicAdd(&z->x, two_s * wv.x);
                    atomicAdd(&z->y, two_s * wv.y);
                }
                __syncthreads();
                nl = forward_from_z0(n0, z0p, w).x;
            } else {
                nl = state_log_psi<float2>(n0, n1, pair, sp, w, shifted).x;
            }
            const float delta = nl - lpr;
            bool accept = delta > 0.0f;
            if (!accept) accept = rng.uniform() <= expf_det(2.0f * delta);
            __syncthreads();
            if (accept) {
                if (threadIdx.x < kMaxWords) w.s[threadIdx.x] = sp[threadIdx.x];
                lpr = nl;
                acc++;
                if (incr && site >= 0) {
                    float2* tz = z0;
                    z0 = z0p;
                    z0p = tz;
                }
            }
            props++;
            __syncthreads();
        }
        const int done = sw + 1 - L.n_therm;
        if (done > 0 && done % L.sweeps_per_sample == 0) {
            const long row = static_cast<long>(L.sample_base + sample) * L.B + walker;
            if (L.sample_spins && threadIdx.x < nw) L.sample_spins[row * nw + threadIdx.x] = w.s[threadIdx.x];
            sample++;
        }
    }
    __syncthreads();
    if (threadIdx.x < nw) L.spins[static_cast<long>(walker) * nw + threadIdx.x] = w.s[threadIdx.x];
    if (threadIdx.x == 0) {
        L.rng_index[walker] = rng.index;
        L.accepts[walker] += acc;
        L.proposals[walker] += props;
    }
}

// ---------------------------------------------------------------- several configurations a block
// Two configurations lie side by side, (x0, x1, y0, y1), and every operation is a packed one on
// both.  A thread evaluates one unit of a layer for NP such pairs: a weight and its connection
// index are read once for 2 NP multiply-adds, whose inputs are shared by the whole warp where
// the layer is dense.  Each configuration's sums are forward_once's, in its order.
struct CPair {
    pair_t re, im;
};
__device__ __forceinline__ CPair ld_pair(const float4* p) {
    const float4 v = *p;
    return CPair{pk2(v.x, v.y), pk2(v.z, v.w)};
}
__device__ __forceinline__ void st_pair(float4* p, CPair v) {
    float4 o;
    up2(v.re, o.x, o.y);
    up2(v.im, o.z, o.w);
    *p = o;
}
// a += w b for both configurations (cadd(a, cmul(w, b)))
__device__ __forceinline__ void cmac(CPair& a, float2 w, CPair b) {
    const pair_t wx = splat2(w.x), wy = splat2(w.y), nwy = splat2(-w.y);
    a.re = add2(a.re, fma2(wx, b.re, mul2(nwy, b.im)));
    a.im = add2(a.im, fma2(wx, b.im, mul2(wy, b.re)));
}
__device__ __forceinline__ CPair cmul(CPair a, CPair b) {
    const pair_t nay = neg2(a.im);
    return CPair{fma2(a.re, b.re, mul2(nay, b.im)), fma2(a.re, b.im, mul2(a.im, b.re))};
}
__device__ __forceinline__ CPair act_pair(CPair z) {
    const Pair2 y = lc_c2(z.re, z.im);
    return CPair{y.re, y.im};
}
__device__ __forceinline__ CPair dact_pair(CPair z) {
    float x0, x1, y0, y1;
    up2(z.re, x0, x1);
    up2(z.im, y0, y1);
    const float2 a = tanh_c(x0, y0), b = tanh_c(x1, y1);
    return CPair{pk2(a.x, b.x), pk2(a.y, b.y)};
}

// sums over the connections of `size` units for `pairs` pairs, NP of them per thread: weight
// w[c * size + t] of connection c times the input in[.][c] (a dense layer: the input is shared
// by the warp) or in[.][ci[c * size + t]]; emit(pair, t, sum)
template <int T, int NP, bool DENSE, typename Emit>
__device__ __forceinline__ void layer_sums(int size, int conn, const float2* __restrict__ w,
                                           const int* __restrict__ ci, const float4* in, int in_size, int pairs,
                                           Emit emit) {
    const int groups = pairs / NP;
    for (int item = threadIdx.x; item < size * groups; item += T) {
        const int grp = item / size, t = item - grp * size;
        const float4* x = in + grp * NP * in_size;
        CPair a[NP];
#pragma unroll
        for (int p = 0; p < NP; p++) a[p] = CPair{splat2(0.0f), splat2(0.0f)};
#pragma unroll 8
        for (int c = 0; c < conn; c++) {
            const float2 wv = __ldg(w + c * size + t);
            const int i = DENSE ? c : __ldg(ci + c * size + t);
#pragma unroll
            for (int p = 0; p < NP; p++) cmac(a[p], wv, ld_pair(x + p * in_size + i));
        }
#pragma unroll
        for (int p = 0; p < NP; p++) emit(grp * NP + p, t, a[p]);
    }
}

// pairs per thread of T: as many as leave work for half of the threads
template <int T, int PAIRS, bool DENSE, typename Emit>
__device__ __forceinline__ void layer_sums_split(int size, int conn, const float2* w, const int* ci, const float4* in,
                                                 int in_size, Emit emit) {
    if (PAIRS >= 4 && 2 * size >= T)
        layer_sums<T, (PAIRS >= 4 ? 4 : 1), DENSE>(size, conn, w, ci, in, in_size, PAIRS, emit);
    else if (PAIRS >= 2 && size * PAIRS >= T)
        layer_sums<T, (PAIRS >= 2 ? 2 : 1), DENSE>(size, conn, w, ci, in, in_size, PAIRS, emit);
    else layer_sums<T, 1, DENSE>(size, conn, w, ci, in, in_size, PAIRS, emit);
}

// layers 1 .. L - 1 from layer 0's activations in bufs[0]; layer l's activations go to
// bufs[l & 1], emit(l, pair, t, angle, activation) sees them.  Ends with a barrier.
template <int T, int PAIRS, typename Emit>
__device__ __forceinline__ void forward_pairs(const DeepNetDev& net, float4* const (&bufs)[2], Emit emit) {
    __syncthreads();
    for (int l = 1; l < net.L; l++) {
        const int size = net.size[l], conn = net.conn[l], below = net.size[l - 1];
        const float4* in = bufs[(l - 1) & 1];
        float4* out = bufs[l & 1];
        const float2* bias = net.b[l];
        auto done = [&](int p, int t, CPair a) {
            const float2 bv = __ldg(bias + t);
            const CPair z{add2(a.re, splat2(bv.x)), add2(a.im, splat2(bv.y))};
            const CPair y = act_pair(z);
            st_pair(out + p * size + t, y);
            emit(l, p, t, z, y);
        };
        if (net.wt[l]) layer_sums_split<T, PAIRS, true>(size, conn, net.w[l], nullptr, in, below, done);
        else layer_sums_split<T, PAIRS, false>(size, conn, net.w[l], net.cidx[l], in, below, done);
        __syncthreads();
    }
}

// sum_j act_j fw_j of one pair by a warp (block_sum's order); every lane receives it
__device__ __forceinline__ CPair final_sum(const DeepNetDev& net, const float4* in, int lane) {
    const int last = net.size[net.L - 1];
    CPair r{splat2(0.0f), splat2(0.0f)};
    for (int q = 0; q < last; q += 32) {
        CPair v{splat2(0.0f), splat2(0.0f)};
        if (q + lane < last) {
            const float2 f = net.fw[q + lane];
            v = cmul(ld_pair(in + q + lane), CPair{splat2(f.x), splat2(f.y)});
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            v.re = add2(v.re, __shfl_xor_sync(0xffffffffu, v.re, off));
            v.im = add2(v.im, __shfl_xor_sync(0xffffffffu, v.im, off));
        }
        r.re = add2(r.re, v.re);
        r.im = add2(r.im, v.im);
    }
    return r;
}

// layer 0's pre-activation of unit u moved by a flip of `site` (ts = 2 x the new spin)
__device__ __forceinline__ float2 move_z0(const DeepNetDev& net, int site, float ts, int u, float2 z) {
    for (int d = 0; d < net.w0n; d++) {
        const float2 w = __ldg(net.w0 + (static_cast<long>(d) * net.N + site) * net.size[0] + u);
        z.x = __fmaf_rn(ts, w.x, z.x);   // ts = +-2: the product is exact
        z.y = __fmaf_rn(ts, w.y, z.y);
    }
    return z;
}

// float4 of the two activation buffers: layers 0 and 2, layer 1
__host__ __device__ inline int pair_buf(const DeepNetDev& n, int which) {
    return which == 0 ? (n.L > 2 && n.size[2] > n.size[0] ? n.size[2] : n.size[0]) : (n.L > 1 ? n.size[1] : 0);
}

size_t deep_mc_pairs_smem(const DeepNetDev& n, int pairs) {
    return sizeof(float4) * pairs * (n.size[0] + pair_buf(n, 0) + pair_buf(n, 1)) +
           2 * pairs * (sizeof(uint64_t) * ((n.N + 63) / 64) + 2 * sizeof(int2));
}

// deep_mc_kernel's single-flip chains (a complex net, no translation sums) for 2 PAIRS walkers
// a block.  Layer 0's pre-activations are kept per walker and moved by the flipped spin's
// weights; an accepted move is committed when the next proposal is formed from them.  Walker
// k's random words, test and counters belong to one lane of the warp that forms its log psi.
// Bound by the FP32 pipe (six operations a complex multiply-add, in forward_once's order).
// Seven blocks an SM: 8192 walkers are 6.7 blocks of eight an SM, and with six resident the
// rest ran after the others (100-200-100-50 net, four sweeps: 67.5 ms with a thread per unit,
// 54.8 ms with six blocks, 35.8 ms; two units per thread 57, weights fetched ahead of their
// use into registers 40 to 43).
// With fewer blocks an SM, of wide layers or few walkers, a block has more threads (pair_threads);
// 128 whatever the layers left an SM with four warps and was slower than the thread per unit.  One
// sweep of thermalisation and one of sampling at N = 32, ms with a thread per unit / 128 threads / now:
// 2048 walkers of 256-256 6.9 / 9.2 / 5.8, 400-400 14.4 / 25.4 / 12.0, 700-700-700 79.6 / 226 / 66.3; 256
// walkers of them 4.8 / 7.4 / 2.7, 8.0 / 21.0 / 5.3, 31.3 / 105 / 24.8; 8192 walkers of 200-200 15.0 /
// 17.1 / 13.4, 200-100-50 15.1 / 9.6 / 9.6 (256 threads: 10.7).
constexpr int kPairsMcBlocks = 7;
template <int PAIRS, int T>
__global__ void __launch_bounds__(T, T == 128 ? kPairsMcBlocks : 1024 / T) deep_mc_pairs_kernel(DeepNetDev net, McLaunch L) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int WPC = 2 * PAIRS;
    const int size0 = net.size[0], N = net.N, nw = (N + 63) / 64;
    float4* zs = reinterpret_cast<float4*>(smem);                       // [PAIRS][size0]
    float4* const bufs[2] = {zs + PAIRS * size0, zs + PAIRS * (size0 + pair_buf(net, 0))};
    uint64_t* s = reinterpret_cast<uint64_t*>(bufs[1] + PAIRS * pair_buf(net, 1));   // [WPC][nw]
    int2* moved = reinterpret_cast<int2*>(s + WPC * nw);         // [WPC] accepted move: site, bits of ts (0: none)
    int2* trial = moved + WPC;                                          // [WPC] proposal
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int first = blockIdx.x * WPC;
    // lane r < 2 of warp q < PAIRS owns walker k = 2 q + r
    const int k_own = 2 * warp + lane;
    const bool own = warp < PAIRS && lane < 2, owner = own && first + k_own < L.B;
    const int mine = first + k_own;
    WalkerRng rng;
    rng.init(L.seed, L.walker_base + static_cast<uint32_t>(mine), owner ? L.rng_index[mine] : 0);
    unsigned long long acc = 0, props = 0;
    float lpr = 0.0f;
    int site = 0;
    if (own) {
        uint64_t* sk = s + k_own * nw;
        for (int k = 0; k < nw; k++) sk[k] = 0;
        if (owner) {
            if (L.init) {
                for (int k = 0; k < nw; k++) {
                    const uint64_t lo = rng.next();
                    const uint64_t hi = rng.next();
                    sk[k] = lo | (hi << 32);
                }
                if (N / 64 < nw) sk[N / 64] &= (1ull << (N % 64)) - 1ull;
            } else {
                for (int k = 0; k < nw; k++) sk[k] = L.spins[static_cast<long>(mine) * nw + k];
            }
        }
    }
    auto none = [](int, int, int, CPair, CPair) {};
    // Re log psi of this lane's walker (lanes 0 and 1 of the owning warps)
    auto log_psi = [&]() {
        float v0 = 0.0f, v1 = 0.0f;
        if (warp < PAIRS) {
            const CPair r = final_sum(net, bufs[(net.L - 1) & 1] + warp * net.size[net.L - 1], lane);
            up2(r.re, v0, v1);
        }
        return lane == 1 ? v1 : v0;
    };
    // the owner's next proposal
    auto propose = [&]() {
        if (!own) return;
        float ts = 0.0f;
        if (owner) {
            site = static_cast<int>(rng.next() % static_cast<uint32_t>(N));
            ts = bit_up(s + k_own * nw, site) ? -2.0f : 2.0f;
        }
        trial[k_own] = make_int2(site, __float_as_int(ts));
    };
    const int total = L.n_therm + L.n_samples * L.sweeps_per_sample;
    int sample = 0;
    for (int sw = 0; sw < total; sw++) {
        __syncthreads();
        // layer 0 and log psi of every state from its spins
        for (int item = t; item < PAIRS * size0; item += T) {
            const int p = item / size0, u = item - p * size0;
            const uint64_t *s0 = s + 2 * p * nw, *s1 = s0 + nw;
            CPair a{splat2(0.0f), splat2(0.0f)};
            const int conn = net.conn[0];
#pragma unroll 4
            for (int c = 0; c < conn; c++) {
                const float2 w = __ldg(net.w[0] + c * size0 + u);
                const int i = __ldg(net.cidx[0] + c * size0 + u);
                const pair_t sg = pk2(bit_up(s0, i) ? 1.0f : -1.0f, bit_up(s1, i) ? 1.0f : -1.0f);
                a.re = fma2(sg, splat2(w.x), a.re);   // sg = +-1: the products are exact
                a.im = fma2(sg, splat2(w.y), a.im);
            }
            const float2 b = net.b[0][u];
            const CPair z{add2(a.re, splat2(b.x)), add2(a.im, splat2(b.y))};
            st_pair(zs + item, z);
            st_pair(bufs[0] + item, act_pair(z));
        }
        forward_pairs<T, PAIRS>(net, bufs, none);
        lpr = log_psi();
        if (own) moved[k_own] = make_int2(0, 0);
        propose();
        __syncthreads();
        for (int p = 0; p < N; p++) {
            for (int item = t; item < PAIRS * size0; item += T) {
                const int q = item / size0, u = item - q * size0;
                float4 z = zs[item];
                float2 z0 = make_float2(z.x, z.z), z1 = make_float2(z.y, z.w);
                const int2 m0 = moved[2 * q], m1 = moved[2 * q + 1];
                if (m0.y | m1.y) {
                    if (m0.y) z0 = move_z0(net, m0.x, __int_as_float(m0.y), u, z0);
                    if (m1.y) z1 = move_z0(net, m1.x, __int_as_float(m1.y), u, z1);
                    zs[item] = make_float4(z0.x, z1.x, z0.y, z1.y);
                }
                const int2 p0 = trial[2 * q], p1 = trial[2 * q + 1];
                z0 = move_z0(net, p0.x, __int_as_float(p0.y), u, z0);
                z1 = move_z0(net, p1.x, __int_as_float(p1.y), u, z1);
                st_pair(bufs[0] + item, act_pair(CPair{pk2(z0.x, z1.x), pk2(z0.y, z1.y)}));
            }
            forward_pairs<T, PAIRS>(net, bufs, none);
            const float nl = log_psi();
            if (own) {
                bool accept = false;
                if (owner) {
                    const float delta = nl - lpr;
                    accept = delta > 0.0f;
                    if (!accept) accept = rng.uniform() <= expf_det(2.0f * delta);
                    if (accept) {
                        s[k_own * nw + (site >> 6)] ^= 1ull << (site & 63);
                        lpr = nl;
                        acc++;
                    }
                    props++;
                }
                moved[k_own] = accept ? trial[k_own] : make_int2(0, 0);
            }
            propose();
            __syncthreads();
        }
        if (owner) rng.index--;   // the word of the proposal that the sweep's end leaves undone
        const int done = sw + 1 - L.n_therm;
        if (done > 0 && done % L.sweeps_per_sample == 0) {
            const long row0 = static_cast<long>(L.sample_base + sample) * L.B;
            if (L.sample_spins)
                for (int i = t; i < WPC * nw; i += T) {
                    const int k = i / nw, word = i % nw;
                    if (first + k < L.B) L.sample_spins[(row0 + first + k) * nw + word] = s[k * nw + word];
                }
            sample++;
        }
    }
    __syncthreads();
    for (int i = t; i < WPC * nw; i += T) {
        const int k = i / nw, word = i % nw;
        if (first + k < L.B) L.spins[static_cast<long>(first + k) * nw + word] = s[k * nw + word];
    }
    if (owner) {
        L.rng_index[mine] = rng.index;
        L.accepts[mine] += acc;
        L.proposals[mine] += props;
    }
}

// ---------------------------------------------------------------- adjoint of E_loc
// Extension (no reference counterpart): reverse-mode derivative of the local energy,
//   d E_loc(s) / d theta = sum_n e_n O(s'_n) - E_loc(s) O(s),  e_n = c_n psi(s'_n) / psi(s),
// with O = d log psi / d theta (holomorphic, final weights d log psi / d fw_j = act_j).
// Per configuration x the reverse pass yields the error vector delta_l(x) = d log psi /
// d z_l of every layer; the parameter gradient is then the weighted sum over
// configurations of the outer products delta_l(x) (x) a_{l-1}(x), formed as batched
// reductions over all configurations of a chunk.  Every forward pass is recomputed
// from the spins (no angles are kept per walker between calls).

// delta_l for every layer after forward_once<STORE>; emit(layer, unit, delta)
template <typename V, bool REAL, typename Emit>
__device__ void backward_deltas(const DeepNetDev& net, Work<V>& w, Emit emit) {
    const int t = threadIdx.x;
    const int L = net.L;
    V* cur = w.in;
    V* nxt = w.out;
    for (int l = L - 1; l >= 0; l--) {
        const int size = net.size[l];
        V d = czero<V>();
        if (t < size) {
            const V ang = w.angles[net.begin_angle[l] + t];
            if (l == L - 1) {
                d = cmul(W_of<V>::fw(net)[t], dact<REAL>(ang));
            } else {
                const int nsize = net.size[l + 1];
                V acc = czero<V>();
                const V* wn = W_of<V>::w(net, l + 1);
                for (int e = net.rptr[l][t]; e < net.rptr[l][t + 1]; e++) {
                    const int q = net.rq[l][e];
                    acc = cadd(acc, cmul(wn[q], nxt[q % nsize]));
                }
                d = cmul(acc, dact<REAL>(ang));
            }
        }
        __syncthreads();
        if (t < size) {
            cur[t] = d;
            emit(l, t, d);
        }
        __syncthreads();
        V* tmp = cur;
        cur = nxt;
        nxt = tmp;
    }
}

// a neighbour's term of the local energy, cf psi(s') / psi(s), in FP64.  One function for the
// kernels below, so that they round alike.
__device__ __noinline__ double2 neighbour_term(double2 cf, float2 lq, float2 lp) {
    const double dr = static_cast<double>(lq.x) - lp.x, di = static_cast<double>(lq.y) - lp.y;
    const double m = exp(dr);
    return make_double2(m * (cf.x * cos(di) - cf.y * sin(di)), m * (cf.x * sin(di) + cf.y * cos(di)));
}

// One CTA per sample: E_loc(s) (FP32 passes, FP64 sum), then for every configuration x
// of the sample (x = s first, then s'_n for the off-diagonal strings in order) its spins,
// activations and alpha_x * delta_l(x), with alpha_{s'_n} = w_s e_n and
// alpha_s = w_s (-sum_{off-diagonal n} e_n + score * 2 Re E_loc(s)) (diagonal strings leave
// the configuration unchanged and drop out of the derivative).  With score, also
// w_s delta_l(s) and w_s (dltsO, alphaO) for the -2 <Re E> <O*> part of the sampling term.
__global__ void deep_adjoint_kernel(DeepNetDev net, OpDev op, int count, const uint64_t* spins, uint64_t enum_base,
                                    int enumerate, const double* weights, int score, double2* eloc, float2* acts,
                                    float2* dlts, float2* alpha, uint64_t* xspins, int xs, float2* dltsO,
                                    float2* alphaO) {
    extern __shared__ __align__(16) unsigned char smem[];
    Work<float2> w = carve<float2>(smem, net, true);
    uint64_t* sp = w.s + kMaxWords;
    // layer 0's pre-activations of the sample and of a neighbour
    float2* z0s = reinterpret_cast<float2*>(w.s + 4 * kMaxWords);
    float2* z0n = z0s + net.size[0];
    const long t = blockIdx.x;
    if (t >= count) return;
    const int nw = (net.N + 63) / 64;
    const int size0 = net.size[0];
    load_config(spins, enum_base, enumerate, t, net.N, w.s);
    __syncthreads();
    layer0_pre(net, w.s, z0s);
    __syncthreads();
    const float2 lp = forward_from_z0(net, z0s, w);
    double er = 0.0, ei = 0.0, eor = 0.0, eoi = 0.0;
    for (int n = 0; n < op.S; n++) {
        if (op.nflip[n] != 0) continue;
        const double2 cf = apply_string(op, n, w.s, sp);
        er += cf.x;
        ei += cf.y;
    }
    const double ws = weights ? weights[t] : 1.0;
    const float wsf = static_cast<float>(ws);
    // the stored forward pass and the reverse pass of configuration xi with coefficient af
    auto pass = [&](const uint64_t* x, long xi, float2 af, bool self) {
        for (int k = threadIdx.x; k < net.units; k += blockDim.x) acts[xi * net.units + k] = w.acts[k];
        if (threadIdx.x < nw) xspins[xi * nw + threadIdx.x] = x[threadIdx.x];
        if (threadIdx.x == 0) alpha[xi] = af;
        backward_deltas<float2, false>(net, w, [&](int l, int j, float2 d) {
            dlts[xi * net.units + net.begin_angle[l] + j] = cmul(af, d);
            if (self) dltsO[t * net.units + net.begin_angle[l] + j] = make_float2(wsf * d.x, wsf * d.y);
        });
    };
    // each off-diagonal string's neighbour: one stored forward pass gives its term of the
    // local energy and feeds its reverse pass (coefficient w_s e_n)
    int q = 0;
    for (int n = 0; n < op.S; n++) {
        if (op.nflip[n] == 0) continue;
        q++;
        const double2 cf = apply_string(op, n, w.s, sp);
        // the neighbour's layer 0: the sample's moved by the flipped spins' connections
        for (int u = threadIdx.x; u < size0; u += blockDim.x) z0n[u] = z0s[u];
        __syncthreads();
        for (int f = 0; f < op.nflip[n]; f++) {
            const int site = op.flip_sites[op.flip_off[n] + f];
            const float two_s = bit_up(w.s, site) ? -2.0f : 2.0f;
            for (int k = net.sptr[site] + threadIdx.x; k < net.sptr[site + 1]; k += blockDim.x) {
                const int e = net.sq[k];
                const float2 wv = net.w[0][e];
                float2* z = z0n + e % size0;
                atomicAdd(&z->x, two_s * wv.x);
                atomicAdd(&z->y, two_s * wv.y);
            }
            // one site at a time: each unit meets a site once, so the sums do not
            // depend on the order of the atomic additions
            __syncthreads();
        }
        const float2 lq = forward_from_z0<true>(net, z0n, w);
        const double2 e = neighbour_term(cf, lq, lp);
        eor += e.x;
        eoi += e.y;
        pass(sp, t * xs + q, make_float2(static_cast<float>(ws * e.x), static_cast<float>(ws * e.y)), false);
    }
    er += eor;
    ei += eoi;
    // the configuration itself last: its coefficient -sum_n e_n (+ 2 E_loc with the
    // sampling term) needs every neighbour's term
    {
        double2 a = make_double2(-eor, -eoi);
        if (score) a.x += 2.0 * er;
        forward_from_z0<true>(net, z0s, w);
        pass(w.s, t * xs, make_float2(static_cast<float>(ws * a.x), static_cast<float>(ws * a.y)), score != 0);
        if (score && threadIdx.x == 0) alphaO[t] = make_float2(wsf, 0.f);
    }
    if (threadIdx.x == 0) eloc[t] = make_double2(er, ei);
}

size_t deep_adjoint_pairs_smem(const DeepNetDev& n, int pairs) {
    return sizeof(float4) * pairs * (n.units + pair_buf(n, 0) + pair_buf(n, 1)) +
           sizeof(float2) * (n.size[0] + 4 * pairs) + sizeof(uint64_t) * kMaxWords + 16;
}

// deep_adjoint_kernel with 2 PAIRS of a sample's off-diagonal neighbours at a time, two in the
// halves of each packed operation.  Every configuration's arithmetic and the local energy's
// order of summation are deep_adjoint_kernel's: the outputs are identical.  The neighbours'
// FP64 exponentials run in the lanes of one warp, once each: in every thread of the block they
// held the FP64 pipe for 28000 cycles a neighbour on the 100-200-100-50 net, which was the
// kernel's whole time.  Bound by the FP32 pipe and, at 128 threads, by the layers' barriers.
// 8192 samples of that net: 70.3 -> 19.4 ms.
// More threads a block for wide layers or few samples, as the sampler (pair_threads): 2048 samples at
// N = 32, ms with a thread per unit / 128 threads / now: 200-200 9.1 / 4.6 / 3.9, 400-400 36 / 22 / 12.2,
// 700-700-700 314 / 217 / 73; 256 samples of 400-400-400 12.1 / 13.0 / 6.3.
constexpr int kPairsAdjBlocks = 5;
template <int PAIRS, int T>
__global__ void __launch_bounds__(T, T == 128 ? kPairsAdjBlocks : 1024 / T) deep_adjoint_pairs_kernel(
    DeepNetDev net, OpDev op, int count, const uint64_t* spins, uint64_t enum_base, int enumerate,
    const double* weights, int score, double2* eloc, float2* acts, float2* dlts, float2* alpha, uint64_t* xspins,
    int xs, float2* dltsO, float2* alphaO) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NB = 2 * PAIRS;
    const int size0 = net.size[0], units = net.units;
    float4* angles = reinterpret_cast<float4*>(smem);                   // [PAIRS][units]
    float4* const bufs[2] = {angles + PAIRS * units, angles + PAIRS * (units + pair_buf(net, 0))};
    float2* z0s = reinterpret_cast<float2*>(bufs[1] + PAIRS * pair_buf(net, 1));   // [size0] the sample's layer 0
    float2* lqs = z0s + size0;                                          // [NB] log psi
    float2* afs = lqs + NB;                                             // [NB] coefficients of the deltas
    // 16-byte aligned whatever size0
    uint64_t* s = reinterpret_cast<uint64_t*>((reinterpret_cast<size_t>(afs + NB) + 15) & ~size_t(15));
    const long t = blockIdx.x;
    if (t >= count) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nw = (net.N + 63) / 64;
    load_config(spins, enum_base, enumerate, t, net.N, s);
    for (int u = tid; u < size0; u += T) {
        float2 a = make_float2(0.0f, 0.0f);
        for (int c = 0; c < net.conn[0]; c++) {
            const float2 w = __ldg(net.w[0] + c * size0 + u);
            const float sg = bit_up(s, __ldg(net.cidx[0] + c * size0 + u)) ? 1.0f : -1.0f;
            a.x = __fmaf_rn(sg, w.x, a.x);
            a.y = __fmaf_rn(sg, w.y, a.y);
        }
        const float2 b = net.b[0][u];
        z0s[u] = make_float2(a.x + b.x, a.y + b.y);
    }
    __syncthreads();
    const double ws = weights ? weights[t] : 1.0;
    // log psi of the pairs in the last buffer to lqs
    auto log_psi = [&](int pairs) {
        if (warp < pairs) {
            const CPair r = final_sum(net, bufs[(net.L - 1) & 1] + warp * net.size[net.L - 1], lane);
            float x0, x1, y0, y1;
            up2(r.re, x0, x1);
            up2(r.im, y0, y1);
            if (lane == 0) {
                lqs[2 * warp] = make_float2(x0, y0);
                lqs[2 * warp + 1] = make_float2(x1, y1);
            }
        }
        __syncthreads();
    };
    // stored forward pass of configurations x0 .. x0 + nb - 1, layer 0 from z0of(pair, u)
    auto forward = [&](auto pairs_c, auto z0of, long x0, int nb) {
        constexpr int P = decltype(pairs_c)::value;
        auto keep = [&](int l, int p, int u, CPair z, CPair y) {
            const int at = net.begin_angle[l] + u;
            st_pair(angles + p * units + at, z);
            float a0, a1, b0, b1;
            up2(y.re, a0, a1);
            up2(y.im, b0, b1);
            float2* row = acts + (x0 + 2 * p) * units + at;
            if (2 * p < nb) row[0] = make_float2(a0, b0);
            if (2 * p + 1 < nb) row[units] = make_float2(a1, b1);
        };
        for (int item = tid; item < P * size0; item += T) {
            const int p = item / size0, u = item - p * size0;
            const CPair z = z0of(p, u);
            const CPair y = act_pair(z);
            st_pair(bufs[0] + item, y);
            keep(0, p, u, z, y);
        }
        forward_pairs<T, P>(net, bufs, keep);
    };
    // reverse pass: alpha_x delta_l(x) of configurations x0 .. x0 + nb - 1; with self also
    // w_s delta_l of the sample
    auto backward = [&](auto pairs_c, long x0, int nb, bool self) {
        constexpr int P = decltype(pairs_c)::value;
        const float wsf = static_cast<float>(ws);
        for (int l = net.L - 1; l >= 0; l--) {
            const int size = net.size[l];
            float4* cur = bufs[l & 1];
            auto done = [&](int p, int u, CPair a) {
                const int at = net.begin_angle[l] + u;
                const CPair d = cmul(a, dact_pair(ld_pair(angles + p * units + at)));
                st_pair(cur + p * size + u, d);
                float d0x, d1x, d0y, d1y;
                up2(d.re, d0x, d1x);
                up2(d.im, d0y, d1y);
                float2* row = dlts + (x0 + 2 * p) * units + at;
                if (2 * p < nb) row[0] = cmul(afs[2 * p], make_float2(d0x, d0y));
                if (2 * p + 1 < nb) row[units] = cmul(afs[2 * p + 1], make_float2(d1x, d1y));
                if (self && p == 0) dltsO[t * units + at] = make_float2(wsf * d0x, wsf * d0y);
            };
            if (l == net.L - 1) {
                for (int item = tid; item < P * size; item += T) {
                    const int p = item / size, u = item - p * size;
                    const float2 f = net.fw[u];
                    done(p, u, CPair{splat2(f.x), splat2(f.y)});
                }
            } else {
                const int above = net.size[l + 1];
                const float4* nxt = bufs[(l + 1) & 1];
                if (net.wt[l + 1]) {
                    layer_sums_split<T, P, true>(size, above, net.wt[l + 1], nullptr, nxt, above, done);
                } else {
                    const float2* wn = net.w[l + 1];
                    for (int item = tid; item < P * size; item += T) {
                        const int p = item / size, u = item - p * size;
                        CPair a{splat2(0.0f), splat2(0.0f)};
                        for (int e = net.rptr[l][u]; e < net.rptr[l][u + 1]; e++) {
                            const int q = net.rq[l][e];
                            cmac(a, wn[q], ld_pair(nxt + p * above + q % above));
                        }
                        done(p, u, a);
                    }
                }
            }
            __syncthreads();
        }
    };
    auto self_z = [&](int, int u) {
        const float2 z = z0s[u];
        return CPair{splat2(z.x), splat2(z.y)};
    };
    const std::integral_constant<int, 1> one;
    const std::integral_constant<int, PAIRS> all;
    forward(one, self_z, t * xs, 1);   // the sample's rows are written again with its reverse pass
    log_psi(1);
    const float2 lp = lqs[0];
    // warp 0: the diagonal strings' sum, in order
    double er = 0.0, ei = 0.0, eor = 0.0, eoi = 0.0;
    auto factor = [&](int n) {
        int parity = 0;
        for (int k = 0; k < kMaxWords; k++) parity += __popcll(op.zmask[n * kMaxWords + k] & ~s[k]);
        const double sg = (parity & 1) ? -1.0 : 1.0;
        const double2 c = op.coef[n];
        const int yp = op.ypow[n] & 3;
        const double2 r = yp == 0 ? c : (yp == 1 ? make_double2(c.y, -c.x)
                                                 : (yp == 2 ? make_double2(-c.x, -c.y) : make_double2(-c.y, c.x)));
        return make_double2(sg * r.x, sg * r.y);
    };
    if (warp == 0) {
        for (int n0 = 0; n0 < op.S; n0 += 32) {
            const bool diag = n0 + lane < op.S && op.nflip[n0 + lane] == 0;
            const double2 cf = diag ? factor(n0 + lane) : make_double2(0.0, 0.0);
            for (unsigned m = __ballot_sync(0xffffffffu, diag); m; m &= m - 1) {
                er += __shfl_sync(0xffffffffu, cf.x, __ffs(m) - 1);
                ei += __shfl_sync(0xffffffffu, cf.y, __ffs(m) - 1);
            }
        }
    }
    for (int q = 0; q < op.num_offdiag; q += NB) {
        const int nb = min(NB, op.num_offdiag - q);
        const long x0 = t * xs + q + 1;
        // a neighbour's layer 0: the sample's moved by the flipped spins, one after the other
        forward(all, [&](int p, int u) {
            float2 z[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                z[h] = z0s[u];
                if (2 * p + h >= nb) continue;
                const int n = op.offdiag[q + 2 * p + h], off = op.flip_off[n];
                for (int f = 0; f < op.nflip[n]; f++) {
                    const int site = op.flip_sites[off + f];
                    z[h] = move_z0(net, site, bit_up(s, site) ? -2.0f : 2.0f, u, z[h]);
                }
            }
            return CPair{pk2(z[0].x, z[1].x), pk2(z[0].y, z[1].y)};
        }, x0, nb);
        log_psi(PAIRS);
        if (warp == 0) {
            double2 e = make_double2(0.0, 0.0);
            if (lane < nb) {
                e = neighbour_term(factor(op.offdiag[q + lane]), lqs[lane], lp);
                const float2 af = make_float2(static_cast<float>(ws * e.x), static_cast<float>(ws * e.y));
                afs[lane] = af;
                alpha[x0 + lane] = af;
            }
            for (int k = 0; k < nb; k++) {
                eor += __shfl_sync(0xffffffffu, e.x, k);
                eoi += __shfl_sync(0xffffffffu, e.y, k);
            }
        }
        for (int i = tid; i < nb * nw; i += T) {
            const int k = i / nw, word = i - k * nw, n = op.offdiag[q + k];
            uint64_t v = s[word];
            for (int f = 0; f < op.nflip[n]; f++) {
                const int site = op.flip_sites[op.flip_off[n] + f];
                if ((site >> 6) == word) v ^= 1ull << (site & 63);
            }
            xspins[(x0 + k) * nw + word] = v;
        }
        __syncthreads();
        backward(all, x0, nb, false);
    }
    // the configuration itself last: its coefficient -sum_n e_n (+ 2 E_loc with the
    // sampling term) needs every neighbour's term
    const long xi = t * xs;
    if (tid == 0) {
        er += eor;
        ei += eoi;
        double2 a = make_double2(-eor, -eoi);
        if (score) a.x += 2.0 * er;
        afs[0] = make_float2(static_cast<float>(ws * a.x), static_cast<float>(ws * a.y));
        alpha[xi] = afs[0];
        if (score) alphaO[t] = make_float2(static_cast<float>(ws), 0.f);
        eloc[t] = make_double2(er, ei);
    }
    if (tid < nw) xspins[xi * nw + tid] = s[tid];
    forward(one, self_z, xi, 1);
    backward(one, xi, 1, score != 0);
}

// The configurations of a launch lie in parts of `rows` (the last one shorter); a part is cut
// into at most kAdjSplits splits of equal length, each an FP32 sum in order.  The sums cancel
// to a small part of their terms (a configuration's against its neighbours'), so the result
// depends on this order in its leading digits: it does not change with the launch.
constexpr int kAdjSplits = 64;
struct AdjSplit {
    int k0, k1;   // configurations of split z
};
__host__ __device__ inline int adj_splits_of(int K) { return K < 512 ? 1 : (K / 256 < kAdjSplits ? K / 256 : kAdjSplits); }
__host__ __device__ inline int adj_grid_splits(int K, int rows) {
    return K <= rows ? adj_splits_of(K) : (K + rows - 1) / rows * kAdjSplits;
}
__device__ __forceinline__ AdjSplit adj_split(int K, int rows, int z) {
    const int part = z / kAdjSplits, q = z - part * kAdjSplits;
    const int n = min(rows, K - part * rows), splits = adj_splits_of(n), per = (n + splits - 1) / splits;
    const int k0 = part * rows + min(n, q * per);
    return AdjSplit{k0, part * rows + min(n, q * per + per)};
}

// partial[z][m][n] = sum over the configurations x of split z of D[x][m] A(x, n), where
// D[x][m] = D[x * ldd + m] and A(x, n) = A[x * lda + n], or with SPINS +-1 for spin n of the spin
// row xsp + x * xld; A(x, Nn) = 1, so that column Nn holds the bias sums.  A thread holds 4 x 4
// (SPINS: 4 x 8) products, so that 16-byte shared loads keep up with the FP32 pipe (2 x 2 with
// 8-byte loads, and the biases as a product of their own, took 22.5 ms for 8192 samples of the
// 100-200-100-50 net); stages of 16 configurations arrive by asynchronous copies while the
// one before is used.  Bound by the FP32 pipe, six operations a product: 11.3 ms.
constexpr int kAdjStage = 16, kAdjTm = 32;

template <bool SPINS>
__global__ void __launch_bounds__(128) adj_cgemm_kernel(int K, int rows, int M, int Nn, const float2* __restrict__ D,
                                                        int ldd, const float2* __restrict__ A, int lda,
                                                        const uint64_t* __restrict__ xsp, int xld,
                                                        float2* __restrict__ partial) {
    constexpr int JN = SPINS ? 8 : 4, TN = 16 * JN;
    using Elem = std::conditional_t<SPINS, float, float2>;
    __shared__ __align__(16) float2 sD[2][kAdjStage][kAdjTm];
    __shared__ __align__(16) Elem sA[2][kAdjStage][TN];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.x * kAdjTm, n0 = blockIdx.y * TN;
    const AdjSplit sp = adj_split(K, rows, blockIdx.z);
    float2 acc[4][JN];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < JN; j++) acc[i][j] = make_float2(0.f, 0.f);
    // 8-byte asynchronous copies (rows are 8-byte aligned); outside the matrix zeros are written
    auto copy = [](float2* dst, const float2* src, bool live) {
        const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(live ? 8 : 0) : "memory");
    };
    auto stage = [&](int s, int kb) {
        for (int e = tid; e < kAdjStage * kAdjTm; e += 128) {
            const int kk = e / kAdjTm, c = e % kAdjTm, x = kb + kk;
            const bool live = x < sp.k1 && m0 + c < M;
            copy(&sD[s][kk][c], live ? D + static_cast<long>(x) * ldd + m0 + c : D, live);
        }
        for (int e = tid; e < kAdjStage * TN; e += 128) {
            const int kk = e / TN, c = e % TN, x = kb + kk, n = n0 + c;
            const bool row = x < sp.k1;
            if constexpr (SPINS) {
                float v = 0.0f;
                if (row && n < Nn) v = ((xsp[static_cast<long>(x) * xld + (n >> 6)] >> (n & 63)) & 1ull) ? 1.0f : -1.0f;
                else if (row && n == Nn) v = 1.0f;
                sA[s][kk][c] = v;
            } else {
                const bool live = row && n < Nn;
                if (n == Nn) sA[s][kk][c] = make_float2(1.0f, 0.0f);   // past the split D is zero
                else copy(&sA[s][kk][c], live ? A + static_cast<long>(x) * lda + n : A, live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, sp.k0);
    for (int kb = sp.k0, s = 0; kb < sp.k1; kb += kAdjStage, s ^= 1) {
        if (kb + kAdjStage < sp.k1) {
            stage(s ^ 1, kb + kAdjStage);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < kAdjStage; kk++) {
            float2 d[4];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float4 v = *reinterpret_cast<const float4*>(&sD[s][kk][4 * ty + 2 * i]);
                d[2 * i] = make_float2(v.x, v.y);
                d[2 * i + 1] = make_float2(v.z, v.w);
            }
            if constexpr (SPINS) {
                // columns 4 tx .. 4 tx + 3 and these + 64
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float4 g4 = *reinterpret_cast<const float4*>(&sA[s][kk][4 * tx + 64 * h]);
                    const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) {   // g = +-1: cmul's products are exact
                            acc[i][4 * h + j].x = fmaf(g[j], d[i].x, acc[i][4 * h + j].x);
                            acc[i][4 * h + j].y = fmaf(g[j], d[i].y, acc[i][4 * h + j].y);
                        }
                }
            } else {
                // columns 2 tx, 2 tx + 1 and these + 32: neighbouring lanes read neighbouring 16 bytes
                float2 a[4];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float4 v = *reinterpret_cast<const float4*>(&sA[s][kk][2 * tx + 32 * h]);
                    a[2 * h] = make_float2(v.x, v.y);
                    a[2 * h + 1] = make_float2(v.z, v.w);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = cadd(acc[i][j], cmul(d[i], a[j]));
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < JN; j++) {
            const int m = m0 + 4 * ty + i, n = n0 + (SPINS ? 4 * tx + 64 * (j >> 2) + (j & 3) : 2 * tx + 32 * (j >> 1) + (j & 1));
            if (m < M && n <= Nn) partial[(static_cast<long>(blockIdx.z) * M + m) * (Nn + 1) + n] = acc[i][j];
        }
}

// the final weights' sums: partial[z][j] = sum over split z of alpha[x] A[x * lda + j], in order
// by one warp from rows that the block stages (the serial sum read from memory took 800 us for
// 8192 samples of the 100-200-100-50 net)
__global__ void __launch_bounds__(256) adj_final_kernel(int K, int rows, int last, const float2* __restrict__ alpha,
                                                        const float2* __restrict__ A, int lda,
                                                        float2* __restrict__ partial) {
    constexpr int kRows = 64;
    __shared__ float2 tile[2][kRows][32];
    __shared__ float2 al[2][kRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = blockIdx.x * 32 + lane;
    const AdjSplit sp = adj_split(K, rows, blockIdx.y);
    float2 a = make_float2(0.f, 0.f);
    float2 v[kRows / 8], w = make_float2(0.f, 0.f);
    auto load = [&](int x0) {
#pragma unroll
        for (int q = 0; q < kRows / 8; q++) {
            const int x = x0 + warp + 8 * q;
            v[q] = x < sp.k1 && j < last ? A[static_cast<long>(x) * lda + j] : make_float2(0.f, 0.f);
        }
        if (threadIdx.x < kRows && x0 + static_cast<int>(threadIdx.x) < sp.k1) w = alpha[x0 + threadIdx.x];
    };
    load(sp.k0);
    for (int x0 = sp.k0, s = 0; x0 < sp.k1; x0 += kRows, s ^= 1) {
#pragma unroll
        for (int q = 0; q < kRows / 8; q++) tile[s][warp + 8 * q][lane] = v[q];
        if (threadIdx.x < kRows) al[s][threadIdx.x] = w;
        __syncthreads();
        if (x0 + kRows < sp.k1) load(x0 + kRows);
        if (warp == 0)
            for (int q = 0; q < min(kRows, sp.k1 - x0); q++) a = cadd(a, cmul(al[s][q], tile[s][q][lane]));
    }
    if (warp == 0 && j < last) partial[static_cast<long>(blockIdx.y) * last + j] = a;
}

// G[m][n] (n < Nn) and Gb[m] (column Nn) += sum over splits of partial[z][m][n], in FP64: eight
// slices of the splits, then the slices in order.  `cols` = Nn + 1, or Nn with no bias column.
__global__ void __launch_bounds__(256) adj_split_sum_kernel(int M, int Nn, int cols, int splits,
                                                            const float2* __restrict__ partial, double2* G,
                                                            double2* Gb) {
    __shared__ double2 red[8][32];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const long total = static_cast<long>(M) * cols, e = blockIdx.x * 32L + lane;
    double2 a = make_double2(0.0, 0.0);
    if (e < total) {
        const int per = (splits + 7) / 8, z1 = min(splits, (slice + 1) * per);
#pragma unroll 8
        for (int z = slice * per; z < z1; z++) {
            const float2 v = partial[z * total + e];
            a.x += v.x;
            a.y += v.y;
        }
    }
    red[slice][lane] = a;
    __syncthreads();
    if (slice != 0 || e >= total) return;
    for (int q = 1; q < 8; q++) a = cadd(a, red[q][lane]);
    const int m = static_cast<int>(e / cols), n = static_cast<int>(e - static_cast<long>(m) * cols);
    double2* out = n < Nn ? G + static_cast<long>(m) * Nn + n : Gb + m;
    *out = cadd(*out, a);
}

int threads_for(const DeepNetDev& n) {
    const int width = std::max(n.width, n.N);
    return std::min(1024, std::max(32, (width + 31) / 32 * 32));
}

size_t smem_for(const DeepNetDev& n, size_t vbytes, bool store) {
    return vbytes * (32 + 2 * n.width + (store ? 2 * n.units : 0)) + sizeof(uint64_t) * 4 * kMaxWords;
}

template <typename K>
cudaError_t set_smem(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

// units of the widest layer
int widest(const DeepNetDev& n) {
    int w = 0;
    for (int l = 0; l < n.L; l++) w = std::max(w, n.size[l]);
    return w;
}

// Threads a block of the pairs kernels, of r blocks an SM (as many as shared memory holds, or the
// launch has): 128 where `many` of them fill the SM, otherwise enough that about 1024 threads are
// resident, but not so many that most have no unit in any layer (512 walkers, N = 20, 128 / 256 /
// 512 / 1024 threads: 40-20-10 650 / 574 / 594 / 634 us, 20-10 392 / 399 / 403 / 450); 256 threads only
// where they take a layer's units in one round (4096 walkers of 320-320-320 43 ms, with 512 29).
int pair_threads(size_t smem, int units, int blocks, int sms, int many) {
    const int r = std::min(static_cast<int>((size_t(228) << 10) / (smem + 1024)), (blocks + sms - 1) / sms);
    int threads = r >= many ? 128 : (r >= 3 && units <= 256 ? 256 : (r >= 2 ? 512 : 1024));
    while (threads > 128 && threads > 8 * units) threads /= 2;
    return threads;
}

// f(PAIRS, T) of the pairs kernels; one and two pairs take 512 threads where four take 256 or 1024
template <typename F>
cudaError_t pairs_launch(int pairs, int threads, F f) {
    if (pairs == 4) {
        const std::integral_constant<int, 4> four;
        if (threads == 128) return f(four, std::integral_constant<int, 128>());
        if (threads == 256) return f(four, std::integral_constant<int, 256>());
        if (threads == 512) return f(four, std::integral_constant<int, 512>());
        return f(four, std::integral_constant<int, 1024>());
    }
    auto few = [&](auto p) {
        if (threads == 128) return f(p, std::integral_constant<int, 128>());
        return f(p, std::integral_constant<int, 512>());
    };
    return pairs == 2 ? few(std::integral_constant<int, 2>()) : few(std::integral_constant<int, 1>());
}

}  // namespace

// ---------------------------------------------------------------- host side
struct DeepHost {
    std::vector<std::unique_ptr<DevBuf>> bufs;
    DeepNetDev net[2];
};

template <typename T>
static cudaError_t upload(DeepHost* h, const std::vector<T>& v, const T** out) {
    auto b = std::make_unique<DevBuf>();
    cudaError_t e = b->ensure(std::max<size_t>(16, sizeof(T) * v.size()));
    if (e != cudaSuccess) return e;
    if (!v.empty()) e = cudaMemcpy(b->p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    *out = static_cast<const T*>(b->p);
    h->bufs.push_back(std::move(b));
    return e;
}

// dst[at[e]] = src[e], in both precisions
__global__ void scatter_entries_kernel(int n, const float2* src, const double2* src64, const int* at, float2* dst,
                                       double2* dst64) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        dst[at[e]] = src[e];
        dst64[at[e]] = src64[e];
    }
}

// dst[c][r] = src[r][c]
__global__ void transpose_kernel(int rows, int cols, const float2* src, float2* dst) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < rows * cols; e += gridDim.x * blockDim.x)
        dst[(e % cols) * rows + e / cols] = src[e];
}

// the layouts formed from the device weights, after an upload or an optimiser step
int deep_derive(const rbmg_psi* psi) {
    if (psi->kind == 2) return RBMG_OK;
    const DeepNetDev& d = psi->deep_dev[0];
    const int n0 = d.conn[0] * d.size[0];
    scatter_entries_kernel<<<(n0 + 255) / 256, 256, 0, stream()>>>(n0, d.w[0], d.w64[0], d.w0at, const_cast<float2*>(d.w0),
                                                                       const_cast<double2*>(d.w064));
    RBMG_CK(cudaGetLastError());
    for (int l = 1; l < d.L; l++) {
        if (!d.wt[l]) continue;
        const int n = d.size[l] * d.size[l - 1];
        transpose_kernel<<<(n + 255) / 256, 256, 0, stream()>>>(d.size[l - 1], d.size[l], d.w[l],
                                                                const_cast<float2*>(d.wt[l]));
        RBMG_CK(cudaGetLastError());
    }
    return RBMG_OK;
}

// Device copy of the net(s): part 0 = complex net (PsiDeep) or real part (PsiPair), 1 = imaginary part.
int deep_upload(rbmg_psi* psi) {
    auto h = std::make_unique<DeepHost>();
    const int nets = psi->kind == 2 ? 2 : 1;
    const int L = static_cast<int>(psi->layers.size());
    for (int part = 0; part < nets; part++) {
        DeepNetDev& d = h->net[part];
        d = DeepNetDev{};
        d.N = psi->N;
        d.L = L;
        d.real_net = psi->kind == 2;
        d.ti = psi->translational_invariance;
        d.P = psi->num_params();
        d.width = psi->width;
        int k = 2 * psi->N, a = 0;
        for (int l = 0; l < L; l++) {
            const auto& Ly = psi->layers[l];
            d.size[l] = Ly.size;
            d.conn[l] = Ly.conn;
            d.begin_params[l] = k - 2 * psi->N;
            d.begin_angle[l] = a;
            k += Ly.size + Ly.conn * Ly.size;
            a += Ly.size;
            auto pick = [&](const cplx& z) -> cplx {
                if (psi->kind != 2) return z;
                return part == 0 ? cplx(z.real(), 0.0) : cplx(z.imag(), 0.0);
            };
            std::vector<float2> w32(Ly.weights.size()), b32(Ly.biases.size());
            std::vector<double2> w64(Ly.weights.size()), b64(Ly.biases.size());
            for (size_t q = 0; q < Ly.weights.size(); q++) {
                const cplx z = pick(Ly.weights[q]);
                w32[q] = make_float2(float(z.real()), float(z.imag()));
                w64[q] = make_double2(z.real(), z.imag());
            }
            for (size_t q = 0; q < Ly.biases.size(); q++) {
                const cplx z = pick(Ly.biases[q]);
                b32[q] = make_float2(float(z.real()), float(z.imag()));
                b64[q] = make_double2(z.real(), z.imag());
            }
            std::vector<int> ci(Ly.connections.begin(), Ly.connections.end());
            RBMG_CK(upload(h.get(), w32, &d.w[l]));
            RBMG_CK(upload(h.get(), b32, &d.b[l]));
            RBMG_CK(upload(h.get(), w64, &d.w64[l]));
            RBMG_CK(upload(h.get(), b64, &d.b64[l]));
            RBMG_CK(upload(h.get(), ci, &d.cidx[l]));
        }
        d.units = a;
        // rhs lists of layer l from the lhs connections of layer l+1, in the order of
        // source/quantum_state/PsiDeep.cu:101-111 (next unit j ascending, connection c inner)
        for (int l = 0; l + 1 < L; l++) {
            const auto& Nx = psi->layers[l + 1];
            const int size = psi->layers[l].size;
            std::vector<std::vector<int>> lists(size);
            for (int j = 0; j < Nx.size; j++)
                for (int c = 0; c < Nx.conn; c++) lists[Nx.connections[c * Nx.size + j]].push_back(c * Nx.size + j);
            std::vector<int> ptr(size + 1, 0), q;
            for (int i = 0; i < size; i++) {
                ptr[i] = static_cast<int>(q.size());
                q.insert(q.end(), lists[i].begin(), lists[i].end());
            }
            ptr[size] = static_cast<int>(q.size());
            RBMG_CK(upload(h.get(), ptr, &d.rptr[l]));
            RBMG_CK(upload(h.get(), q, &d.rq[l]));
        }
        {
            const auto& L0 = psi->layers[0];
            std::vector<std::vector<int>> lists(psi->N);
            for (int c = 0; c < L0.conn; c++)
                for (int j = 0; j < L0.size; j++) {
                    const int i = static_cast<int>(L0.connections[static_cast<size_t>(c) * L0.size + j]);
                    if (i < psi->N) lists[i].push_back(c * L0.size + j);
                }
            std::vector<int> ptr(psi->N + 1, 0), q;
            for (int i = 0; i < psi->N; i++) {
                ptr[i] = static_cast<int>(q.size());
                q.insert(q.end(), lists[i].begin(), lists[i].end());
            }
            ptr[psi->N] = static_cast<int>(q.size());
            if (q.empty()) q.push_back(0);
            RBMG_CK(upload(h.get(), ptr, &d.sptr));
            RBMG_CK(upload(h.get(), q, &d.sq));
        }
        if (psi->kind != 2) {
            // layer 0 by spin: a unit's further connections to a spin go to further planes
            const auto& L0 = psi->layers[0];
            std::vector<int> at(L0.connections.size());
            std::vector<int> seen(static_cast<size_t>(psi->N) * L0.size, 0);
            d.w0n = 1;
            for (size_t e = 0; e < at.size(); e++) {
                const size_t cell = static_cast<size_t>(L0.connections[e]) * L0.size + e % L0.size;
                const int plane = seen[cell]++;
                d.w0n = std::max(d.w0n, plane + 1);
                at[e] = static_cast<int>(static_cast<size_t>(plane) * psi->N * L0.size + cell);
            }
            RBMG_CK(upload(h.get(), at, &d.w0at));
            for (const size_t bytes : {sizeof(float2), sizeof(double2)}) {
                auto w0 = std::make_unique<DevBuf>();
                const size_t n = bytes * d.w0n * psi->N * L0.size;
                RBMG_CK(w0->ensure(n));
                RBMG_CK(cudaMemset(w0->p, 0, n));
                (bytes == sizeof(float2) ? reinterpret_cast<const void*&>(d.w0)
                                         : reinterpret_cast<const void*&>(d.w064)) = w0->p;
                h->bufs.push_back(std::move(w0));
            }
            for (int l = 1; l < L; l++) {
                const auto& Ly = psi->layers[l];
                bool dense = Ly.conn == psi->layers[l - 1].size;
                for (size_t e = 0; dense && e < Ly.connections.size(); e++)
                    dense = Ly.connections[e] == e / Ly.size;
                if (!dense) continue;
                auto b = std::make_unique<DevBuf>();
                RBMG_CK(b->ensure(sizeof(float2) * Ly.weights.size()));
                d.wt[l] = b->as<float2>();
                h->bufs.push_back(std::move(b));
            }
        }
        std::vector<float2> f32(psi->final_weights.size());
        std::vector<double2> f64(psi->final_weights.size());
        for (size_t q = 0; q < f32.size(); q++) {
            const cplx z = psi->kind != 2 ? psi->final_weights[q]
                                          : (part == 0 ? cplx(psi->final_weights[q].real(), 0.0)
                                                       : cplx(psi->final_weights[q].imag(), 0.0));
            f32[q] = make_float2(float(z.real()), float(z.imag()));
            f64[q] = make_double2(z.real(), z.imag());
        }
        RBMG_CK(upload(h.get(), f32, &d.fw));
        RBMG_CK(upload(h.get(), f64, &d.fw64));
    }
    if (nets == 1) h->net[1] = h->net[0];
    psi->deep_dev[0] = h->net[0];
    psi->deep_dev[1] = h->net[1];
    psi->deep_host = std::shared_ptr<void>(h.release(), [](void* p) { delete static_cast<DeepHost*>(p); });
    // the uploads went through the legacy stream, which stream() does not wait for
    RBMG_CK(cudaStreamSynchronize(cudaStreamLegacy));
    const int r = deep_derive(psi);
    if (r != RBMG_OK) return r;
    RBMG_CK(cudaStreamSynchronize(stream()));
    return RBMG_OK;
}

static DeepNetDev net_of(const rbmg_psi* psi, int part) {
    DeepNetDev d = psi->deep_dev[part];
    d.ti = psi->translational_invariance;
    return d;
}

int deep_log_psi(const rbmg_psi* psi, int count, const uint64_t* d_spins, uint64_t enum_base, int enumerate,
                 double2* d_out, cudaStream_t st) {
    if (count <= 0) return RBMG_OK;
    const DeepNetDev n0 = net_of(psi, 0), n1 = net_of(psi, 1);
    // FP64: exact-summation weights and the psi vector are built from these values
    const size_t sm = smem_for(n0, sizeof(double2), false) + sizeof(uint64_t) * kMaxWords;
    RBMG_CK(set_smem(deep_logpsi_kernel<double2>, sm));
    deep_logpsi_kernel<double2><<<count, threads_for(n0), sm, st>>>(n0, n1, psi->kind == 2, count, d_spins, enum_base,
                                                                     enumerate, d_out);
    RBMG_CK(cudaGetLastError());
    return RBMG_OK;
}

// neighbours per batch of deep_local64_kernel: as many as leave room for three blocks an SM, at
// most 16, at least one
static int local64_batch(const DeepNetDev& n, bool grad) {
    int nb = 16;
    while (nb > 1 && deep_local64_smem(n, nb, grad) > 72 * 1024) nb /= 2;
    return nb;
}
// f(T) with the kernel's threads a block
template <typename F>
static cudaError_t local64_launch(const DeepNetDev& n, F f) {
    return widest(n) <= 128 ? f(std::integral_constant<int, 128>()) : f(std::integral_constant<int, 512>());
}

int deep_hsd64_chunk(const rbmg_psi* psi, const rbmg_psi* pp, const rbmg_operator* op, const Chunk& c,
                     double2* d_eloc, double2* d_dlp, cudaStream_t st) {
    if (c.count <= 0) return RBMG_OK;
    if (pp && (pp->width != psi->width || pp->layers.size() != psi->layers.size()))
        return fail(RBMG_EUNSUPPORTED, "hsd: psi and psi_prime need the same layer shapes");
    const rbmg_psi* p = pp ? pp : psi;
    const DeepNetDev n0 = net_of(psi, 0), n1 = net_of(psi, 1), q0 = net_of(p, 0), q1 = net_of(p, 1);
    bool alike = psi->kind == 1 && !n0.ti && !q0.ti;   // psi' is evaluated in psi's buffers
    for (int l = 0; l < n0.L; l++) alike = alike && n0.size[l] == q0.size[l];
    if (alike) {
        const int nb = local64_batch(n0, false);
        const size_t sm = deep_local64_smem(n0, nb, false);
        RBMG_CK(local64_launch(n0, [&](auto t) -> cudaError_t {
            const auto kernel = deep_local64_kernel<false, decltype(t)::value>;
            const cudaError_t e = set_smem(kernel, sm);
            if (e != cudaSuccess) return e;
            kernel<<<c.count, decltype(t)::value, sm, st>>>(n0, op->dev(), c.count, c.spins, c.enum_base, c.enumerate, nb,
                                                            q0, d_dlp, make_double2(0.0, 0.0), d_eloc, nullptr, nullptr,
                                                            0);
            return cudaGetLastError();
        }));
    } else {
        const size_t sm = smem_for(n0, sizeof(double2), false) + 2 * sizeof(uint64_t) * kMaxWords;
        auto run = [&](auto kernel) -> cudaError_t {
            const cudaError_t e = set_smem(kernel, sm);
            if (e != cudaSuccess) return e;
            kernel<<<c.count, threads_for(n0), sm, st>>>(n0, n1, psi->kind == 2, q0, q1, op->dev(), c.count, c.spins,
                                                         c.enum_base, c.enumerate, d_eloc, d_dlp);
            return cudaSuccess;
        };
        RBMG_CK(pp ? run(deep_eloc_kernel<double2, true>) : run(deep_eloc_kernel<double2, false>));
    }
    RBMG_CK(cudaGetLastError());
    return RBMG_OK;
}

int deep_eloc_chunk(const rbmg_psi* psi, const rbmg_operator* op, const Chunk& c, double2* d_eloc, cudaStream_t st) {
    return deep_hsd64_chunk(psi, nullptr, op, c, d_eloc, nullptr, st);
}

static DevBuf& rows_buf(int which) {
    static thread_local DevBuf b[3];
    return b[which];
}

static int col_reduce(int count, int P, const double2* c, const double2* A, long ld, int conj_a, double2* out,
                      cudaStream_t st) {
    if (count <= 0) return RBMG_OK;
    const int per_split = std::max(64, (count + 63) / 64);
    const int splits = (count + per_split - 1) / per_split;
    DevBuf& part = rows_buf(2);
    RBMG_CK(part.ensure(sizeof(double2) * static_cast<size_t>(splits) * P));
    const dim3 grid((P + 255) / 256, splits);
    col_reduce_kernel<<<grid, 256, 0, st>>>(count, P, c, A, ld, conj_a, part.as<double2>(), per_split);
    col_finish_kernel<<<(P + 255) / 256, 256, 0, st>>>(P, splits, part.as<double2>(), out);
    RBMG_CK(cudaGetLastError());
    return RBMG_OK;
}

// O_k rows (k >= 2N) of `count` configurations into rows [count][ld] (FP64, PsiDeep)
int deep_ok_rows(const rbmg_psi* psi, int count, const uint64_t* d_spins, uint64_t enum_base, int enumerate,
                 double2* rows, long ld, cudaStream_t st) {
    if (psi->kind != 1) return fail(RBMG_EUNSUPPORTED, "O_k rows: PsiDeep only (PsiPair.hpp:73-76 defines none)");
    if (count <= 0) return RBMG_OK;
    const DeepNetDev net = net_of(psi, 0);
    const size_t sm = smem_for(net, sizeof(double2), true);
    RBMG_CK(set_smem(deep_ok_kernel<false>, sm));
    deep_ok_kernel<false><<<count, threads_for(net), sm, st>>>(net, count, d_spins, enum_base, enumerate, rows, ld);
    RBMG_CK(cudaGetLastError());
    return RBMG_OK;
}

int deep_hsd_okreduce(const rbmg_psi* pp, int pair_part, int count, const uint64_t* d_spins, uint64_t enum_base,
                      int enumerate, const double2* d_coef, double2* acc, cudaStream_t st) {
    const DeepNetDev net = net_of(pp, pair_part == 1 ? 1 : 0);
    const int P = net.P - 2 * net.N;
    const int chunk = std::max(1, static_cast<int>((size_t(256) << 20) / (sizeof(double2) * P)));
    DevBuf& rows = rows_buf(0);
    RBMG_CK(rows.ensure(sizeof(double2) * static_cast<size_t>(std::min(chunk, count)) * P));
    const size_t sm = smem_for(net, sizeof(double2), true);
    for (int base = 0; base < count; base += chunk) {
        const int cnt = std::min(chunk, count - base);
        const uint64_t* sp = d_spins ? d_spins + static_cast<size_t>(base) * ((net.N + 63) / 64) : nullptr;
        if (pp->kind == 2) {
            RBMG_CK(set_smem(deep_ok_kernel<true>, sm));
            deep_ok_kernel<true><<<cnt, threads_for(net), sm, st>>>(net, cnt, sp, enum_base + base, enumerate,
                                                                    rows.as<double2>(), P);
        } else {
            RBMG_CK(set_smem(deep_ok_kernel<false>, sm));
            deep_ok_kernel<false><<<cnt, threads_for(net), sm, st>>>(net, cnt, sp, enum_base + base, enumerate,
                                                                     rows.as<double2>(), P);
        }
        RBMG_CK(cudaGetLastError());
        // real O_k (PsiPair) multiply the real or complex coefficient; complex O_k enter conjugated
        const int r = col_reduce(cnt, P, d_coef + base, rows.as<double2>(), P, pp->kind == 2 ? 0 : 1, acc, st);
        if (r != RBMG_OK) return r;
    }
    return RBMG_OK;
}

int deep_ok_vector(const rbmg_psi* psi, const uint64_t* d_spins, double2* d_out, cudaStream_t st) {
    if (psi->kind == 2) return fail(RBMG_EUNSUPPORTED, "psi_O_k_vector: not defined for PsiPair (PsiPair.hpp:73-76)");
    const DeepNetDev net = net_of(psi, 0);
    const int P = net.P - 2 * net.N;
    DevBuf& rows = rows_buf(0);
    RBMG_CK(rows.ensure(sizeof(double2) * P));
    const size_t sm = smem_for(net, sizeof(double2), true);
    RBMG_CK(set_smem(deep_ok_kernel<false>, sm));
    deep_ok_kernel<false><<<1, threads_for(net), sm, st>>>(net, 1, d_spins, 0, 0, rows.as<double2>(), P);
    RBMG_CK(cudaGetLastError());
    RBMG_CK(cudaMemsetAsync(d_out, 0, sizeof(double2) * P, st));
    DevBuf& one = rows_buf(1);
    RBMG_CK(one.ensure(sizeof(double2)));
    const double2 h1 = make_double2(1.0, 0.0);
    RBMG_CK(cudaMemcpyAsync(one.p, &h1, sizeof(double2), cudaMemcpyHostToDevice, st));
    return col_reduce(1, P, one.as<double2>(), rows.as<double2>(), P, 0, d_out, st);
}

int deep_gradient_chunk(const rbmg_psi* psi, const rbmg_operator* op, const Chunk& c, double2 e_shift,
                        double2* d_eloc, double2* acc_O, double2* acc_EO, double2* acc_Ek, double2* coef1,
                        double2* coef2, cudaStream_t st, double2* acc_B, double2* coef3) {
    if (psi->kind == 2) return fail(RBMG_EUNSUPPORTED, "gradient: not instantiated for PsiPair (ExpectationValue.cu:553)");
    const DeepNetDev net = net_of(psi, 0);
    const int P = net.P - 2 * net.N;
    const int chunk = std::max(1, static_cast<int>((size_t(512) << 20) / (2 * sizeof(double2) * P)));
    DevBuf& orows = rows_buf(0);
    DevBuf& erows = rows_buf(1);
    RBMG_CK(orows.ensure(sizeof(double2) * static_cast<size_t>(std::min(chunk, c.count)) * P));
    RBMG_CK(erows.ensure(sizeof(double2) * static_cast<size_t>(std::min(chunk, c.count)) * P));
    int dev = 0, sms = 0;
    RBMG_CK(cudaGetDevice(&dev));
    RBMG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int nb = local64_batch(net, true);
    const size_t sm = deep_local64_smem(net, nb, true);
    DevBuf& part = rows_buf(2);
    RBMG_CK(launch_coef(c.count, c.weights, nullptr, 1.0, coef1, st));
    for (int base = 0; base < c.count; base += chunk) {
        const int cnt = std::min(chunk, c.count - base);
        const uint64_t* sp = c.spins ? c.spins + static_cast<size_t>(base) * ((net.N + 63) / 64) : nullptr;
        RBMG_CK(local64_launch(net, [&](auto t) -> cudaError_t {
            const auto kernel = deep_local64_kernel<true, decltype(t)::value>;
            const cudaError_t e = set_smem(kernel, sm);
            if (e != cudaSuccess) return e;
            kernel<<<cnt, decltype(t)::value, sm, st>>>(net, op->dev(), cnt, sp, c.enum_base + base, c.enumerate, nb, net,
                                                        nullptr, e_shift, d_eloc + base, orows.as<double2>(),
                                                        erows.as<double2>(), P);
            return cudaGetLastError();
        }));
        const double* wb = c.weights ? c.weights + base : nullptr;
        RBMG_CK(launch_coef(cnt, wb, d_eloc + base, 1.0, coef2 + base, st, e_shift));
        // sum w conj(E - E0) (E_k - E0 O_k): the fluctuation gradient's covariance term
        if (acc_B) RBMG_CK(launch_coef_conj(cnt, wb, d_eloc + base, e_shift, coef3 + base, st));
        // enough splits of the samples for four blocks an SM, of eight samples at least
        const int cols = (P + 127) / 128, want = std::max(1, 4 * sms / cols);
        const int per = std::max(8, (cnt + want - 1) / want);
        const int splits = (cnt + per - 1) / per;
        RBMG_CK(part.ensure(sizeof(double2) * 4 * static_cast<size_t>(splits) * P));
        row_sums_kernel<<<dim3(cols, splits), 128, 0, st>>>(cnt, P, coef1 + base, coef2 + base,
                                                            acc_B ? coef3 + base : nullptr, orows.as<double2>(),
                                                            erows.as<double2>(), P, part.as<double2>(), per);
        row_sums_finish_kernel<<<dim3(cols, 4), 128, 0, st>>>(P, splits, part.as<double2>(),
                                                              RowSums{{acc_O, acc_EO, acc_Ek, acc_B}});
        RBMG_CK(cudaGetLastError());
    }
    return RBMG_OK;
}

// Adjoint of the local energy over one chunk of samples, accumulated into the dense
// per-layer gradient blocks G (double2): for layer l, G_w[l] [size_l][in_l] (in_0 = N)
// and G_b[l] [size_l], then G_fw [last]; offsets in `goff`.  d_eloc receives E_loc.
int deep_adjoint_chunk(const rbmg_psi* psi, const rbmg_operator* op, const Chunk& c, int score, double2* d_eloc,
                       double2* G, double2* GO, const std::vector<size_t>& goff, cudaStream_t st) {
    const DeepNetDev net = net_of(psi, 0);
    const int nw = (net.N + 63) / 64;
    const int xs = 1 + op->num_offdiag;
    static thread_local DevBuf acts, dlts, alpha, xsp, dltsO, alphaO, partial;
    const size_t per_sample = static_cast<size_t>(xs) * (2 * sizeof(float2) * net.units + sizeof(float2) + 8 * nw) +
                              sizeof(float2) * (net.units + 1);
    // parts of the FP32 sums (AdjSplit) of at most 768 MB of stored activations and errors, and as many
    // parts per launch as fit 4 GB of them, held by the thread (N = 100, 200-100-50, 8192 samples: one
    // part 35.3 ms, 1.6 GB 33.5, 4 GB 32.0, 8 GB 32.0); one part where the device has no room for more
    const int part = std::max(1, static_cast<int>(std::min<size_t>(c.count, (size_t(768) << 20) / per_sample)));
    int chunk = static_cast<int>(std::min<size_t>(
        c.count, static_cast<size_t>(part) * std::max<size_t>(1, (size_t(4) << 30) / (per_sample * part))));
    auto room = [&]() {
        cudaError_t e = acts.ensure(sizeof(float2) * static_cast<size_t>(chunk) * xs * net.units);
        if (e == cudaSuccess) e = dlts.ensure(sizeof(float2) * static_cast<size_t>(chunk) * xs * net.units);
        if (e == cudaSuccess) e = alpha.ensure(sizeof(float2) * static_cast<size_t>(chunk) * xs);
        if (e == cudaSuccess) e = xsp.ensure(sizeof(uint64_t) * static_cast<size_t>(chunk) * xs * nw);
        if (e == cudaSuccess) e = dltsO.ensure(sizeof(float2) * static_cast<size_t>(chunk) * net.units);
        return e == cudaSuccess ? alphaO.ensure(sizeof(float2) * static_cast<size_t>(chunk)) : e;
    };
    cudaError_t held = room();
    if (held == cudaErrorMemoryAllocation && chunk > part) {
        cudaGetLastError();
        acts.release();
        dlts.release();
        chunk = part;
        held = room();
    }
    RBMG_CK(held);
    const size_t sm = smem_for(net, sizeof(float2), true) + 2 * sizeof(float2) * net.size[0];
    RBMG_CK(set_smem(deep_adjoint_kernel, sm));
    // neighbours per pass of the reverse kernel: eight, or as many as the widest nets leave room
    // for in a block's shared memory (three layers of 720 units: four), or what
    // RBMG_DEEP_ADJOINT_BATCH = 1, 2, 4 or 8 says; the same outputs
    int nbatch = 8, dev = 0, sms = 0;
    RBMG_CK(cudaGetDevice(&dev));
    RBMG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (const char* v = std::getenv("RBMG_DEEP_ADJOINT_BATCH")) {
        nbatch = std::atoi(v);
    } else {
        int limit = 0;
        RBMG_CK(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        while (nbatch > 2 && deep_adjoint_pairs_smem(net, nbatch / 2) > static_cast<size_t>(limit)) nbatch /= 2;
    }
    if (nbatch != 1 && nbatch != 2 && nbatch != 4 && nbatch != 8)
        return fail(RBMG_EINVAL, "RBMG_DEEP_ADJOINT_BATCH: 1, 2, 4 or 8");
    const size_t smb = deep_adjoint_pairs_smem(net, nbatch / 2);
    // narrow nets keep 128 threads from three blocks an SM on (512 samples of 128-128, N = 20: 672 us,
    // with 256 threads 700)
    const int units = widest(net);
    const int threads = pair_threads(smb, units, std::min(c.count, chunk), sms, units <= 128 ? 3 : kPairsAdjBlocks);
    for (int base = 0; base < c.count; base += chunk) {
        const int cnt = std::min(chunk, c.count - base);
        const uint64_t* sp = c.spins ? c.spins + static_cast<size_t>(base) * nw : nullptr;
        const double* wb = c.weights ? c.weights + base : nullptr;
        auto pairs_kernel = [&](auto pairs, auto t) -> cudaError_t {
            const auto kernel = deep_adjoint_pairs_kernel<decltype(pairs)::value, decltype(t)::value>;
            const cudaError_t e = set_smem(kernel, smb);
            if (e != cudaSuccess) return e;
            kernel<<<cnt, decltype(t)::value, smb, st>>>(
                net, op->dev(), cnt, sp, c.enum_base + base, c.enumerate, wb, score, d_eloc + base,
                acts.as<float2>(), dlts.as<float2>(), alpha.as<float2>(), xsp.as<uint64_t>(), xs, dltsO.as<float2>(),
                alphaO.as<float2>());
            return cudaGetLastError();
        };
        if (nbatch > 1) {
            RBMG_CK(pairs_launch(nbatch / 2, threads, pairs_kernel));
        } else {
            deep_adjoint_kernel<<<cnt, threads_for(net), sm, st>>>(
                net, op->dev(), cnt, sp, c.enum_base + base, c.enumerate, wb, score, d_eloc + base,
                acts.as<float2>(), dlts.as<float2>(), alpha.as<float2>(), xsp.as<uint64_t>(), xs, dltsO.as<float2>(),
                alphaO.as<float2>());
            RBMG_CK(cudaGetLastError());
        }
        auto sum = [&](int M, int Nn, int cols, int splits, double2* out, double2* bias) -> cudaError_t {
            const long total = static_cast<long>(M) * cols;
            adj_split_sum_kernel<<<static_cast<unsigned>((total + 31) / 32), 256, 0, st>>>(M, Nn, cols, splits,
                                                                                         partial.as<float2>(), out, bias);
            return cudaGetLastError();
        };
        // pass 0: all configurations with alpha-weighted deltas -> G; pass 1 (score): the
        // samples themselves with weight w_s -> GO
        for (int pass = 0; pass < (score ? 2 : 1); pass++) {
            const int K = pass == 0 ? cnt * xs : cnt, rows = pass == 0 ? part * xs : part;
            const int splits = adj_grid_splits(K, rows);
            const int row = pass == 0 ? net.units : xs * net.units;     // activation row stride
            const float2* dl = pass == 0 ? dlts.as<float2>() : dltsO.as<float2>();
            double2* out = pass == 0 ? G : GO;
            for (int l = 0; l < net.L; l++) {
                const int size = net.size[l], in = l == 0 ? net.N : net.size[l - 1];
                RBMG_CK(partial.ensure(sizeof(float2) * static_cast<size_t>(splits) * size * (in + 1)));
                const int tn = l == 0 ? 128 : 64;
                const dim3 grid((size + kAdjTm - 1) / kAdjTm, (in + tn) / tn, splits);
                if (l == 0)
                    adj_cgemm_kernel<true><<<grid, 128, 0, st>>>(K, rows, size, in, dl, net.units, nullptr, 0,
                                                                  xsp.as<uint64_t>(), pass == 0 ? nw : xs * nw,
                                                                  partial.as<float2>());
                else
                    adj_cgemm_kernel<false><<<grid, 128, 0, st>>>(
                        K, rows, size, in, dl + net.begin_angle[l], net.units, acts.as<float2>() + net.begin_angle[l - 1], row,
                        nullptr, 0, partial.as<float2>());
                RBMG_CK(cudaGetLastError());
                RBMG_CK(sum(size, in, in + 1, splits, out + goff[2 * l], out + goff[2 * l + 1]));
            }
            const int last = net.size[net.L - 1];
            RBMG_CK(partial.ensure(sizeof(float2) * static_cast<size_t>(splits) * last));
            adj_final_kernel<<<dim3((last + 31) / 32, splits), 256, 0, st>>>(
                K, rows, last, pass == 0 ? alpha.as<float2>() : alphaO.as<float2>(),
                acts.as<float2>() + net.begin_angle[net.L - 1], row, partial.as<float2>());
            RBMG_CK(cudaGetLastError());
            RBMG_CK(sum(1, last, last, splits, out + goff[2 * net.L], nullptr));
        }
    }
    return RBMG_OK;
}

// MonteCarloLoop::foreach for PsiDeep / PsiPair (MonteCarloLoop.hpp:294-339)
int deep_stream(rbmg_ensemble* e, const rbmg_psi* psi, const rbmg_operator* op, bool want_eloc,
                size_t max_chunk_samples, bool defer, const std::function<int(const Chunk&)>& fn) {
    (void)op;
    (void)want_eloc;
    if (e->total_z) return fail(RBMG_EUNSUPPORTED, "PsiDeep chains: S_z symmetry is not provided");
    const int nw = (psi->N + 63) / 64;
    const int B = static_cast<int>(e->num_chains);
    const int steps = static_cast<int>(e->num_samples / e->num_chains);
    RBMG_CK(e->spins.ensure(sizeof(uint64_t) * nw * B));
    RBMG_CK(cudaMemsetAsync(e->accepts.p, 0, sizeof(unsigned long long) * B, stream()));
    RBMG_CK(cudaMemsetAsync(e->proposals.p, 0, sizeof(unsigned long long) * B, stream()));
    static thread_local DevBuf samples;
    const int rows_per_chunk = static_cast<int>(std::max<size_t>(1, std::min<size_t>(steps, max_chunk_samples / B)));
    RBMG_CK(samples.ensure(sizeof(uint64_t) * nw * B * rows_per_chunk));
    const DeepNetDev n0 = net_of(psi, 0), n1 = net_of(psi, 1);
    // + layer 0's pre-activations of the state and of a proposal
    const size_t sm = smem_for(n0, sizeof(float2), false) + 2 * sizeof(float2) * n0.size[0];
    RBMG_CK(set_smem(deep_mc_kernel, sm));
    // single-flip chains of a complex net: several walkers per CTA (RBMG_DEEP_WALKERS_PER_BLOCK
    // = 1, 2, 4 or 8; default 8, the fastest on the 100-200-100-50 net), the same chains
    int wpc = 8;
    if (const char* v = std::getenv("RBMG_DEEP_WALKERS_PER_BLOCK")) wpc = std::atoi(v);
    if (wpc != 1 && wpc != 2 && wpc != 4 && wpc != 8) return fail(RBMG_EINVAL, "RBMG_DEEP_WALKERS_PER_BLOCK: 1, 2, 4 or 8");
    if (e->fast_sweep_tries != 0 || psi->kind == 2 || n0.ti) wpc = 1;
    const size_t smm = deep_mc_pairs_smem(n0, wpc / 2);
    const int blocks = (B + wpc - 1) / wpc;
    int dev = 0, sms = 0;
    RBMG_CK(cudaGetDevice(&dev));
    RBMG_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int threads = pair_threads(smm, widest(n0), blocks, sms, kPairsMcBlocks);
    bool first = true;
    for (int row0 = 0; row0 < steps; row0 += rows_per_chunk) {
        const int rows = std::min(rows_per_chunk, steps - row0);
        McLaunch L{};
        L.B = B;
        L.seed = e->seed;
        L.spins = e->spins.as<uint64_t>();
        L.rng_index = e->rng_index.as<uint64_t>();
        L.init = first ? 1 : 0;
        L.fast_tries = static_cast<int>(e->fast_sweep_tries);
        L.n_therm = first ? static_cast<int>(e->num_therm) : 0;
        L.n_samples = rows;
        L.sweeps_per_sample = static_cast<int>(e->num_sweeps);
        L.sample_spins = samples.as<uint64_t>();
        L.accepts = e->accepts.as<unsigned long long>();
        L.proposals = e->proposals.as<unsigned long long>();
        auto pairs_kernel = [&](auto pairs, auto t) -> cudaError_t {
            const auto kernel = deep_mc_pairs_kernel<decltype(pairs)::value, decltype(t)::value>;
            const cudaError_t e = set_smem(kernel, smm);
            if (e != cudaSuccess) return e;
            kernel<<<blocks, decltype(t)::value, smm, stream()>>>(n0, L);
            return cudaGetLastError();
        };
        if (wpc > 1) {
            RBMG_CK(pairs_launch(wpc / 2, threads, pairs_kernel));
        } else {
            deep_mc_kernel<<<B, threads_for(n0), sm, stream()>>>(n0, n1, psi->kind == 2, L);
            RBMG_CK(cudaGetLastError());
        }
        first = false;
        Chunk c;
        c.count = c.group = rows * B;
        c.spins = samples.as<uint64_t>();
        const int r = fn(c);
        if (r != RBMG_OK) return r;
    }
    RBMG_CK(e->counts_copy());
    if (defer) return RBMG_OK;
    RBMG_CK(cudaStreamSynchronize(stream()));
    e->counts_take();
    return RBMG_OK;
}

}  // namespace rbmg
