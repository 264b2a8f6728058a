// Launchers of the deterministic per-sample reductions (reduce_kernels.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.h"

namespace rbmg {

constexpr int kMaxSeries = 6;
constexpr int kSumBlocks = 512;
// a sum's scratch in double2: the blocks' partial sums, then the arrival counter of its blocks
// (zero before the first sum; every sum leaves it zero)
constexpr int kSumScratch = kSumBlocks * kMaxSeries + 1;

struct SeriesSet {
    int n;
    const double2* v[kMaxSeries];
};

// up to kMaxOuter sums over the same rows A: out_q[r][j] += sum_s c_q[s] f_q(A[s][j]) g_r(s),
// g_0 = 1, g_{1+i} = s_i; f_q = conj if conj_q.  partial: scratch of
// n * outer_splits(count, max_splits) * (1+N) * M double2.
constexpr int kMaxOuter = 3;
struct OuterSet {
    int n;
    const double2* c[kMaxOuter];
    int conj[kMaxOuter];
    double2* out[kMaxOuter];
    void add(const double2* coef, int conjugate, double2* sum) {
        c[n] = coef;
        conj[n] = conjugate;
        out[n++] = sum;
    }
};
// A sum's partials over the splits of its samples, added to (or stored as) the outputs:
// out_q[e] (+)= scale sum_z partial[z][q][e], and to out_0 before that -2 sum_z pre[z][e]
struct SplitSum {
    long elems;
    int splits, nc;
    const double2* partial;
    double2* out[kMaxOuter];
    double scale;
    const double2* pre;
    int pre_splits;
};
// the splits that the sums below make of so many samples, and the blocks of one split of an outer sum
int outer_splits(int count, int max_splits);
int vterm_splits(int count, int max_splits);
int outer_tiles(int N, int M);
// with job: the partials are left for launch_split_sums
cudaError_t launch_outer_reduce(int count, int N, int nw, int M, const uint64_t* spins, uint64_t enum_base,
                                int enumerate, const OuterSet& set, const float2* A, int lda, double2* partial,
                                int max_splits, cudaStream_t st, SplitSum* job = nullptr);
cudaError_t launch_split_sums(const SplitSum* jobs, int n, bool add, cudaStream_t st);
// out[1+i][j] += -2 sum_s w[s] s_i sum_{slots of site i} X[s][slot][j]; with cw the per-sample
// coefficient is the complex cw[s] (w ignored)
cudaError_t launch_vterm_reduce(int count, int N, int nw, int M, int Mpad, const uint64_t* spins, uint64_t enum_base,
                                int enumerate, const double* w, const float2* X, int num_offdiag,
                                const int* site_ptr, const int* site_slots, double2* out, double2* partial,
                                int max_splits, cudaStream_t st, const double2* cw = nullptr);
// U [count][Mpad] (EstLaunch) and the V sums of launch_vterm_reduce for an operator whose
// off-diagonal strings flip one site each, no two the same, from the strings' terms `en`
// [count][num_offdiag] and the angles `theta` [count][Mpad]; partial: grad_vectors_bytes
struct GradVectors {
    int count, N, nw, M, Mpad;
    int group;            // the samples come in groups of so many, the FP32 sums formed within each
    int max_splits;       // over at most so many splits of a group
    const uint64_t* spins;
    uint64_t enum_base;
    int enumerate;
    const double* w;
    const float2* W;      // [N][Mpad]
    const float2* theta;
    const float2* T;      // [count][Mpad] tanh(theta)
    const float2* en;
    float2* U;
    const double2* e_shift;   // U is stored as U - e_shift T
    const int* site_ptr;  // [N + 1]
};
size_t grad_vectors_bytes(int count, int group, int N, int M, int Mpad, int max_splits, int sms);
// the V sums' partials are left in job's pre
cudaError_t launch_grad_vectors(const GradVectors& g, const OpDev& op, double2* partial, int sms, cudaStream_t st,
                                SplitSum* job);
// sums[q] += sum_s w[s] v_q[s]; block_scratch: kSumScratch double2
cudaError_t launch_weighted_sums(int count, const double* w, const SeriesSet& set, double2* block_scratch,
                                 double2* sums, cudaStream_t st);
// mean[0] = sum_s w[s] v[s] / sum_s w[s] (0 if the weights sum to nothing); scratch as above
cudaError_t launch_weighted_mean(int count, const double* w, const double2* v, double2* block_scratch, double2* mean,
                                 cudaStream_t st);
// The weights of exact summation, w[s] = exp(2 Re lp[s] - log Z): stat[0] = (m, sum_s exp(2 Re
// lp[s] - m)) with m the largest 2 Re lp, stat[1].x = log Z
cudaError_t launch_exact_weights(int count, const double2* lp, double* w, double2* block_scratch, double2* stat,
                                 cudaStream_t st);
// the samples' coefficients of the gradient's sums: c1 = (w, 0), c2 = w (v - shift), and c3 (may
// be null) = (w (Re v - Re shift), 0), or w conj(v - shift) with conj3
cudaError_t launch_grad_coefs(int count, const double* w, const double2* v, const double2* shift, double2* c1,
                              double2* c2, double2* c3, int conj3, cudaStream_t st);
// The gradient from its sums, entries below first zero (GradOut::mode), and the energy
struct GradOut {
    int mode;              // 0: the estimator; 1, 2: derivative of <E_loc>, samples held fixed / with the sampling term
    const double2 *O, *A, *B, *C;   // sums of O and, mode 0, (E - E0) O*, E_k - E0 O; else E_k - E0 O, (E - E0) O, (Re E - Re E0) O*
    const double2* sums;   // [1] sum of w E
    const double2* e0;
    const double2* stat;   // exact summation (launch_exact_weights), else null
    double norm;           // the sums' factor; exact summation: the log of the prefactor squared
    int first;
    long count;
    double2* grad;
    double* status;        // [4] E (normalised), the factor, stat's largest 2 Re log psi (host memory)
};
cudaError_t launch_grad_out(const GradOut& g, cudaStream_t st);
cudaError_t launch_max_re2(int count, const double2* lp, double* block_max, int* blocks_out, cudaStream_t st);
cudaError_t launch_exp_weights(int count, const double2* lp, double shift, double* w, cudaStream_t st);
// c[s] = scale w[s] (v[s] - shift), or scale w[s] when v is null
cudaError_t launch_coef(int count, const double* w, const double2* v, double scale, double2* c, cudaStream_t st,
                        double2 shift = make_double2(0.0, 0.0));
cudaError_t launch_abs2(int count, const double2* v, double2* out, cudaStream_t st);
// c[s] = w[s] conj(v[s] - shift)
cudaError_t launch_coef_conj(int count, const double* w, const double2* v, double2 shift, double2* c,
                             cudaStream_t st);
// rw[s] = w[s] |psi(s) / psi'(s)|^2 from log psi and log psi', rwc[s] = (rw[s], 0)
cudaError_t launch_ratio_weights(int count, const double* w, const double2* lp, const double2* lpp, double* rw,
                                 double2* rwc, cudaStream_t st);
// a[s] = exp(2 Im E + Re(E E - E)), the weight of ExpectationValue::corrected
cudaError_t launch_corrected_terms(int count, const double2* e, double2* a, cudaStream_t st);

}  // namespace rbmg
