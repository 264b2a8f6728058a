// Host-side objects behind the C ABI handles, shared by capi.cu and deep.cu.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <complex>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <memory>
#include <string>
#include <thread>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/rbmg.h"
#include "kernels.h"

namespace rbmg {

using cplx = std::complex<double>;

void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* where);

#define RBMG_CK(call)                                                    \
    do {                                                                 \
        cudaError_t e__ = (call);                                        \
        if (e__ != cudaSuccess) return ::rbmg::cuda_fail(e__, #call);    \
    } while (0)

// grow-only device buffer
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    cudaError_t ensure(size_t n) {
        if (n <= bytes) return cudaSuccess;
        release();
        cudaError_t e = cudaMalloc(&p, n);
        if (e != cudaSuccess) { p = nullptr; return e; }
        bytes = n;
        return cudaSuccess;
    }
    template <typename T>
    T* as() const { return static_cast<T*>(p); }
};

// grow-only pinned host buffer, addressable by the device
struct HostBuf {
    void* p = nullptr;
    size_t bytes = 0;
    HostBuf() = default;
    HostBuf(const HostBuf&) = delete;
    HostBuf& operator=(const HostBuf&) = delete;
    ~HostBuf() { release(); }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
    }
    cudaError_t ensure(size_t n) {
        if (n <= bytes) return cudaSuccess;
        release();
        cudaError_t e = cudaMallocHost(&p, n);
        if (e != cudaSuccess) { p = nullptr; return e; }
        bytes = n;
        return cudaSuccess;
    }
    template <typename T>
    T* as() const { return static_cast<T*>(p); }
};

// Makes the pages of a host output present before the GPU writes them: the copy to pageable
// memory is a direct write of the GPU, which takes the first-touch fault of every page of a
// freshly allocated array one by one (measured: 300 KB into fresh pages 226 us, into touched
// ones 18 us and 25 us for the touches; 16 MB 13.5 ms against 0.10 and 0.73).  One byte of
// every page is written, so only for memory that the copy then overwrites.  Large outputs are
// touched by a thread per 4 MB (16 at most) from the construction on, while the GPU works;
// join() ends them, or touches a smaller output itself, and comes before the copy.
class Prefault {
  public:
    Prefault(void* p, size_t bytes) : p_(static_cast<char*>(p)), bytes_(bytes) {
        if (bytes < size_t(8) << 20) return;
        if (present(p_, bytes)) {   // memory that the allocator has handed out again
            started_ = bytes;
            return;
        }
        // asked for once: a call reads a file, 5 to 10 us
        static const size_t cores = std::max(1u, std::thread::hardware_concurrency());
        const size_t n = std::min<size_t>({16, cores, bytes >> 22});
        if (n < 2) return;
        const size_t per = ((bytes + n - 1) / n + 65535) / 65536 * 65536;
        try {
            threads_.reserve(n);
            for (; started_ < bytes; started_ += per) {
                char* a = p_ + started_;
                const size_t len = std::min(per, bytes - started_);
                threads_.emplace_back([=]() { touch(a, len); });
            }
        } catch (const std::exception&) {   // no more threads: join() touches the rest
        }
    }
    Prefault(const Prefault&) = delete;
    Prefault& operator=(const Prefault&) = delete;
    void join() {
        if (started_ < bytes_ && bytes_ >= kSmall) touch(p_ + started_, bytes_ - started_);
        started_ = bytes_;
        for (auto& t : threads_) t.join();
        threads_.clear();
    }
    ~Prefault() {
        for (auto& t : threads_) t.join();
    }

  private:
    // below, the array comes from pages the process already holds (19 us either way at 64 KB)
    static constexpr size_t kSmall = size_t(96) << 10;
    static size_t page_size() {
        static const size_t page = static_cast<size_t>(std::max(4096L, sysconf(_SC_PAGESIZE)));
        return page;
    }
    // whether every page is in memory (a few us for 32 MB of 64 KB pages; making eight threads for
    // nothing took 160 us of an S matrix of 1100)
    static bool present(char* a, size_t bytes) {
        const size_t page = page_size(), lo = reinterpret_cast<size_t>(a) / page * page;
        const size_t pages = (reinterpret_cast<size_t>(a) + bytes - lo + page - 1) / page;
        try {
            std::vector<unsigned char> in(pages);
            return mincore(reinterpret_cast<void*>(lo), pages * page, in.data()) == 0 &&
                   std::all_of(in.begin(), in.end(), [](unsigned char v) { return v & 1; });
        } catch (const std::exception&) {
            return false;
        }
    }
    static void touch(char* a, size_t bytes) {
        const size_t page = page_size();
        for (size_t q = 0; q < bytes; q += page) *reinterpret_cast<volatile char*>(a + q) = 0;
        *reinterpret_cast<volatile char*>(a + bytes - 1) = 0;   // the last page of an unaligned array
    }
    char* p_;
    size_t bytes_, started_ = 0;
    std::vector<std::thread> threads_;
};
inline void prefault(void* p, size_t bytes) { Prefault(p, bytes).join(); }

cudaStream_t stream();

inline int nwords_of(int N) { return (N + 63) / 64; }

struct DeepLayerHost {
    int size = 0, conn = 0;
    std::vector<uint32_t> connections;   // [conn][size]
    std::vector<cplx> biases;            // [size]
    std::vector<cplx> weights;           // [conn][size]
};

struct DeepDev;   // deep.cu

}  // namespace rbmg

struct rbmg_psi {
    int kind = 0;     // 0 RBM, 1 PsiDeep, 2 PsiPair
    int N = 0;
    double prefactor = 1.0;
    std::vector<double> alpha, beta;
    int free_quantum_axis = 0;   // the Hilbert-space distance's alpha / beta terms (PsiBase.hpp:164)
    // RBM
    int M = 0, Mpad = 0;
    std::vector<rbmg::cplx> b, W;
    rbmg::DevBuf dW, db, dWq, dbq;     // complex64 rows, and the sampler's paired copies (kernels.h)
    rbmg::DevBuf dWg, dbg;             // paired copies of the grouped sampler (RbmDev::Wg)
    rbmg::DevBuf dWt;                  // W transposed, units paired [Mpad / 2][N] (RbmDev::Wt4)
    rbmg::DevBuf dWtc;                 // W as BF16 hi / mid / lo tensor-core operands (angles_tc.cu), if supported
    rbmg::DevBuf tc_error;             // set when a tensor-core pass of this psi gave up waiting
    mutable rbmg::DevBuf dW64, db64;   // FP64 copies for the Hilbert-space distance pass, uploaded on use
    mutable bool f64_valid = false;
    // deep / pair
    std::vector<rbmg::DeepLayerHost> layers;
    std::vector<rbmg::cplx> final_weights;
    int translational_invariance = 0;
    rbmg::DeepNetDev deep_dev[2] = {};     // device nets (deep.cu): complex net, or PsiPair real / imaginary
    std::shared_ptr<void> deep_host;       // owner of the device buffers behind deep_dev
    int width = 0;

    // device master copy of the packed parameter vector [P] complex128, written by the
    // device optimiser (optim.cu); while host_stale is set the vectors above are out of
    // date and psi_sync_host refreshes them before any host read
    rbmg::DevBuf dmaster;
    bool master_valid = false;
    mutable bool host_stale = false;

    int num_params() const;
    rbmg::RbmDev rbm_dev() const {
        return rbmg::RbmDev{N, M, Mpad, static_cast<const float2*>(dW.p), static_cast<const float2*>(db.p),
                            static_cast<const float4*>(dWq.p), static_cast<const float4*>(dbq.p),
                            static_cast<const float4*>(dWt.p), static_cast<const float4*>(dWg.p),
                            static_cast<const float4*>(dbg.p)};
    }
};

namespace rbmg {
// optim.cu: host copy of the parameters from the device master when the optimiser
// has moved them; packed device master from the host copy; device parameters (the
// layouts the kernels read) from a packed vector on the device
int psi_sync_host(const rbmg_psi* psi);
int psi_master_ensure(rbmg_psi* psi);
int psi_scatter(rbmg_psi* psi, const double2* packed);

// One chunk of samples: spins on the device (or basis indices when enumerate),
// per-sample weights (null = equal weights) and, for MC, the sampler's log psi / E_loc.
struct Chunk {
    int count = 0;
    int group = 0;   // the samples of a chunk of the plain size, of which this one may hold several
    const uint64_t* spins = nullptr;
    int enumerate = 0;
    uint64_t enum_base = 0;
    const double* weights = nullptr;
    const double2* eloc = nullptr;      // filled by the sampler when requested
};

// deep.cu: the layouts of a deep net that are derived from its device weights
int deep_derive(const rbmg_psi* psi);
// capi.cu: the energy gradient formed on the device, d_grad [P]; energy to value[2]
int ev_gradient_device(const rbmg_psi* psi, const rbmg_operator* op, rbmg_ensemble* ens, double2* d_grad,
                       double* value);
// angles_tc.cu: hidden angles from scratch on the tensor cores
bool rbm_tc_supported(int N, int Mpad);
size_t rbm_tc_pack_elems(int Mpad, int Kp);
int rbm_tc_kp(int N);
cudaError_t launch_rbm_tc_pack(int N, int M, int Mpad, const float2* W, __nv_bfloat16* out, cudaStream_t st);
cudaError_t launch_angles_tc(int count, int N, int Mpad, const uint64_t* spins, const float2* b,
                             const __nv_bfloat16* images, float4* theta, float2* re, float2* plain, int* error,
                             cudaStream_t st);
// density.cu: out = a - b elementwise
cudaError_t launch_sub(int count, const double2* a, const double2* b, double2* out, cudaStream_t st);
// density.cu: out [2^na] += w_s |eloc_s|^2 at the bin of the first na spins
cudaError_t launch_diag_density(int count, int enumerate, uint64_t enum_base, const uint64_t* spins, int nw,
                                const double* w, const double2* eloc, int na, double* out, cudaStream_t st);
}  // namespace rbmg

struct rbmg_operator {
    int S = 0, L = 0;
    std::vector<rbmg::cplx> coef;
    std::vector<int> types, idx;
    // compact form
    std::vector<int> ypow, nflip, flip_off, flip_sites, offdiag_slot;
    std::vector<uint64_t> zmask;
    int num_offdiag = 0;
    int max_site = -1;
    bool single_flips = false;   // every off-diagonal string flips one site, no two the same
    bool in_pairs = false;       // OpDev::in_pairs
    rbmg::DevBuf d_coef, d_coef32, d_site1, d_next1, d_ypow, d_zmask, d_nflip, d_flip_off, d_flip_sites, d_slot;
    rbmg::DevBuf d_offdiag;
    // per-site CSR of the off-diagonal slots whose string flips the site (E_k term)
    std::vector<int> site_ptr, site_slots;
    rbmg::DevBuf d_site_ptr, d_site_slots;
    int site_ptr_N = -1;
    rbmg::OpDev dev() const {
        return rbmg::OpDev{S,
                           d_coef.as<double2>(),
                           d_ypow.as<int>(),
                           d_zmask.as<uint64_t>(),
                           d_nflip.as<int>(),
                           d_flip_off.as<int>(),
                           d_flip_sites.as<int>(),
                           d_slot.as<int>(),
                           num_offdiag,
                           d_coef32.as<float2>(),
                           d_site1.as<int>(),
                           d_next1.as<int>(),
                           d_offdiag.as<int>(),
                           in_pairs ? 1 : 0};
    }
};

// per-site lists of the off-diagonal strings flipping each site, built (once per N) on the
// device for the E_k term (capi.cu)
int op_site_lists(rbmg_operator* op, int N);

struct rbmg_ensemble {
    int kind = 0;   // 0 MonteCarloLoop, 1 ExactSummation, 2 fixed sample set
    // MonteCarloLoop
    uint32_t num_samples = 0, num_sweeps = 1, num_therm = 0, num_chains = 1;
    uint64_t seed = 0;
    int total_z = 0, sector = 0;
    uint32_t fast_sweep_tries = 0;
    rbmg::DevBuf spins, rng_index, accepts, proposals;
    int spins_words = 0;
    std::vector<uint64_t> last_accepts, last_proposals;
    rbmg::HostBuf counts;   // the accept and proposal counts of a pass, on their way to the two above
    // ExactSummation
    uint32_t num_spins = 0;
    int exact_total_z = 0;
    std::vector<uint64_t> allowed;          // sector configurations
    rbmg::DevBuf d_allowed;                 // sector configurations; fixed sample set (kind 2)
    uint64_t fixed_count = 0;               // fixed sample set: number of configurations

    uint64_t num_steps() const;

    // a Monte-Carlo pass's counts: the copies enqueued; taken once the stream has been waited for
    cudaError_t counts_copy() {
        const size_t n = sizeof(unsigned long long) * num_chains;
        cudaError_t e = counts.ensure(2 * n);
        if (e == cudaSuccess) e = cudaMemcpyAsync(counts.p, accepts.p, n, cudaMemcpyDeviceToHost, rbmg::stream());
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(counts.as<char>() + n, proposals.p, n, cudaMemcpyDeviceToHost, rbmg::stream());
        return e;
    }
    void counts_take() {
        const unsigned long long* c = counts.as<unsigned long long>();
        last_accepts.assign(c, c + num_chains);
        last_proposals.assign(c + num_chains, c + 2 * static_cast<size_t>(num_chains));
    }
};

// walkers that persist on the device between calls (capi.cu); the learned-proposal
// steps (proposal.cu) keep their angles and logits in `learned`
struct rbmg_chain {
    int N = 0, nw = 0;
    uint32_t walkers = 0;
    uint64_t seed = 0;
    rbmg::DevBuf spins, rng_index, accepts, proposals;
    bool initialised = false;
    int learned_streams = 0;   // frozen learned steps on 1 to 4 streams; 0: automatic
    std::shared_ptr<void> learned;
};
