// Two persistent phases of one CTA an SM each, of any of the kernels: whether the second one's CTAs
// all start while the first one's wait.  No challenge is ever written, so a phase publishes its
// first round and waits until its limit or until it is told to return, whichever is first.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "bn254.cuh"
#include "kernels.cuh"

using namespace gkrgpu;

#define CK(x)                                                           \
    do {                                                                \
        const cudaError_t e_ = (x);                                     \
        if (e_ != cudaSuccess) {                                        \
            fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e_));    \
            exit(3);                                                    \
        }                                                               \
    } while (0)

constexpr unsigned long long kWaitNs = 400ull * 1000 * 1000;

// A phase from round 1 of n on tables of zeros, its mailbox, and what it publishes, in host memory.
// kind 0: M31 phase two, 1: M31 phase one, 2: BN254 phase two, 3: BN254 phase one.
struct Phase {
    int kind;
    uint32_t n, N, slot_words, words;  // of a mailbox slot; published in the first round
    cudaStream_t s = nullptr;
    uint32_t *host = nullptr, *dev = nullptr;
    PhaseArgs m = {};
    bn::PhaseArgsBn b = {};

    static constexpr uint32_t kMbox = 64, kOut = kMbox + 12 * kMboxRounds;
    bool bn254() const { return kind >= 2; }

    template <class T>
    static T* zeros(size_t count) {
        void* p = nullptr;
        CK(cudaMalloc(&p, count * sizeof(T)));
        CK(cudaMemset(p, 0, count * sizeof(T)));
        return static_cast<T*>(p);
    }
    template <class A>
    void common(A& a) const {
        a.k0 = 1;
        a.n = n;
        a.N = N;
        a.parity = 1;
        a.mbox = dev + kMbox;
        a.evals_out = dev + kOut;
        a.rows_out = dev + kOut + words;
        a.err = dev;
        a.wait_ns = kWaitNs;
    }
    Phase(int kind_, uint32_t n_, uint32_t sms) : kind(kind_), n(n_) {
        N = bn254() ? sms : 4 * sms;
        slot_words = bn254() ? bn::kDigitWords : 4;
        words = 3 * N * (bn254() ? bn::kDigitWords : 1);
        const size_t bytes = 4 * ((size_t)kOut + 2 * words), rows = (size_t)1 << n;
        void *h = nullptr, *d = nullptr;
        CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        CK(cudaHostAlloc(&h, bytes, cudaHostAllocMapped));
        memset(h, 0, bytes);
        CK(cudaHostGetDevicePointer(&d, h, 0));
        host = static_cast<uint32_t*>(h);
        dev = static_cast<uint32_t*>(d);
        if (bn254()) {
            common(b);
            for (uint32_t** t : {&b.fA, &b.fB, &b.hA, &b.hB}) *t = zeros<uint32_t>(rows * N * 8);
            b.s = zeros<bn::Fr>(rows);
            b.vx = zeros<uint32_t>((size_t)N * 8);
        } else {
            common(m);
            m.priv_stride = phase_priv_quads(rows);
            m.priv = zeros<uint4>(m.priv_stride * sms);
            m.fsrc[0] = zeros<uint32_t>(rows * N);
            m.hsrc[0] = zeros<uint32_t>(rows * N);
            m.s[0] = zeros<uint32_t>(rows);
            m.vx = zeros<uint32_t>(N);
            m.reps = m.tpr = 1;
        }
    }
    void launch() const { CK(bn254() ? bn::launch_phase(kind & 1, b, s) : launch_phase(kind & 1, m, s)); }
    bool published() const {
        const volatile uint32_t* out = host + kOut;
        for (uint32_t i = 0; i < words; i++)
            if (!(out[i] >> 31)) return false;
        return true;
    }
    bool expired() const { return *static_cast<const volatile uint32_t*>(host) != 0; }
    // Until the first round is out, or well past the limit of both phases.
    bool wait_published() const {
        const auto t0 = std::chrono::steady_clock::now();
        while (!published())
            if (std::chrono::steady_clock::now() - t0 > std::chrono::nanoseconds(3 * kWaitNs)) return false;
        return true;
    }
    void tell_to_return() const {
        volatile uint32_t* mbox = host + kMbox;
        for (uint32_t k = 0; k < kMboxRounds; k++) mbox[slot_words * (k + 1) - 1] = 1u;
    }
};

// phases_side_by_side kind n kind n: exits 0 when the second ran beside the first, 1 when not.
int main(int argc, char** argv) {
    if (argc != 5) return 2;
    int sms = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0));
    printf("%d and %d CTAs an SM\n", phase_ctas_per_sm(), bn::phase_ctas_per_sm());
    if (phase_ctas_per_sm() < 2 || bn::phase_ctas_per_sm() < 2) return 0;  // (none would be admitted)
    // nothing is allocated or cleared while a phase waits
    const Phase first(atoi(argv[1]), (uint32_t)atoi(argv[2]), (uint32_t)sms);
    const Phase second(atoi(argv[3]), (uint32_t)atoi(argv[4]), (uint32_t)sms);
    CK(cudaDeviceSynchronize());
    first.launch();
    const bool started = first.wait_published();
    second.launch();
    const bool both = started && second.wait_published() && !first.expired();
    first.tell_to_return();
    second.tell_to_return();
    CK(cudaDeviceSynchronize());
    printf("%s\n", both ? "side by side" : "one after the other");
    return both ? 0 : 1;
}
