// The verifiers of csrc/verifier.cuh on the host, for what they do with a proof's bytes: the device
// side is a stand-in that launches nothing (every gate sum and evaluation reads zero), and the
// array that the transcript is in has a guard zone behind it.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "bn254.cuh"
#include "fr_host.hpp"
#include "kernels.cuh"
#include "transcript.hpp"

using namespace gkrgpu;

namespace {

constexpr size_t kGuard = 1u << 20;
size_t g_overrun = 0;  // bytes of guard zones written

}  // namespace

void* operator new[](size_t n) {
    auto* p = static_cast<unsigned char*>(malloc(16 + n + kGuard));
    if (!p) throw std::bad_alloc();
    memcpy(p, &n, sizeof(n));
    memset(p + 16 + n, 0xa5, kGuard);
    return p + 16;
}
void operator delete[](void* v) noexcept {
    if (!v) return;
    auto* p = static_cast<unsigned char*>(v) - 16;
    size_t n;
    memcpy(&n, p, sizeof(n));
    for (size_t i = 0; i < kGuard; i++) g_overrun += p[16 + n + i] != 0xa5;
    free(p);
}
void operator delete[](void* v, size_t) noexcept { operator delete[](v); }

extern "C" {
cudaError_t CUDARTAPI cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFreeAsync(void* p, cudaStream_t) {
    free(p);
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
}

namespace {

void ck(cudaError_t, const char*) {}
size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct DevLayer {
    uint32_t nin = 0, nout = 0;
    uint64_t nmul = 0, nadd = 0;
    uint32_t *mo_off = nullptr, *ao_off = nullptr;
    uint4* mo_g = nullptr;
    uint2* ao_g = nullptr;
    const bn::Fr *mo_c = nullptr, *ao_c = nullptr;
};
struct gkrgpu_circuit {
    std::vector<DevLayer> layers;
    uint64_t in_rows(size_t l) const { return 1ull << layers[l].nin; }
};
struct gkrgpu_ctx {
    cudaMemPool_t pool = nullptr;
    int fs_hash = kFsSha256;
    uint32_t block = 256;
    Geo geo(uint32_t N, int) const { return Geo{N, 1, 256}; }
    uint32_t cta_budget(int) const { return 1; }
};
struct PinnedBuf {
    void* p = nullptr;
    std::vector<char> b;
    void ensure(size_t n, const char*) {
        b.assign(n, 0);
        p = b.data();
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p);
    }
};
// Copies and launches since the last wait are counted: none may be left when a call returns, as
// they read the caller's proof and write what the next call uses.
struct Lane {
    cudaStream_t stream = nullptr;
    std::vector<char> mapped;
    PinnedBuf h_cv;
    int launches = 0, in_flight = 0;
    void ensure_mapped(size_t, size_t extra) { mapped.assign(extra, 0); }
    char* extra_h() { return mapped.data(); }
    char* extra_d() { return mapped.data(); }
    template <class F>
    void launch(int, double, F&&) {
        launches++;
        in_flight++;
    }
    void copy(void*, const void*, size_t, cudaMemcpyKind, const char*) { in_flight++; }
    void sync() { in_flight = 0; }
    void resolve_events() {}
    void came_back(uint64_t) {}
};
EqArgs eq_args(int, const uint32_t (*)[32], const uint32_t (*)[32], uint32_t, uint32_t, uint32_t) { return EqArgs{}; }
bn::EqArgsBn eq_args_bn(const frh::Fr*, const frh::Fr*, const frh::Fr&, const frh::Fr&, uint32_t) { return bn::EqArgsBn{}; }
bn::GeoBn geo_bn(const gkrgpu_ctx&, uint32_t N, int) { return bn::GeoBn{N, 1, 256}; }

#include "verifier.cuh"

}  // namespace

// verifier_on_host field copies reps length nin nout [nin nout ...], layers from the input up:
// prints accepted, bytes written past the transcript, launches, and operations left in flight.
int main(int argc, char** argv) {
    if (argc < 7) return 2;
    const bool bn254 = atoi(argv[1]) != 0;
    const uint32_t N = (uint32_t)atoi(argv[2]);
    const int R = atoi(argv[3]);
    const uint64_t len = strtoull(argv[4], nullptr, 10);
    gkrgpu_circuit C;
    for (int i = 5; i + 1 < argc; i += 2) {
        C.layers.emplace_back();
        C.layers.back().nin = (uint32_t)atoi(argv[i]);
        C.layers.back().nout = (uint32_t)atoi(argv[i + 1]);
    }
    std::vector<uint8_t> proof(len, 7);
    std::vector<uint32_t> claims((size_t)R * N * 8, 0);
    gkrgpu_ctx ctx;
    Lane lane;
    bool ok;
    if (bn254)
        ok = BnVerifier(ctx, lane, C, N).run(0, proof.data(), len, claims.data());
    else
        ok = Verifier(ctx, lane, C, N, R).run(0, proof.data(), len, claims.data());
    printf("%d %zu %d %d\n", (int)ok, g_overrun, lane.launches, lane.in_flight);
    return 0;
}
