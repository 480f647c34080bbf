// Persistent sumcheck phases: the rounds of a phase whose tables are small, in one launch
// that waits on the device for the challenges the host derives between rounds.
//
// Reference counterpart: the round loop of sumcheck_prove_gkr_layer
// (include/LinearGKR/sumcheck.hpp:72-103) over receive_challenge and poly_eval_at
// (include/LinearGKR/sumcheck_helper.hpp:68-133), and with k0 = 0 in phase one
// _prepare_g_x_vals (sumcheck_helper.hpp:172-231) as well.
//
// What bounds it: the serial chain challenge -> fold -> sums -> host -> challenge.  A round
// launched by itself takes 14-16 us on small tables (the launch, an atomic reduction across
// CTAs with a last-CTA finisher, system-scope fences), of which the arithmetic is under 2.
// So the copies are split over CTAs and nothing else is: each CTA owns 4 tpr copies and every
// row of them, its sums stay inside the CTA, and no CTA waits on another.  The repetitions
// are split over the CTA's warps (4 warps each), which keeps a thread at one repetition's
// sums.  Small tables sit in shared memory, larger ones go through L1/L2.
//
// Host traffic without fences or counters: an M31 value leaves bit 31 free, so every word
// published to the host carries the round's parity there, and the host takes a word when its
// parity is the round's; likewise the host's challenges carry bit 31 in a 16-byte mailbox slot
// per round (r_0, r_1, r_2, abort) that it clears before the launch, read in one load.
#include <atomic>

#include "kernels.cuh"
#include "m31.cuh"

namespace gkrgpu {

namespace {

constexpr uint32_t kWarps = 4;                 // warps per repetition
constexpr uint32_t kRepThreads = 32 * kWarps;  // threads per repetition
constexpr uint32_t kSmemRows = 256;            // rows x tpr of a table kept in shared memory
constexpr uint32_t kSpins = 256;               // mailbox polls before sleeping between them

__device__ __forceinline__ uint32_t comp(const uint4& v, int l) { return l == 0 ? v.x : l == 1 ? v.y : l == 2 ? v.z : v.w; }
__device__ __forceinline__ void mad64(uint64_t& acc, uint32_t a, uint32_t b) { acc += (uint64_t)a * b; }
// x mod p, partly reduced: 2^32 == 2, so lo + 2 hi < 3 2^32; four more products of canonical
// values keep a 64-bit sum below 2^64 (4 (p - 1)^2 = 2^64 - 2^35 + 16).
__device__ __forceinline__ uint64_t fold64(uint64_t x) { return (uint64_t)(uint32_t)x + 2ull * (uint32_t)(x >> 32); }
__device__ __forceinline__ uint32_t reduce64(uint64_t x) {
    x = (x & m31::P) + (x >> 31);
    x = (x & m31::P) + (x >> 31);
    const uint32_t s = (uint32_t)x;
    return m31::umin(s, s - m31::P);
}
__device__ __forceinline__ uint4 lerp4(const uint4& a, const uint4& b, const m31::Lerp& c) {
    return make_uint4(m31::lerp(a.x, b.x, c), m31::lerp(a.y, b.y, c), m31::lerp(a.z, b.z, c), m31::lerp(a.w, b.w, c));
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint4 ld_mailbox(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

// A per-copy table as one thread sees it: row r at p[r * stride] (four copies).
struct Rows {
    uint4* p;
    size_t stride;
    __device__ __forceinline__ uint4& operator[](uint32_t r) const { return p[(size_t)r * stride]; }
};

// p0 += f0 h0, p1 += f1 h1, p2raw += (f0 + f1)(h0 + h1), unreduced in 64 bits.
__device__ __forceinline__ void accum(uint64_t (&acc)[3][4], const uint4& f0, const uint4& f1, const uint4& h0,
                                      const uint4& h1) {
#pragma unroll
    for (int l = 0; l < 4; l++) {
        mad64(acc[0][l], comp(f0, l), comp(h0, l));
        mad64(acc[1][l], comp(f1, l), comp(h1, l));
        mad64(acc[2][l], m31::add(comp(f0, l), comp(f1, l)), m31::add(comp(h0, l), comp(h1, l)));
    }
}

// hg_j of input row x for four copies: a_j[x] + sum over its mul gates (x, y, k) of
// v[y] w_j[k]; gates in pairs, so that two gathers are in flight.
__device__ __forceinline__ uint4 build_h(const PhaseArgs& a, uint32_t j, uint32_t x, const uint4* v, size_t stride) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a.w4) + j;
    uint32_t k = __ldg(a.mx_off + x);
    const uint32_t k1 = __ldg(a.mx_off + x + 1);
    const uint32_t a0 = __ldg(reinterpret_cast<const uint32_t*>(a.a4 + x) + j);
    if (k == k1) return make_uint4(a0, a0, a0, a0);
    uint64_t s[4] = {a0, a0, a0, a0};
    for (; k + 1 < k1; k += 2) {
        const uint32_t y0 = __ldg(&a.mx_g[k].x), y1 = __ldg(&a.mx_g[k + 1].x);
        const uint32_t w0 = __ldg(w + 4 * (size_t)k), w1 = __ldg(w + 4 * (size_t)k + 4);
        const uint4 v0 = __ldg(v + y0 * stride), v1 = __ldg(v + y1 * stride);
#pragma unroll
        for (int l = 0; l < 4; l++) {
            mad64(s[l], comp(v0, l), w0);
            mad64(s[l], comp(v1, l), w1);
            s[l] = fold64(s[l]);
        }
    }
    if (k < k1) {
        const uint32_t y0 = __ldg(&a.mx_g[k].x), w0 = __ldg(w + 4 * (size_t)k);
        const uint4 v0 = __ldg(v + y0 * stride);
#pragma unroll
        for (int l = 0; l < 4; l++) mad64(s[l], comp(v0, l), w0);
    }
    return make_uint4(reduce64(s[0]), reduce64(s[1]), reduce64(s[2]), reduce64(s[3]));
}

template <bool LANE_HG>
__global__ void __launch_bounds__(3 * kRepThreads, 2) k_phase(PhaseArgs a) {
    extern __shared__ uint4 psm[];
    __shared__ uint32_t rch[3];
    __shared__ int stop;
    const uint32_t R = a.reps, tid = threadIdx.x, tpr = a.tpr, N = a.N;
    const uint32_t warp = tid >> 5, j = warp / kWarps, t = tid - j * kRepThreads;
    const uint32_t q = t & (tpr - 1), slot = t / tpr, nslots = kRepThreads / tpr;
    const uint32_t quad = blockIdx.x * tpr + q;  // this thread's four copies: 4 quad ..
    const bool active = 4 * quad < N;
    const size_t gs = N / 4;  // row stride of a table in memory
    // shared memory: two buffers of small tables (f, then hg in phase one), phase two's scalar
    // tables (two buffers), the warps' partial sums
    constexpr uint32_t kTabs = LANE_HG ? 6 : 3;
    const uint32_t kf = a.k0 ? a.k0 : 1;  // the first round that folds
    const uint32_t S1 = 1u << (a.n - kf);
    uint32_t* const sbuf = reinterpret_cast<uint32_t*>(psm + 2 * kTabs * kSmemRows);
    uint32_t* const part = sbuf + (LANE_HG ? 0 : 3 * (S1 + S1 / 2));
    // the table round k leaves (2^(n-k) rows): which = 0 f, 1 hg of this thread's repetition
    auto table = [&](uint32_t k, uint32_t which) -> Rows {
        const uint32_t rows = 1u << (a.n - k);
        if (rows * tpr <= kSmemRows)
            return Rows{psm + ((k & 1) * kTabs + which * 3 + j) * kSmemRows + q, tpr};
        uint32_t* b;
        if (which == 0) b = (k & 1) ? (j == 0 ? a.fA[0] : j == 1 ? a.fA[1] : a.fA[2]) : (j == 0 ? a.fB[0] : j == 1 ? a.fB[1] : a.fB[2]);
        else b = (k & 1) ? (j == 0 ? a.hA[0] : j == 1 ? a.hA[1] : a.hA[2]) : (j == 0 ? a.hB[0] : j == 1 ? a.hB[1] : a.hB[2]);
        return Rows{reinterpret_cast<uint4*>(b) + quad, gs};
    };
    // the stored tables the first round reads are in memory whatever their size
    auto stored = [&](uint32_t which) -> Rows {
        uint32_t* b;
        if (which == 0) b = (a.k0 & 1) ? (j == 0 ? a.fB[0] : j == 1 ? a.fB[1] : a.fB[2]) : (j == 0 ? a.fA[0] : j == 1 ? a.fA[1] : a.fA[2]);
        else b = (a.k0 & 1) ? (j == 0 ? a.hB[0] : j == 1 ? a.hB[1] : a.hB[2]) : (j == 0 ? a.hA[0] : j == 1 ? a.hA[1] : a.hA[2]);
        return Rows{reinterpret_cast<uint4*>(b) + quad, gs};
    };
    const uint4* const v = reinterpret_cast<const uint4*>(a.v) + quad;
    uint4* const h0t = reinterpret_cast<uint4*>(j == 0 ? a.h0[0] : j == 1 ? a.h0[1] : a.h0[2]) + quad;
    const uint32_t* const s0t = j == 0 ? a.s[0] : j == 1 ? a.s[1] : a.s[2];
    // the finisher's (repetition, copy) of this thread and phase two's factor v(rx) there
    const uint32_t fj = tid / (4 * tpr), fl = tid - fj * 4 * tpr, flane = blockIdx.x * 4 * tpr + fl;
    const bool finisher = fj < R && flane < N;
    uint32_t xv = 0;
    if (!LANE_HG && finisher) xv = __ldcv(a.vx + (size_t)fj * N + flane);
    if (tid == 0) stop = 0;

    for (uint32_t k = a.k0; k < a.n; k++) {
        if (k == a.k0) {
            if (tid < 3) rch[tid] = tid == 0 ? a.r_first[0] : tid == 1 ? a.r_first[1] : a.r_first[2];
        } else if (tid == 0) {
            const uint32_t* box = a.mbox + 4 * (k - 1);
            uint64_t t0 = 0;
            for (uint32_t it = 0;; it++) {
                const uint4 m = ld_mailbox(box);
                uint32_t ok = m.x;
                if (R > 1) ok &= m.y;
                if (R > 2) ok &= m.z;
                if (ok >> 31) {
                    rch[0] = m.x & m31::P;
                    rch[1] = m.y & m31::P;
                    rch[2] = m.z & m31::P;
                    break;
                }
                if (m.w) {
                    stop = 1;
                    break;
                }
                if (it < kSpins) continue;
                const uint64_t now = global_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > a.wait_ns) {
                    *reinterpret_cast<volatile unsigned int*>(a.err) = 1u;
                    stop = 1;
                    break;
                }
                __nanosleep(100);
            }
        }
        __syncthreads();  // the challenges, and the previous round's tables, are visible
        if (stop) return;
        const uint32_t npairs = 1u << (a.n - k - 1);
        const m31::Lerp c = m31::lerp_at(rch[j]);
        uint64_t acc[3][4] = {};
        uint32_t since = 0;
        if (active) {
            if (k == 0) {
                for (uint32_t i = slot; i < npairs; i += nslots) {
                    const uint4 f0 = __ldg(v + (size_t)(2 * i) * gs), f1 = __ldg(v + (size_t)(2 * i + 1) * gs);
                    uint4 h0, h1;
                    if (LANE_HG) {
                        h0 = build_h(a, j, 2 * i, v, gs);
                        h1 = build_h(a, j, 2 * i + 1, v, gs);
                        h0t[(size_t)(2 * i) * gs] = h0;
                        h0t[(size_t)(2 * i + 1) * gs] = h1;
                    } else {
                        const uint2 s = __ldg(reinterpret_cast<const uint2*>(s0t) + i);
                        h0 = make_uint4(s.x, s.x, s.x, s.x);
                        h1 = make_uint4(s.y, s.y, s.y, s.y);
                    }
                    accum(acc, f0, f1, h0, h1);
                    if ((++since & 3) == 0)
#pragma unroll
                        for (int l = 0; l < 4; l++)
#pragma unroll
                            for (int e = 0; e < 3; e++) acc[e][l] = fold64(acc[e][l]);
                }
            } else {
                Rows fs, hs = {};
                if (k == a.k0) fs = stored(0);
                else if (k == 1) fs = Rows{const_cast<uint4*>(v), gs};
                else fs = table(k - 1, 0);
                const Rows fd = table(k, 0);
                Rows hd = {};
                const uint32_t* ssrc = nullptr;
                uint32_t* sdst = nullptr;
                if (LANE_HG) {
                    if (k == a.k0) hs = stored(1);
                    else if (k == 1) hs = Rows{h0t, gs};
                    else hs = table(k - 1, 1);
                    hd = table(k, 1);
                } else {
                    ssrc = k == kf ? s0t : sbuf + ((k - kf) & 1 ? 0 : 3 * S1) + j * ((k - kf) & 1 ? S1 : S1 / 2);
                    sdst = sbuf + ((k - kf) & 1 ? 3 * S1 : 0) + j * ((k - kf) & 1 ? S1 / 2 : S1);
                }
                for (uint32_t i = slot; i < npairs; i += nslots) {
                    const uint4 x0 = fs[4 * i], x1 = fs[4 * i + 1], x2 = fs[4 * i + 2], x3 = fs[4 * i + 3];
                    uint4 h0, h1;
                    if (LANE_HG) {
                        const uint4 y0 = hs[4 * i], y1 = hs[4 * i + 1], y2 = hs[4 * i + 2], y3 = hs[4 * i + 3];
                        h0 = lerp4(y0, y1, c);
                        h1 = lerp4(y2, y3, c);
                        hd[2 * i] = h0;
                        hd[2 * i + 1] = h1;
                    } else {
                        const uint4 s = reinterpret_cast<const uint4*>(ssrc)[i];
                        const uint32_t s0 = m31::lerp(s.x, s.y, c), s1 = m31::lerp(s.z, s.w, c);
                        if (q == 0) reinterpret_cast<uint2*>(sdst)[i] = make_uint2(s0, s1);
                        h0 = make_uint4(s0, s0, s0, s0);
                        h1 = make_uint4(s1, s1, s1, s1);
                    }
                    const uint4 f0 = lerp4(x0, x1, c), f1 = lerp4(x2, x3, c);
                    fd[2 * i] = f0;
                    fd[2 * i + 1] = f1;
                    accum(acc, f0, f1, h0, h1);
                    if ((++since & 3) == 0)
#pragma unroll
                        for (int l = 0; l < 4; l++)
#pragma unroll
                            for (int e = 0; e < 3; e++) acc[e][l] = fold64(acc[e][l]);
                }
            }
        }
        // sums over the repetition's threads with the same q: shuffles within a warp, then the
        // warps that had pairs (all of them when npairs tpr covers the repetition's threads)
        const uint32_t nw = npairs * tpr >= kRepThreads ? kWarps : (npairs * tpr + 31) / 32;
        const uint32_t w = warp - j * kWarps;
        if (w < nw) {
            uint32_t x[12];
#pragma unroll
            for (int e = 0; e < 3; e++)
#pragma unroll
                for (int l = 0; l < 4; l++) x[4 * e + l] = reduce64(acc[e][l]);
            for (uint32_t off = 16; off >= tpr; off >>= 1)
#pragma unroll
                for (int e = 0; e < 12; e++) x[e] = m31::add(x[e], __shfl_xor_sync(0xffffffffu, x[e], off));
            if ((tid & 31) < tpr)
#pragma unroll
                for (int e = 0; e < 3; e++)
#pragma unroll
                    for (int l = 0; l < 4; l++) part[((j * kWarps + w) * 3 + e) * 4 * tpr + 4 * q + l] = x[4 * e + l];
        }
        __syncthreads();
        if (finisher) {
            uint32_t p0 = 0, p1 = 0, p2 = 0;
            for (uint32_t i = 0; i < nw; i++) {
                const uint32_t* s = part + (fj * kWarps + i) * 3 * 4 * tpr + fl;
                p0 = m31::add(p0, s[0]);
                p1 = m31::add(p1, s[4 * tpr]);
                p2 = m31::add(p2, s[8 * tpr]);
            }
            p2 = m31::eval_at_two(p0, p1, p2);
            if (!LANE_HG) {
                p0 = m31::mul(p0, xv);
                p1 = m31::mul(p1, xv);
                p2 = m31::mul(p2, xv);
            }
            const uint32_t par = (a.parity ^ (k - a.k0)) << 31;
            volatile uint32_t* out = a.evals_out + (size_t)(3 * fj) * N + flane;
            out[0] = p0 | par;
            out[N] = p1 | par;
            out[2 * (size_t)N] = p2 | par;
            if (k + 1 == a.n) {
                // rows 0 and 1 of the last folded f table (the layer input when it has no fold)
                uint32_t r0, r1;
                if (k == 0) {
                    r0 = __ldg(a.v + flane);
                    r1 = __ldg(a.v + N + flane);
                } else {  // two rows are always in shared memory
                    const uint32_t* s = reinterpret_cast<const uint32_t*>(psm + ((k & 1) * kTabs + fj) * kSmemRows);
                    r0 = s[fl];
                    r1 = s[4 * tpr + fl];
                }
                volatile uint32_t* ro = a.rows_out + (size_t)(2 * fj) * N + flane;
                ro[0] = r0 | (a.rows_parity << 31);
                ro[N] = r1 | (a.rows_parity << 31);
            }
        }
    }
}

}  // namespace

// Copies per CTA: the smallest power of two of quads (4 copies) that needs at most max_ctas
// CTAs; 0 where 32 quads are not enough.  Few copies per CTA give a round the most SMs.
uint32_t phase_tpr(uint32_t N, uint32_t max_ctas) {
    for (uint32_t tpr = 1; tpr <= 32; tpr *= 2)
        if ((N / 4 + tpr - 1) / tpr <= max_ctas) return tpr;
    return 0;
}
uint32_t phase_ctas(uint32_t N, uint32_t tpr) { return (N / 4 + tpr - 1) / tpr; }

cudaError_t launch_phase(bool lane_hg, const PhaseArgs& a, cudaStream_t s) {
    if (a.reps < 1 || a.reps > 3 || a.k0 >= a.n || a.n - a.k0 > kMboxRounds || a.N % 4) return cudaErrorInvalidValue;
    if (a.tpr < 1 || a.tpr > 32 || (a.tpr & (a.tpr - 1))) return cudaErrorInvalidValue;
    // rows of the first round's source tables; with k0 = 0 the layer input itself
    const uint64_t rows = 1ull << (a.n - (a.k0 ? a.k0 - 1 : 0));
    if (rows * a.tpr > kPhaseItems) return cudaErrorInvalidValue;
    if (a.k0 == 0 && (!a.v || (lane_hg && (!a.h0[0] || !a.mx_off || !a.a4 || !a.w4)))) return cudaErrorInvalidValue;
    if (!lane_hg && (!a.vx || !a.s[0])) return cudaErrorInvalidValue;
    static std::atomic<uint64_t> opted{0};  // one bit per device: shared memory above 48 KiB
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(opted.load(std::memory_order_relaxed) & bit)) {
        cudaFuncSetAttribute(k_phase<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        cudaFuncSetAttribute(k_phase<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        opted.fetch_or(bit);
    }
    const uint32_t kf = a.k0 ? a.k0 : 1, S1 = a.n >= kf ? 1u << (a.n - kf) : 1u;
    const size_t smem = 2 * (lane_hg ? 6 : 3) * (size_t)kSmemRows * 16 + (lane_hg ? 0 : 4 * 3 * (size_t)(S1 + S1 / 2)) +
                        4 * (size_t)a.reps * kWarps * 3 * 4 * a.tpr;
    const dim3 grid(phase_ctas(a.N, a.tpr)), block(a.reps * kRepThreads);
    if (lane_hg)
        k_phase<true><<<grid, block, smem, s>>>(a);
    else
        k_phase<false><<<grid, block, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace gkrgpu
