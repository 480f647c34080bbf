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
// sums.
//
// A CTA's tables are its own, [row][4 tpr copies], with the rows r of equal r mod 4 side by
// side: a round reads rows 4i .. 4i+3 in four contiguous streams (with the rows of the
// caller's tables, N copies apart, every lane of a load touches another line, which made the
// first two rounds of 2^10 rows 18 us of 63).  Tables of up to 1024 words are in shared memory
// and taken one copy a thread, which leaves a quarter of the instructions on the chain of a
// late round (3400 clocks with four copies a thread).
//
// Host traffic without fences or counters: an M31 value leaves bit 31 free, so every word
// published to the host carries the round's parity there, and the host takes a word when its
// parity is the round's; likewise the host's challenges carry bit 31 in a 16-byte mailbox slot
// per round (r_0, r_1, r_2, abort) that it clears before the launch, read in one load.  A
// word there and one back take 1.47 us, two turns of polling; loads of the slot in flight
// together do not shorten that (they come back one after another, 1400 clocks apart).
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
// (as one instruction: the compiler's own choice for acc += a * b with foldings between ran at
// 10.5 products per clock and SM, this at 17.5)
__device__ __forceinline__ void mad64(uint64_t& acc, uint32_t a, uint32_t b) {
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}
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
// Rows x[0], x[re], x[2 re], x[3 re] folded twice.
__device__ __forceinline__ uint4 lerp4(const uint4* x, size_t re, const m31::Lerp2& c) {
    const uint4 a = x[0], b = x[re], d = x[2 * re], e = x[3 * re];
    return make_uint4(m31::lerp2(a.x, b.x, d.x, e.x, c), m31::lerp2(a.y, b.y, d.y, e.y, c),
                      m31::lerp2(a.z, b.z, d.z, e.z, c), m31::lerp2(a.w, b.w, d.w, e.w, c));
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

// Place of row r in a table of `rows` rows (a power of two): rows of equal r mod 4 side by side.
__device__ __forceinline__ uint32_t place(uint32_t rows, uint32_t r) {
    return rows >= 4 ? (r & 3) * (rows >> 2) + (r >> 2) : r;
}

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

// Waits for the challenges of a round in its mailbox slot: 0 they are in rch, 1 abort, 2 the
// limit passed.
__device__ __forceinline__ int wait_challenge(const uint32_t* box, uint32_t R, unsigned long long wait_ns, uint32_t* rch) {
    uint64_t t0 = 0;
    for (uint32_t it = 0;; it++) {
        const uint4 m = ld_mailbox(box);
        if ((m.x & (R > 1 ? m.y : m.x) & (R > 2 ? m.z : m.x)) >> 31) {
            rch[0] = m.x & m31::P;
            rch[1] = m.y & m31::P;
            rch[2] = m.z & m31::P;
            return 0;
        }
        if (m.w) return 1;
        if (it < kSpins) continue;
        const uint64_t now = global_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > wait_ns) return 2;
        __nanosleep(100);
    }
}

// TWO: the first round folds the caller's tables twice (its own instance: the copies of that
// round's body in one cost the rounds of every phase spilled registers).
template <bool LANE_HG, bool TWO>
__global__ void __launch_bounds__(3 * kRepThreads, 2) k_phase(PhaseArgs a) {
    extern __shared__ uint4 psm[];
    __shared__ uint32_t rch[3];
    __shared__ int stop;
    const uint32_t R = a.reps, tid = threadIdx.x, tpr = a.tpr, N = a.N, L = 4 * tpr;
    const uint32_t warp = tid >> 5, j = warp / kWarps, w = warp - j * kWarps, t = tid - j * kRepThreads;
    const uint32_t q = t & (tpr - 1), slot = t / tpr, nslots = kRepThreads / tpr;
    const uint32_t quad = blockIdx.x * tpr + q;  // this thread's four copies: 4 quad ..
    const bool active = 4 * quad < N;
    // the CTA's tables in memory: the layer input and hg_0 of each repetition (k0 = 0), then
    // two buffers of up to six tables; the first folding round kf leaves S1 rows
    const uint32_t kf = a.k0 ? a.k0 : 1, S1 = 1u << (a.n - kf), I = 1u << a.n;
    uint4* const mine = a.priv + (size_t)blockIdx.x * a.priv_stride;
    uint4* const folded = mine + (a.k0 ? 0u : (1 + 3) * I * tpr);
    // shared memory: two buffers of small tables (f, then hg in phase one), phase two's scalar
    // tables (two buffers), partial sums
    constexpr uint32_t kTabs = LANE_HG ? 6 : 3;
    uint32_t* const sbuf = reinterpret_cast<uint32_t*>(psm + 2 * kTabs * kSmemRows);
    uint32_t* const part = sbuf + (LANE_HG ? 0 : 3 * (S1 + S1 / 2));
    // the table round k leaves (2^(n-k) rows): which = 0 f, 1 hg of this thread's repetition
    auto in_smem = [&](uint32_t k) { return (tpr << (a.n - k)) <= kSmemRows; };
    auto table = [&](uint32_t k, uint32_t which) -> uint4* {
        if (in_smem(k)) return psm + ((k & 1) * kTabs + which * 3 + j) * kSmemRows;
        const uint32_t odd = (k - kf) & 1;
        return folded + ((odd ? 6 * S1 : 0) + (which * 3 + j) * (odd ? S1 / 2 : S1)) * tpr;
    };
    const uint32_t* const s0t = j == 0 ? a.s[0] : j == 1 ? a.s[1] : a.s[2];
    // the first 4 tpr threads of a repetition finish its copies; phase two's factor v(rx) there
    const uint32_t flane = blockIdx.x * L + t;
    const bool finisher = t < L && flane < N;
    uint32_t xv = 0;
    if (!LANE_HG && finisher) xv = __ldcv(a.vx + (size_t)j * N + flane);
    if (tid == 0) stop = 0;

    for (uint32_t k = a.k0; k < a.n; k++) {
        if (k == a.k0) {
            if (tid < 3) rch[tid] = tid == 0 ? a.r_first[0] : tid == 1 ? a.r_first[1] : a.r_first[2];
        } else if (tid == 0) {
            const int got = wait_challenge(a.mbox + 4 * (k - 1), R, a.wait_ns, rch);
            if (got == 2) *reinterpret_cast<volatile unsigned int*>(a.err) = 1u;
            if (got) stop = 1;
        }
        __syncthreads();  // the challenges, and the previous round's tables, are visible
        if (stop) return;
        const uint32_t npairs = 1u << (a.n - k - 1), out_rows = 2 * npairs;
        const m31::Lerp c = m31::lerp_at(rch[j]);
        // phase two's scalar tables: read from memory by the first round that folds them
        const bool odd = (k - kf) & 1;
        const uint32_t* ssrc = k <= kf ? s0t : (odd ? sbuf + j * S1 : sbuf + 3 * S1 + j * (S1 / 2));
        uint32_t* sdst = odd ? sbuf + 3 * S1 + j * (S1 / 2) : sbuf + j * S1;
        uint32_t ns;  // partial sums per copy and repetition
        bool across;  // a finisher reads what another warp wrote (the same for the whole CTA)
        if (k > kf && in_smem(k - 1)) {
            // one copy a thread: pair idx / L, copy idx % L; at most two pairs a thread
            const uint32_t* fs = reinterpret_cast<const uint32_t*>(table(k - 1, 0));
            uint32_t* fd = reinterpret_cast<uint32_t*>(table(k, 0));
            const uint32_t* hs = LANE_HG ? reinterpret_cast<const uint32_t*>(table(k - 1, 1)) : nullptr;
            uint32_t* hd = LANE_HG ? reinterpret_cast<uint32_t*>(table(k, 1)) : nullptr;
            const uint32_t items = npairs * L;
            uint64_t acc[3] = {0ull, 0ull, 0ull};
            for (uint32_t idx = t; idx < items; idx += kRepThreads) {
                const uint32_t i = idx / L, lane = idx & (L - 1);
                const uint32_t f0 = m31::lerp(fs[idx], fs[items + idx], c);
                const uint32_t f1 = m31::lerp(fs[2 * items + idx], fs[3 * items + idx], c);
                const uint32_t o0 = place(out_rows, 2 * i) * L + lane, o1 = place(out_rows, 2 * i + 1) * L + lane;
                uint32_t h0, h1;
                if (LANE_HG) {
                    h0 = m31::lerp(hs[idx], hs[items + idx], c);
                    h1 = m31::lerp(hs[2 * items + idx], hs[3 * items + idx], c);
                    hd[o0] = h0;
                    hd[o1] = h1;
                } else {
                    const uint4 s = reinterpret_cast<const uint4*>(ssrc)[i];
                    h0 = m31::lerp(s.x, s.y, c);
                    h1 = m31::lerp(s.z, s.w, c);
                    if (lane == 0) reinterpret_cast<uint2*>(sdst)[i] = make_uint2(h0, h1);
                }
                fd[o0] = f0;
                fd[o1] = f1;
                mad64(acc[0], f0, h0);
                mad64(acc[1], f1, h1);
                mad64(acc[2], m31::add(f0, f1), m31::add(h0, h1));
            }
            // threads of one copy: within a warp when a pair's copies fit in one
            const uint32_t used = items < kRepThreads ? items : kRepThreads;
            ns = L <= 32 ? (used + 31) / 32 : (used + L - 1) / L;
            across = ns > 1;  // (one sum: the finisher's own, or its warp's)
            if (32 * w < used) {
                uint32_t x[3];
#pragma unroll
                for (int e = 0; e < 3; e++) x[e] = reduce64(acc[e]);
                for (uint32_t off = 16; off >= L; off >>= 1)
#pragma unroll
                    for (int e = 0; e < 3; e++) x[e] = m31::add(x[e], __shfl_xor_sync(0xffffffffu, x[e], off));
                const uint32_t sl = L <= 32 ? w : t / L, lane = t & (L - 1);
                if (L > 32 || (tid & 31) < L)
#pragma unroll
                    for (int e = 0; e < 3; e++) part[((j * kWarps + sl) * 3 + e) * L + lane] = x[e];
            }
        } else {
            uint64_t acc[3][4] = {};
            uint32_t since = 0;
            auto tidy = [&] {
                if ((++since & 3) == 0)
#pragma unroll
                    for (int l = 0; l < 4; l++)
#pragma unroll
                        for (int e = 0; e < 3; e++) acc[e][l] = fold64(acc[e][l]);
            };
            if (active && k == 0) {
                const uint4 *fs = mine + q, *hs = mine + (1 + j) * I * tpr + q;
                for (uint32_t i = slot; i < npairs; i += nslots) {
                    const uint32_t o0 = place(out_rows, 2 * i) * tpr, o1 = place(out_rows, 2 * i + 1) * tpr;
                    uint4 h0, h1;
                    if (LANE_HG) {
                        h0 = hs[o0];
                        h1 = hs[o1];
                    } else {
                        const uint2 s = __ldg(reinterpret_cast<const uint2*>(s0t) + i);
                        h0 = make_uint4(s.x, s.x, s.x, s.x);
                        h1 = make_uint4(s.y, s.y, s.y, s.y);
                    }
                    accum(acc, fs[o0], fs[o1], h0, h1);
                    tidy();
                }
            } else if (active) {
                // the first round reads the caller's tables (row r at r N + copy) when k0 > 0
                const bool given = k == a.k0;
                const uint4 *fs, *hs = nullptr;
                if (given) {
                    fs = reinterpret_cast<const uint4*>(j == 0 ? a.fsrc[0] : j == 1 ? a.fsrc[1] : a.fsrc[2]) + quad;
                    if (LANE_HG) hs = reinterpret_cast<const uint4*>(j == 0 ? a.hsrc[0] : j == 1 ? a.hsrc[1] : a.hsrc[2]) + quad;
                } else {
                    fs = (k == 1 ? mine : table(k - 1, 0)) + q;
                    if (LANE_HG) hs = (k == 1 ? mine + (1 + j) * I * tpr : table(k - 1, 1)) + q;
                }
                // row 4i + e: at 4i + e of the caller's tables, at e rows / 4 + i of the CTA's
                const size_t step = given ? N / 4 : tpr, ri = given ? (TWO ? 8 : 4) * step : step;
                const size_t re = given ? step : (size_t)npairs * step;
                uint4* fd = table(k, 0) + q;
                uint4* hd = LANE_HG ? table(k, 1) + q : nullptr;
                if (TWO && given) {
                    const m31::Lerp2 c01 =
                        m31::lerp2_at(j == 0 ? a.r_before[0] : j == 1 ? a.r_before[1] : a.r_before[2], rch[j]);
                    for (uint32_t i = slot; i < npairs; i += nslots) {
                        const uint4* x = fs + i * ri;
                        const uint32_t o0 = place(out_rows, 2 * i) * tpr, o1 = place(out_rows, 2 * i + 1) * tpr;
                        uint4 h0, h1;
                        if (LANE_HG) {
                            const uint4* y = hs + i * ri;
                            h0 = lerp4(y, re, c01);
                            h1 = lerp4(y + 4 * re, re, c01);
                            hd[o0] = h0;
                            hd[o1] = h1;
                        } else {
                            const uint4 sa = reinterpret_cast<const uint4*>(ssrc)[2 * i];
                            const uint4 sb = reinterpret_cast<const uint4*>(ssrc)[2 * i + 1];
                            const uint32_t s0 = m31::lerp2(sa.x, sa.y, sa.z, sa.w, c01);
                            const uint32_t s1 = m31::lerp2(sb.x, sb.y, sb.z, sb.w, c01);
                            if (q == 0) reinterpret_cast<uint2*>(sdst)[i] = make_uint2(s0, s1);
                            h0 = make_uint4(s0, s0, s0, s0);
                            h1 = make_uint4(s1, s1, s1, s1);
                        }
                        const uint4 f0 = lerp4(x, re, c01), f1 = lerp4(x + 4 * re, re, c01);
                        fd[o0] = f0;
                        fd[o1] = f1;
                        accum(acc, f0, f1, h0, h1);
                        tidy();
                    }
                }
                for (uint32_t i = TWO && given ? npairs : slot; i < npairs; i += nslots) {
                    const uint4* x = fs + i * ri;
                    const uint4 x0 = x[0], x1 = x[re], x2 = x[2 * re], x3 = x[3 * re];
                    const uint32_t o0 = place(out_rows, 2 * i) * tpr, o1 = place(out_rows, 2 * i + 1) * tpr;
                    uint4 h0, h1;
                    if (LANE_HG) {
                        const uint4* y = hs + i * ri;
                        const uint4 y0 = y[0], y1 = y[re], y2 = y[2 * re], y3 = y[3 * re];
                        h0 = lerp4(y0, y1, c);
                        h1 = lerp4(y2, y3, c);
                        hd[o0] = h0;
                        hd[o1] = h1;
                    } else {
                        const uint4 s = reinterpret_cast<const uint4*>(ssrc)[i];
                        const uint32_t s0 = m31::lerp(s.x, s.y, c), s1 = m31::lerp(s.z, s.w, c);
                        if (q == 0) reinterpret_cast<uint2*>(sdst)[i] = make_uint2(s0, s1);
                        h0 = make_uint4(s0, s0, s0, s0);
                        h1 = make_uint4(s1, s1, s1, s1);
                    }
                    const uint4 f0 = lerp4(x0, x1, c), f1 = lerp4(x2, x3, c);
                    fd[o0] = f0;
                    fd[o1] = f1;
                    accum(acc, f0, f1, h0, h1);
                    tidy();
                }
            }
            // sums over the repetition's threads with the same q: shuffles within a warp, then
            // the warps that had pairs
            const uint32_t used = npairs * tpr < kRepThreads ? npairs * tpr : kRepThreads;
            ns = (used + 31) / 32;
            across = ns > 1 || L > 32;  // warp 0 has the sums and rows of all the CTA's copies
            if (w < ns) {
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
                        for (int l = 0; l < 4; l++) part[((j * kWarps + w) * 3 + e) * L + 4 * q + l] = x[4 * e + l];
            }
        }
        if (across) __syncthreads();
        else __syncwarp();
        if (finisher) {
            uint32_t p0 = 0, p1 = 0, p2 = 0;
            for (uint32_t i = 0; i < ns; i++) {
                const uint32_t* s = part + (j * kWarps + i) * 3 * L + t;
                p0 = m31::add(p0, s[0]);
                p1 = m31::add(p1, s[L]);
                p2 = m31::add(p2, s[2 * L]);
            }
            p2 = m31::eval_at_two(p0, p1, p2);
            if (!LANE_HG) {
                p0 = m31::mul(p0, xv);
                p1 = m31::mul(p1, xv);
                p2 = m31::mul(p2, xv);
            }
            const uint32_t par = (a.parity ^ (k - a.k0)) << 31;
            volatile uint32_t* out = a.evals_out + (size_t)(3 * j) * N + flane;
            out[0] = p0 | par;
            out[N] = p1 | par;
            out[2 * (size_t)N] = p2 | par;
            if (k + 1 == a.n) {
                // rows 0 and 1 of the last folded f table (the layer input when it has no fold;
                // two rows are always in shared memory)
                const uint32_t* s = k == 0 ? reinterpret_cast<const uint32_t*>(mine)
                                           : reinterpret_cast<const uint32_t*>(psm + ((k & 1) * kTabs + j) * kSmemRows);
                volatile uint32_t* ro = a.rows_out + (size_t)(2 * j) * N + flane;
                ro[0] = s[t] | (a.rows_parity << 31);
                ro[N] = s[L + t] | (a.rows_parity << 31);
            }
        }
    }
}

}  // namespace

uint32_t phase_ctas(uint32_t N, uint32_t tpr) { return (N / 4 + tpr - 1) / tpr; }

// Shared memory of a launch whose first folding round leaves S1 rows.
static size_t phase_smem(bool lane_hg, uint32_t S1, uint32_t reps, uint32_t tpr) {
    return 2 * (lane_hg ? 6 : 3) * (size_t)kSmemRows * 16 + (lane_hg ? 0 : 4 * 3 * (size_t)(S1 + S1 / 2)) +
           4 * (size_t)reps * kWarps * 3 * 4 * tpr;
}

int phase_ctas_per_sm() {
    static std::atomic<int> known[64];  // of each device, plus one
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int>& k = known[dev & 63];
    if (const int v = k.load(std::memory_order_relaxed)) return v - 1;
    int least = 0;
    for (int i = 0; i < 4; i++) {
        const bool lane_hg = i < 2;
        auto* const kernel = lane_hg ? (i & 1 ? k_phase<true, true> : k_phase<true, false>)
                                     : (i & 1 ? k_phase<false, true> : k_phase<false, false>);
        size_t most = 0;  // over the tiles that launch_phase takes
        for (uint32_t tpr = 1; tpr <= 32; tpr *= 2) {
            const size_t b = phase_smem(lane_hg, kPhaseItems / 2 / tpr, 3, tpr);
            if (b > most) most = b;
        }
        int n = 0;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 3 * kRepThreads, most);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (i == 0 || n < least) least = n;
    }
    k.store(least + 1, std::memory_order_relaxed);
    return least;
}

size_t phase_priv_quads(uint64_t items, bool whole) { return (whole ? items * 4 : 0) + items / 2 * 6 + items / 4 * 6; }

cudaError_t launch_phase(bool lane_hg, const PhaseArgs& a, cudaStream_t s) {
    if (a.reps < 1 || a.reps > 3 || a.k0 >= a.n || a.n - a.k0 > kMboxRounds || a.N % 4) return cudaErrorInvalidValue;
    if (a.tpr < 1 || a.tpr > 32 || (a.tpr & (a.tpr - 1))) return cudaErrorInvalidValue;
    // rows of the first round's source tables; with k0 = 0 the layer input itself
    const uint64_t rows = 1ull << (a.n - (a.k0 ? a.k0 - 1 : 0));
    if (rows * a.tpr > kPhaseItems || !a.priv || a.priv_stride < phase_priv_quads(rows * a.tpr, a.k0 == 0)) return cudaErrorInvalidValue;
    if (a.two && a.k0 < 2) return cudaErrorInvalidValue;
    if (a.k0 && (!a.fsrc[0] || (lane_hg && !a.hsrc[0]))) return cudaErrorInvalidValue;
    if (!lane_hg && (!a.vx || !a.s[0])) return cudaErrorInvalidValue;
    if (phase_ctas_per_sm() < 1) return cudaErrorInvalidConfiguration;
    const uint32_t kf = a.k0 ? a.k0 : 1, S1 = 1u << (a.n - kf);
    const size_t smem = phase_smem(lane_hg, S1, a.reps, a.tpr);
    const dim3 grid(phase_ctas(a.N, a.tpr)), block(a.reps * kRepThreads);
    auto* const kernel = lane_hg ? (a.two ? k_phase<true, true> : k_phase<true, false>)
                                 : (a.two ? k_phase<false, true> : k_phase<false, false>);
    kernel<<<grid, block, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace gkrgpu
