// Hand-written sm_103a kernels of the GKR prove path (M31).
//
// Data layout in HBM: every per-copy table is row-major rows x N u32 (row r, copy k at
// r*N + k), the byte layout of a proof vector (VectorizedM31::to_bytes, M31.hpp:420-426),
// so a warp's 16-byte loads along a row are fully coalesced.  Scalar tables that do not
// depend on the copy (gate weights, the phase-two h(y) factor) are plain
// arrays of u32 read by broadcast.
//
// Reference counterparts:
//   k_evaluate       CircuitLayer::evaluate                     include/circuit/circuit.hpp:92-105
//   eq_build, eq_at  _eq_evals_at                               include/LinearGKR/sumcheck_common.hpp:17-53
//   k_weights        the scalar factors of _prepare_g_x_vals    include/LinearGKR/sumcheck_helper.hpp:188-229
//   k_hg_round0      _prepare_g_x_vals + poly_eval_at(0)        sumcheck_helper.hpp:172-231, 68-102
//   k_hg_round1      hg rebuilt + receive_challenge + poly_eval_at(1)
//   k_round          receive_challenge + poly_eval_at(k)        sumcheck_helper.hpp:104-133, 68-102
//   k_round_pair     two rounds from one pass over large tables (the second's sums are quadratic
//                    in the first's challenge); k_pair_fin finishes the second
//   k_s_build        _prepare_h_y_vals (copy-independent part)  sumcheck_helper.hpp:233-261
//   k_p2_round01     phase-two poly_eval_at of rounds 0 and 1 from one pass (round 1's sums are
//                    quadratic in round 0's challenge), k_p2_round01_mma the same on the tensor
//                    cores; k_p2_round1_fin finishes round 1
//   k_p2_round2      phase-two round 2 refolding the layer input
//   k_wsum, k_wsum_mma  eval_multilinear                        include/poly_commit/poly.hpp:88-104
// (Phases on small tables: phase.cu.)
//
// k_round gives each CTA one repetition j = blockIdx.x % R: the R CTAs of a row chunk are
// adjacent in launch order, run together and share their common source rows through L2,
// while each thread keeps only one repetition's state.  The kernels whose source is the
// layer input itself (k_hg_round0/1, k_p2_round01, k_p2_round2) keep all R repetitions in a
// thread, so each input row is read once.
#include <atomic>

#include "kernels.cuh"
#include "m31.cuh"

namespace gkrgpu {

const char* const kKernelNames[K_NUM_KERNELS] = {"check_canonical", "evaluate", "gate_weights",
                                                 "hg_build_round0", "round_fold_lane", "round_fold_scalar",
                                                 "phase2_s_build", "weighted_row_sum", "hg_rebuild_round1",
                                                 "verifier_gate_sums", "canonicalize", "phase2_round0", "stage_words", "round_tail", "hg_build",
                                                 "bn254_load",
                                                 "bn254_evaluate", "bn254_gate_weights",
                                                 "bn254_hg_build_round0", "bn254_round_fold_lane",
                                                 "bn254_round_fold_scalar", "bn254_phase2_s_build",
                                                 "bn254_weighted_row_sum", "bn254_unload", "bn254_phase"};

namespace {

using m31::add;
using m31::fold;
using m31::mul;
using m31::sub;

__device__ __forceinline__ uint4 ld4(const uint32_t* __restrict__ base, uint64_t row, uint32_t N, uint32_t lane0) {
    return __ldg(reinterpret_cast<const uint4*>(base + row * N + lane0));
}
__device__ __forceinline__ void st4(uint32_t* base, uint64_t row, uint32_t N, uint32_t lane0, uint4 v) {
    *reinterpret_cast<uint4*>(base + row * N + lane0) = v;
}
__device__ __forceinline__ uint32_t comp(const uint4& v, int l) { return l == 0 ? v.x : l == 1 ? v.y : l == 2 ? v.z : v.w; }
__device__ __forceinline__ uint4 mk4(const uint32_t (&a)[4]) { return make_uint4(a[0], a[1], a[2], a[3]); }

// Canonical residue of a sum of many canonical values (< 2^64 total).
__device__ __forceinline__ uint32_t reduce64(unsigned long long x) {
    x = (x & m31::P) + (x >> 31);
    x = (x & m31::P) + (x >> 31);
    uint32_t s = (uint32_t)x;
    return m31::umin(s, s - m31::P);
}

// x == x mod p for any 64-bit x: x = hi 2^32 + lo and 2^32 == 2 (mod 2^31 - 1), so the result
// lo + 2 hi < 3 * 2^32.  Formed with a shift and an add with carry on the integer ALU (the
// multiply pipe is what the sum kernels saturate).  After it, four more products
// <= (p - 1)^2 keep a 64-bit sum below 3 * 2^32 + 2^64 - 2^35 + 16 < 2^64.
__device__ __forceinline__ uint64_t fold64(uint64_t x) {
    const uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
    uint32_t nl, nh;
    asm("{\n\t"
        ".reg .u32 t;\n\t"
        "shl.b32 t, %2, 1;\n\t"
        "add.cc.u32 %0, %3, t;\n\t"
        "shr.u32 t, %2, 31;\n\t"
        "addc.u32 %1, t, 0;\n\t"
        "}"
        : "=r"(nl), "=r"(nh)
        : "r"(hi), "r"(lo));
    return ((uint64_t)nh << 32) | nl;
}

// acc += a * b with one 32 x 32 -> 64-bit multiply-add.
__device__ __forceinline__ void mad64(uint64_t& acc, uint32_t a, uint32_t b) {
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}

// Canonical total of component c at `lane`, re-zeroing the accumulator for the next launch.
__device__ __forceinline__ uint32_t take(const RedScratch& red, uint32_t c, uint32_t N, uint32_t lane) {
    unsigned long long* p = &red.acc[(size_t)c * N + lane];
    const uint32_t v = reduce64(__ldcg(p));
    *p = 0ull;
    return v;
}

// Reduction of C components x 4 lanes per thread: a shared-memory reduction over the CTA's
// row slices, one 64-bit atomic add per (component, lane) into red.acc at component
// comp_base + c, then the last CTA of this lane group (ticket blockIdx.y) hands every lane
// of the group to fin(lane), which collects the totals with take().
template <class Fin>
__device__ __forceinline__ void finish_group(const RedScratch& red, uint32_t base, uint32_t lanes, uint32_t N, Fin& fin);

template <int C, class Fin>
__device__ __forceinline__ void reduce_group(const uint32_t (&acc)[C][4], const Geo& g, bool active, RedScratch red,
                                             uint32_t comp_base, Fin fin) {
    extern __shared__ uint32_t smem[];
    const uint32_t tid = threadIdx.x, B = blockDim.x;
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) smem[(c * 4 + l) * B + tid] = active ? acc[c][l] : 0u;
    __syncthreads();
    const uint32_t tpr = g.tpr, rps = g.rps;
    for (uint32_t o = tid; o < (uint32_t)C * 4 * tpr; o += B) {
        const uint32_t cl = o / tpr, q = o - cl * tpr;
        const uint32_t* col = smem + cl * B + q;
        unsigned long long s = 0;
        for (uint32_t r = 0; r < rps; r++) s += col[r * tpr];
        const uint32_t c = cl >> 2, l = cl & 3;
        const uint32_t lane = (blockIdx.y * tpr + q) * 4 + l;
        if (lane < g.N) atomicAdd(&red.acc[(size_t)(comp_base + c) * g.N + lane], s);
    }
    finish_group(red, blockIdx.y * 4 * tpr, 4 * tpr, g.N, fin);
}

// After a CTA's atomic adds: the last CTA of lane group blockIdx.y (ticket) hands lanes
// base .. base + lanes - 1 (below N) to fin(lane), re-arms the ticket and, with red.done, publishes
// the group's results to the host (system-scope fence, then the completion counter).
template <class Fin>
__device__ __forceinline__ void finish_group(const RedScratch& red, uint32_t base, uint32_t lanes, uint32_t N, Fin& fin) {
    const uint32_t tid = threadIdx.x, B = blockDim.x;
    __threadfence();
    __syncthreads();
    __shared__ unsigned int is_last;
    if (tid == 0) is_last = (atomicAdd(&red.ticket[blockIdx.y], 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (uint32_t li = tid; li < lanes && base + li < N; li += B) fin(base + li);
    if (tid == 0) red.ticket[blockIdx.y] = 0u;
    if (red.done) {
        __threadfence_system();
        __syncthreads();
        if (tid == 0) atomicAdd_system(red.done, 1u);
    }
}

// reduce_group for kernels with one copy per thread: g.tpr threads (copies) per row slice,
// acc[c] the thread's canonical partial of component c for copy blockIdx.y * g.tpr + q.
template <int C, class Fin>
__device__ __forceinline__ void reduce_group1(const uint32_t (&acc)[C], const Geo& g, bool active, RedScratch red,
                                              Fin fin) {
    extern __shared__ uint32_t smem[];
    const uint32_t tid = threadIdx.x, B = blockDim.x, L = g.tpr, rps = g.rps;
#pragma unroll
    for (int c = 0; c < C; c++) smem[c * B + tid] = active ? acc[c] : 0u;
    __syncthreads();
    for (uint32_t o = tid; o < (uint32_t)C * L; o += B) {
        const uint32_t c = o / L, q = o - c * L;
        const uint32_t* col = smem + c * B + q;
        unsigned long long s = 0;
        for (uint32_t r = 0; r < rps; r++) s += col[r * L];
        if (blockIdx.y * L + q < g.N) atomicAdd(&red.acc[(size_t)c * g.N + blockIdx.y * L + q], s);
    }
    finish_group(red, blockIdx.y * L, L, g.N, fin);
}

struct TileIdx {
    uint32_t q, rs, lane0;
    bool active;
};
__device__ __forceinline__ TileIdx tile_idx(const Geo& g) {
    TileIdx t;
    t.q = threadIdx.x % g.tpr;
    t.rs = threadIdx.x / g.tpr;
    t.lane0 = (blockIdx.y * g.tpr + t.q) * 4;
    t.active = t.rs < g.rps && t.lane0 < g.N;
    return t;
}

// Index of the i-th group a kernel works on: with a list, its i-th entry (the groups that
// have gates, in increasing order), otherwise i itself.
__device__ __forceinline__ uint64_t group_at(const uint32_t* __restrict__ list, uint64_t i) {
    return list ? (uint64_t)__ldg(list + i) : i;
}

// ---------------------------------------------------------------- input check
__global__ void k_check_canonical(const uint32_t* __restrict__ v, uint64_t n, unsigned int* flag) {
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned int bad = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n / 4; i += stride) {
        uint4 x = __ldg(reinterpret_cast<const uint4*>(v) + i);
        bad |= (x.x >= m31::P) | (x.y >= m31::P) | (x.z >= m31::P) | (x.w >= m31::P);
    }
    // every writer stores the same 1, so a plain store works for device and host-mapped flags
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *reinterpret_cast<volatile unsigned int*>(flag) = 1u;
}

// ---------------------------------------------------------------- small transfers
// dst[k * n + i] = src_k[i] for i < n, k < nsrc: small tables moved between device memory and
// host-mapped memory by the SMs, so a proof's stream never waits behind a bulk copy of another
// proof on the copy engine.  With `done`, each CTA makes its writes visible to the host and
// then increments the counter (system scope).
__global__ void k_stage_words(uint32_t* dst, const uint32_t* s0, const uint32_t* s1, const uint32_t* s2, uint32_t nsrc,
                              uint64_t n, unsigned int* done) {
    const uint64_t total = n * nsrc, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const uint64_t k = i / n, e = i - k * n;
        const uint32_t* src = k == 0 ? s0 : (k == 1 ? s1 : s2);
        dst[i] = src[e];
    }
    if (done) {
        __threadfence_system();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd_system(done, 1u);
    }
}

// In-place M31::from_bytes of u32 words (the verifier reads the commitment from proof bytes).
__global__ void k_canonicalize(uint32_t* v, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) v[i] = m31::from_u32(v[i]);
}

// ---------------------------------------------------------------- layer evaluation
// out[o] = sum over mul gates (o, i0, i1, c) of in[i0]*in[i1]*c + sum over add gates
// (o, i0, c) of in[i0]*c, gates grouped by o, so every output row is written once.  Bound by the
// chain of dependent loads to an output's rows (L2 for most): an output of one mul gate or two
// add gates, nearly all, has its gates in one record, loaded an output ahead, and both its rows
// are in flight together; by the CSR lists alone the chain was offsets, gate, row, next gate.
__global__ void __launch_bounds__(256) k_evaluate(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint64_t O,
                                                  const uint4* __restrict__ ev, const uint32_t* __restrict__ mo_off,
                                                  const uint4* __restrict__ mo_g, const uint32_t* __restrict__ ao_off,
                                                  const uint2* __restrict__ ao_g, Geo g) {
    const TileIdx t = tile_idx(g);
    if (!t.active) return;
    const uint64_t step = (uint64_t)gridDim.x * g.rps;
    uint64_t o = (uint64_t)blockIdx.x * g.rps + t.rs;
    uint4 next = o < O ? __ldg(ev + o) : make_uint4(0u, 0u, 0u, 0u);
    for (; o < O; o += step) {
        const uint4 e = next;
        if (o + step < O) next = __ldg(ev + o + step);
        const uint32_t kind = e.x >> 30;
        uint32_t acc[4] = {0u, 0u, 0u, 0u};
        if (kind == kEvMul || kind == kEvAdd) {
            const uint4 a = ld4(in, e.x & 0x3fffffffu, g.N, t.lane0), b = ld4(in, e.y, g.N, t.lane0);
            if (kind == kEvMul) {
#pragma unroll
                for (int l = 0; l < 4; l++) acc[l] = mul(comp(a, l), comp(b, l));
                if (e.z != 1u)
#pragma unroll
                    for (int l = 0; l < 4; l++) acc[l] = mul(acc[l], e.z);
            } else {
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    uint64_t s = (uint64_t)comp(a, l) * e.z;
                    mad64(s, comp(b, l), e.w);
                    acc[l] = reduce64(s);
                }
            }
        } else if (kind == kEvList) {
            const uint32_t m0 = __ldg(mo_off + o), m1 = __ldg(mo_off + o + 1);
            for (uint32_t k = m0; k < m1; k++) {
                const uint4 gt = __ldg(mo_g + k);
                const uint4 a = ld4(in, gt.x, g.N, t.lane0), b = ld4(in, gt.y, g.N, t.lane0);
#pragma unroll
                for (int l = 0; l < 4; l++) acc[l] = add(acc[l], mul(mul(comp(a, l), comp(b, l)), gt.z));
            }
            const uint32_t a0 = __ldg(ao_off + o), a1 = __ldg(ao_off + o + 1);
            for (uint32_t k = a0; k < a1; k++) {
                const uint2 gt = __ldg(ao_g + k);
                const uint4 a = ld4(in, gt.x, g.N, t.lane0);
#pragma unroll
                for (int l = 0; l < 4; l++) acc[l] = add(acc[l], mul(comp(a, l), gt.y));
            }
        }
        st4(out, o, g.N, t.lane0, mk4(acc));
    }
}

// ---------------------------------------------------------------- eq factors
// eq(r_j, z) = prod over bits t of z of (bit ? r_j[t] : 1 - r_j[t]), bit t paired with r[t]
// (little-endian, _eq_evals_at, sumcheck_common.hpp:17-53).  No table over z is stored: a CTA
// builds one table of 32 entries per five bits, repetition and point (at most 36 of them), and
// a kernel multiplies the entries of z where it needs the factor, three products at 2^20.  The
// tables over z took a launch of their own per use (7 us at 2^10 entries, 71 us for two points
// at 2^20, 18 products an entry) and a gather from memory per gate.
constexpr uint32_t kEqBits = 5, kEqTabs = 6, kEqWords = 3 * kEqTabs * 32;  // words per point

__device__ __forceinline__ uint32_t eq_digits(const EqArgs& a) {
    return a.nvars > kEqBits ? (a.nvars + kEqBits - 1) / kEqBits : 1u;
}
// Fills t (kEqWords words per point); the caller synchronises the CTA.
__device__ __forceinline__ void eq_build(uint32_t* t, const EqArgs& a) {
    const uint32_t nd = eq_digits(a), per = nd * a.reps * 32, total = per * (a.f2 ? 2 : 1);
    for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
        const uint32_t p = i / per, k = i - p * per, x = k & 31, jd = k >> 5, j = jd / nd, d = jd - j * nd;
        uint32_t e = d ? 1u : (p ? a.f2 : a.f1);
#pragma unroll
        for (uint32_t b = 0; b < kEqBits; b++) {
            const uint32_t v = d * kEqBits + b;
            if (v >= a.nvars) break;
            const uint32_t r = p ? a.r2[j][v] : a.r1[j][v];
            e = mul(e, (x >> b) & 1 ? r : sub(1u, r));
        }
        t[p * kEqWords + (j * kEqTabs + d) * 32 + x] = e;
    }
}
// f1 eq(r1_j, z) + f2 eq(r2_j, z)
__device__ __forceinline__ uint32_t eq_at(const uint32_t* t, uint32_t nd, bool two, uint32_t j, uint32_t z) {
    const uint32_t* t1 = t + j * kEqTabs * 32;
    uint32_t e = t1[z & 31];
    for (uint32_t d = 1; d < nd; d++) e = mul(e, t1[d * 32 + ((z >> (kEqBits * d)) & 31)]);
    if (!two) return e;
    const uint32_t* t2 = t1 + kEqWords;
    uint32_t f = t2[z & 31];
    for (uint32_t d = 1; d < nd; d++) f = mul(f, t2[d * 32 + ((z >> (kEqBits * d)) & 31)]);
    return add(e, f);
}

// ---------------------------------------------------------------- phase-one scalar factors
// w[k].j = c_k * eqc_j(z_k) for every mul gate k (gates in CSR-by-x order) and
// a[x].j = sum over add gates (z, x, c) of c * eqc_j(z): the copy-independent parts of
// hg(x) = sum_mul v(y) c eqc(z) + sum_add c eqc(z) (sumcheck_helper.hpp:203-229), with
// eqc_j = alpha eq(rz1_j) + beta eq(rz2_j).
__global__ void __launch_bounds__(256) k_weights(uint64_t I, uint64_t Gm, const __grid_constant__ EqArgs eqc,
                                                 const uint4* __restrict__ mx_g, const uint32_t* __restrict__ ax_off,
                                                 const uint2* __restrict__ ax_g, uint4* __restrict__ a_out,
                                                 uint4* __restrict__ w_out) {
    __shared__ uint32_t t[2 * kEqWords];
    eq_build(t, eqc);
    __syncthreads();
    const uint32_t nd = eq_digits(eqc), reps = eqc.reps;
    const bool two = eqc.f2 != 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n = I > Gm ? I : Gm;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (i < Gm) {
            const uint4 gt = __ldg(mx_g + i);  // (y, z, c, 0)
            uint32_t w[3] = {0u, 0u, 0u};
#pragma unroll
            for (uint32_t j = 0; j < 3; j++)
                if (j < reps) w[j] = mul(gt.z, eq_at(t, nd, two, j, gt.y));
            w_out[i] = make_uint4(w[0], w[1], w[2], 0u);
        }
        if (i < I) {
            uint32_t s[3] = {0u, 0u, 0u};
            const uint32_t k0 = __ldg(ax_off + i), k1 = __ldg(ax_off + i + 1);
            for (uint32_t k = k0; k < k1; k++) {
                const uint2 gt = __ldg(ax_g + k);  // (z, c)
#pragma unroll
                for (uint32_t j = 0; j < 3; j++)
                    if (j < reps) s[j] = add(s[j], mul(gt.y, eq_at(t, nd, two, j, gt.x)));
            }
            a_out[i] = make_uint4(s[0], s[1], s[2], 0u);
        }
    }
}

// hg of a layer whose phase one runs in one launch (phase.cu), with a copy of the layer input,
// in the CTAs' own tables: hg_j(x) = sum over add gates (z, x, c) of c eqc_j(z) + sum over mul
// gates (z, x, y, c) of c eqc_j(z) v(y), the weights computed where they are used (a thread per
// row and four copies; the factors are few products next to a launch that stored them).
// Building it inside the phase, whose few CTAs have a chain of three gathers a row, took 11 us
// of a 63 us phase at 2^10 rows and 16 copies.
template <bool STORED>
__global__ void __launch_bounds__(256) k_hg_build(const uint32_t* __restrict__ v, uint32_t I, uint32_t N, uint32_t tpr,
                                                  const __grid_constant__ EqArgs eqc, const uint32_t* __restrict__ mx_off,
                                                  const uint4* __restrict__ mx_g, const uint32_t* __restrict__ ax_off,
                                                  const uint2* __restrict__ ax_g, const uint4* __restrict__ a4,
                                                  const uint4* __restrict__ w4, uint4* __restrict__ priv,
                                                  size_t priv_stride) {
    __shared__ uint32_t t[STORED ? 1 : 2 * kEqWords];
    if (!STORED) {
        eq_build(t, eqc);
        __syncthreads();
    }
    const uint32_t nd = eq_digits(eqc), reps = eqc.reps, Q = N / 4;
    const bool two = eqc.f2 != 0;
    const uint64_t total = (uint64_t)I * Q, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const uint32_t x = (uint32_t)(i / Q), quad = (uint32_t)(i - (uint64_t)x * Q);
        const uint32_t m0 = __ldg(mx_off + x), m1 = __ldg(mx_off + x + 1);
        uint32_t s[3] = {0u, 0u, 0u};
        if (STORED) {
            const uint4 w = __ldg(a4 + x);
            s[0] = w.x; s[1] = w.y; s[2] = w.z;
        } else {
            const uint32_t a0 = __ldg(ax_off + x), a1 = __ldg(ax_off + x + 1);
            for (uint32_t k = a0; k < a1; k++) {
                const uint2 gt = __ldg(ax_g + k);  // (z, c)
#pragma unroll
                for (uint32_t j = 0; j < 3; j++)
                    if (j < reps) s[j] = add(s[j], mul(gt.y, eq_at(t, nd, two, j, gt.x)));
            }
        }
        uint64_t h[3][4];
#pragma unroll
        for (int j = 0; j < 3; j++)
#pragma unroll
            for (int l = 0; l < 4; l++) h[j][l] = s[j];
        for (uint32_t k = m0; k < m1; k++) {
            const uint4 gt = __ldg(mx_g + k);  // (y, z, c, 0)
            const uint4 vy = ld4(v, gt.x, N, 4 * quad);
            const uint4 ws = STORED ? __ldg(w4 + k) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (uint32_t j = 0; j < 3; j++)
                if (j < reps) {
                    const uint32_t w = STORED ? comp(ws, j) : mul(gt.z, eq_at(t, nd, two, j, gt.y));
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        mad64(h[j][l], comp(vy, l), w);
                        h[j][l] = fold64(h[j][l]);
                    }
                }
        }
        const uint32_t at = (I >= 4 ? (x & 3) * (I >> 2) + (x >> 2) : x) * tpr + quad % tpr;  // place() of phase.cu
        uint4* o = priv + (size_t)(quad / tpr) * priv_stride + at;
        o[0] = ld4(v, x, N, 4 * quad);
#pragma unroll
        for (uint32_t j = 0; j < 3; j++)
            if (j < reps)
                o[(size_t)(1 + j) * I * tpr] =
                    make_uint4(reduce64(h[j][0]), reduce64(h[j][1]), reduce64(h[j][2]), reduce64(h[j][3]));
    }
}

// ---------------------------------------------------------------- verifier gate sums
// eval_sparse_circuit_connect_poly (include/LinearGKR/sumcheck_verifier_utils.hpp:22-56)
// for R points at once: mul sums c * eqz_j(o) * eqx_j(i0) * eqy_j(i1) over the mul gates
// (MUL), or add sums c * eqz_j(o) * eqx_j(i0) over the add gates, walked by output o (the
// evaluate CSR).  Block partials go to 64-bit accumulators; the last block writes the R
// canonical totals and re-zeroes the scratch.
template <bool MUL>
__global__ void __launch_bounds__(256) k_gate_sums(uint64_t O, const uint32_t* __restrict__ off,
                                                   const uint32_t* __restrict__ gates, const __grid_constant__ GateEq eq,
                                                   unsigned long long* acc, unsigned int* ticket, uint32_t* out) {
    __shared__ uint32_t tz[2 * kEqWords], tx[kEqWords], ty[MUL ? kEqWords : 1];
    eq_build(tz, eq.z);
    eq_build(tx, eq.x);
    if (MUL) eq_build(ty, eq.y);
    __syncthreads();
    const uint32_t ndz = eq_digits(eq.z), ndx = eq_digits(eq.x), reps = eq.z.reps;
    const bool two = eq.z.f2 != 0;
    uint32_t s[3] = {0u, 0u, 0u};
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; o < O; o += stride) {
        const uint32_t k0 = __ldg(off + o), k1 = __ldg(off + o + 1);
        if (k0 == k1) continue;
        uint32_t ez[3] = {0u, 0u, 0u};
#pragma unroll
        for (uint32_t j = 0; j < 3; j++)
            if (j < reps) ez[j] = eq_at(tz, ndz, two, j, (uint32_t)o);
        for (uint32_t k = k0; k < k1; k++) {
            uint32_t i0, i1 = 0, c;
            if (MUL) {
                const uint4 g = __ldg(reinterpret_cast<const uint4*>(gates) + k);  // (i0, i1, c, 0)
                i0 = g.x; i1 = g.y; c = g.z;
            } else {
                const uint2 g = __ldg(reinterpret_cast<const uint2*>(gates) + k);  // (i0, c)
                i0 = g.x; c = g.y;
            }
#pragma unroll
            for (uint32_t j = 0; j < 3; j++)
                if (j < reps) {
                    uint32_t t = mul(mul(c, ez[j]), eq_at(tx, ndx, false, j, i0));
                    if (MUL) t = mul(t, eq_at(ty, ndx, false, j, i1));
                    s[j] = add(s[j], t);
                }
        }
    }
    __shared__ unsigned long long part[3];
    if (threadIdx.x < 3) part[threadIdx.x] = 0ull;
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < 3; j++) {
        unsigned long long x = s[j];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
        if ((threadIdx.x & 31) == 0) atomicAdd(&part[j], x);
    }
    __syncthreads();
    if (threadIdx.x < reps) atomicAdd(&acc[threadIdx.x], part[threadIdx.x]);
    __threadfence();
    __syncthreads();
    __shared__ unsigned int is_last;
    if (threadIdx.x == 0) is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (threadIdx.x < reps) {
        out[threadIdx.x] = reduce64(__ldcg(&acc[threadIdx.x]));
        acc[threadIdx.x] = 0ull;
    }
    if (threadIdx.x == 0) *ticket = 0u;
}

// w_j[k] (1 - r_j) for the mul gates of even input rows x, w_j[k] r_j for odd x: the weights
// of k_hg_round1, whose sum over the gates of rows 2i and 2i+1 is then hg folded at r_j.
__global__ void k_scale_weights(uint64_t I, const uint32_t* __restrict__ mx_off, const uint4* __restrict__ w4,
                                uint4* __restrict__ w4r, uint4 r) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < I; x += stride) {
        const bool odd = x & 1;
        const uint32_t s0 = odd ? r.x : sub(1u, r.x), s1 = odd ? r.y : sub(1u, r.y), s2 = odd ? r.z : sub(1u, r.z);
        const uint32_t k0 = __ldg(mx_off + x), k1 = __ldg(mx_off + x + 1);
        for (uint32_t k = k0; k < k1; k++) {
            const uint4 w = __ldg(w4 + k);
            w4r[k] = make_uint4(mul(w.x, s0), mul(w.y, s1), mul(w.z, s2), 0u);
        }
    }
}

// ---------------------------------------------------------------- finishers
// Evaluations at 0, 1, 2 of every repetition's round polynomial for one lane; with vx the
// phase-two sums are multiplied by v(rx) (h = v(rx) * s).
struct RoundFin {
    RedScratch red;
    uint32_t* out;       // R x 3 x N
    const uint32_t* vx;  // R x N, or null
    uint32_t N, reps;
    __device__ void operator()(uint32_t lane) const {
        for (uint32_t j = 0; j < reps; j++) {
            uint32_t p0 = take(red, 3 * j, N, lane), p1 = take(red, 3 * j + 1, N, lane);
            uint32_t p2 = m31::eval_at_two(p0, p1, take(red, 3 * j + 2, N, lane));
            if (vx) {
                const uint32_t x = vx[(size_t)j * N + lane];
                p0 = mul(p0, x); p1 = mul(p1, x); p2 = mul(p2, x);
            }
            out[(size_t)(3 * j) * N + lane] = p0;
            out[(size_t)(3 * j + 1) * N + lane] = p1;
            out[(size_t)(3 * j + 2) * N + lane] = p2;
            if (red.evals_dev) {
                red.evals_dev[(size_t)(3 * j) * N + lane] = p0;
                red.evals_dev[(size_t)(3 * j + 1) * N + lane] = p1;
                red.evals_dev[(size_t)(3 * j + 2) * N + lane] = p2;
            }
        }
    }
};

// Round evaluations from two sums per repetition, p0 and p2raw: p1 is the round's claim less
// p0 (an honest prover's round polynomial meets p0 + p1 = claim, the verifier's check in
// sumcheck.hpp:152, so p1 is the same field element as its direct sum).  The claim is
// `claim` (R x N, written by the host before the launch), or without it the previous
// round's polynomial at its challenge r_j, eval_degree2 of the three evaluations in
// red.evals_dev, which this finisher then overwrites (each lane read before it is written).
// With vx (phase two) the sums are multiplied by v(rx) first; the claim is of the multiplied
// polynomial.
struct ClaimFin {
    RedScratch red;
    uint32_t* out;            // R x 3 x N
    const uint32_t* claim;    // R x N, or null
    uint32_t r[3];
    uint32_t N, reps;
    const uint32_t* vx = nullptr;  // R x N, or null
    __device__ void operator()(uint32_t lane) const {
        uint32_t* dev = red.evals_dev;
        for (uint32_t j = 0; j < reps; j++) {
            uint32_t cl;
            if (claim) {
                cl = __ldcv(claim + (size_t)j * N + lane);
            } else {
                const uint32_t rj = j == 0 ? r[0] : (j == 1 ? r[1] : r[2]);
                cl = m31::eval_degree2(dev[(size_t)(3 * j) * N + lane], dev[(size_t)(3 * j + 1) * N + lane],
                                       dev[(size_t)(3 * j + 2) * N + lane], rj);
            }
            uint32_t p0 = take(red, 2 * j, N, lane), p2raw = take(red, 2 * j + 1, N, lane);
            if (vx) {
                const uint32_t x = vx[(size_t)j * N + lane];
                p0 = mul(p0, x);
                p2raw = mul(p2raw, x);
            }
            const uint32_t p1 = sub(cl, p0), p2 = m31::eval_at_two(p0, p1, p2raw);
            out[(size_t)(3 * j) * N + lane] = p0;
            out[(size_t)(3 * j + 1) * N + lane] = p1;
            out[(size_t)(3 * j + 2) * N + lane] = p2;
            if (dev) {
                dev[(size_t)(3 * j) * N + lane] = p0;
                dev[(size_t)(3 * j + 1) * N + lane] = p1;
                dev[(size_t)(3 * j + 2) * N + lane] = p2;
            }
        }
    }
};

struct CopyFin {
    RedScratch red;
    uint32_t* out;  // reps x N
    uint32_t N, reps;
    __device__ void operator()(uint32_t lane) const {
        for (uint32_t j = 0; j < reps; j++) out[(size_t)j * N + lane] = take(red, j, N, lane);
    }
};

// ---------------------------------------------------------------- asynchronous row staging
// cp.async copies (global -> shared, no registers held while in flight) let a thread keep
// several iterations' rows in flight.  Each thread copies and later reads back only its
// own slots, so no barrier is needed between threads; a slot is refilled only after the
// values read from it have been used.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory");
}

// ---------------------------------------------------------------- gathered gate terms
// h_j += sum over mul gates k0 .. k1 - 1 of v[y_k] w_j[k] for the thread's four copies, each
// product added unreduced below 2^32 (mac_lazy).  U gates per step: their gathers (a gate
// index, then a row) are all in flight before the products (8 registers per extra gate).
template <int R, int U>
__device__ __forceinline__ void gate_terms(const uint32_t* __restrict__ v, const uint4* __restrict__ mx_g,
                                           const uint4* __restrict__ w4, uint32_t k0, uint32_t k1, uint32_t N,
                                           uint32_t lane0, uint32_t (&h)[R][4]) {
    uint32_t k = k0;
    for (; U > 1 && k + U <= k1; k += U) {
        uint32_t y[U];
        uint4 w[U], vy[U];
#pragma unroll
        for (int u = 0; u < U; u++) y[u] = __ldg(&mx_g[k + u].x);
#pragma unroll
        for (int u = 0; u < U; u++) w[u] = __ldg(w4 + k + u);
#pragma unroll
        for (int u = 0; u < U; u++) vy[u] = ld4(v, y[u], N, lane0);
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < R; j++)
#pragma unroll
                for (int l = 0; l < 4; l++) h[j][l] = m31::mac_lazy(h[j][l], comp(vy[u], l), comp(w[u], j));
    }
    for (; k < k1; k++) {
        const uint32_t y = __ldg(&mx_g[k].x);
        const uint4 w = __ldg(w4 + k);
        const uint4 vy = ld4(v, y, N, lane0);
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int l = 0; l < 4; l++) h[j][l] = m31::mac_lazy(h[j][l], comp(vy, l), comp(w, j));
    }
}

// ---------------------------------------------------------------- phase one: hg build + round 0
// For each pair (x0, x1) = (2i, 2i+1): hg_j[x] = a_j[x] + sum over mul gates (x, y, k) of
// v[y] * w_j[k], then the round-0 sums of v(x) hg_j(x).  hg is not stored: round 1
// (k_hg_round1) rebuilds it, which costs the gathers again but saves writing and re-reading
// R full-width tables.  All repetitions in one thread: each gathered v[y] row serves the R
// weights.
// The round reads 4 bytes per copy and row and is bound by the integer multiply pipe, so it
// sums only p0 = sum f0 h0 and p2raw = sum (f0 + f1)(h0 + h1), each product added unreduced
// below 2^32 (mac_lazy); p1 is the layer's claim less p0 (ClaimFin).  A pair whose rows both
// lack mul gates (most pairs of a wide layer) has the scalar add weights as h and costs two
// products per copy and repetition: f0 a0 and (f0 + f1)(a0 + a1).  The pair's two input rows,
// their add-gate weights and CSR offsets are staged by cp.async kStages - 1 iterations ahead.
constexpr int kStages = 3;
constexpr int kStageFields = 5;  // v(2i), v(2i+1), a(2i), a(2i+1), (off(2i), off(2i+1), off(2i+2))
constexpr int kMaxStagedSmem = kStages * kStageFields * 16 * 256;
constexpr int kHg0Gates = 2, kHg1Gates = 2;  // gathers in flight per thread (gate_terms)

template <int R>
__global__ void __launch_bounds__(256, 2) k_hg_round0(const uint32_t* __restrict__ v, uint64_t npairs,
                                                      const uint32_t* __restrict__ pairs,
                                                      const uint32_t* __restrict__ mx_off,
                                                      const uint4* __restrict__ mx_g, const uint4* __restrict__ a4,
                                                      const uint4* __restrict__ w4, Geo g, RedScratch red,
                                                      const uint32_t* claim, uint32_t* evals_out) {
    extern __shared__ uint4 ring[];  // kStages x kStageFields x blockDim.x
    const TileIdx t = tile_idx(g);
    const uint32_t B = blockDim.x, tid = threadIdx.x;
    uint32_t acc[2 * R][4];  // 2j: p0, 2j + 1: p2raw
#pragma unroll
    for (int c = 0; c < 2 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = 0u;
    // adds the mul-gate terms of input row x (gates k0 .. k1) to h, canonical before and after
    auto gates = [&](uint32_t k0, uint32_t k1, uint32_t (&h)[R][4]) {
        if (k0 == k1) return;
        gate_terms<R, kHg0Gates>(v, mx_g, w4, k0, k1, g.N, t.lane0, h);
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int l = 0; l < 4; l++) h[j][l] = m31::from_u32(h[j][l]);
    };
    if (t.active) {
        // iteration i works on pair q = group_at(pairs, i) (rows 2q, 2q+1); the list entry of
        // the iteration staged next is loaded one iteration ahead of its staging
        const uint64_t step = (uint64_t)gridDim.x * g.rps;
        const uint64_t i0 = (uint64_t)blockIdx.x * g.rps + t.rs;
        auto stage = [&](uint64_t i, uint64_t q, int slot) {
            if (i < npairs) {
                uint4* st = ring + (size_t)slot * kStageFields * B + tid;
                cp_async16(st, v + (2 * q) * g.N + t.lane0);
                cp_async16(st + B, v + (2 * q + 1) * g.N + t.lane0);
                cp_async16(st + 2 * B, a4 + 2 * q);
                cp_async16(st + 3 * B, a4 + 2 * q + 1);
                cp_async8(st + 4 * B, mx_off + 2 * q);
                cp_async4(reinterpret_cast<uint32_t*>(st + 4 * B) + 2, mx_off + 2 * q + 2);
            }
            cp_async_commit();  // one group per iteration, empty past the end
        };
#pragma unroll
        for (int s = 0; s < kStages - 1; s++) {
            const uint64_t i = i0 + s * step;
            stage(i, i < npairs ? group_at(pairs, i) : 0, s);
        }
        uint64_t next_q = i0 + (kStages - 1) * step < npairs ? group_at(pairs, i0 + (kStages - 1) * step) : 0;
        int slot = 0;
        for (uint64_t i = i0; i < npairs; i += step) {
            // refill the slot read in the previous iteration, then wait for this one
            const uint64_t is = i + (kStages - 1) * step, q = next_q;
            next_q = is + step < npairs ? group_at(pairs, is + step) : 0;
            stage(is, q, slot == 0 ? kStages - 1 : slot - 1);
            cp_async_wait<kStages - 1>();
            const uint4* st = ring + (size_t)slot * kStageFields * B + tid;
            const uint4 f0 = st[0], f1 = st[B], off = st[4 * B];
            uint32_t f01[4];
#pragma unroll
            for (int l = 0; l < 4; l++) f01[l] = add(comp(f0, l), comp(f1, l));
            if (off.x == off.z) {  // neither row has mul gates
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const uint32_t a0 = reinterpret_cast<const uint32_t*>(st + 2 * B)[j];
                    const uint32_t a01 = add(a0, reinterpret_cast<const uint32_t*>(st + 3 * B)[j]);
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        acc[2 * j][l] = m31::mac_lazy(acc[2 * j][l], comp(f0, l), a0);
                        acc[2 * j + 1][l] = m31::mac_lazy(acc[2 * j + 1][l], f01[l], a01);
                    }
                }
            } else {
                // h = hg(2q), then hg(2q) + hg(2q+1): row 2q+1's add weights and gate terms are
                // added onto row 2q's hg
                uint32_t h[R][4];
                const uint4 a0 = st[2 * B], a1 = st[3 * B];
#pragma unroll
                for (int j = 0; j < R; j++)
#pragma unroll
                    for (int l = 0; l < 4; l++) h[j][l] = comp(a0, j);
                gates(off.x, off.y, h);
#pragma unroll
                for (int j = 0; j < R; j++)
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        acc[2 * j][l] = m31::mac_lazy(acc[2 * j][l], comp(f0, l), h[j][l]);
                        h[j][l] = add(h[j][l], comp(a1, j));
                    }
                gates(off.y, off.z, h);
#pragma unroll
                for (int j = 0; j < R; j++)
#pragma unroll
                    for (int l = 0; l < 4; l++) acc[2 * j + 1][l] = m31::mac_lazy(acc[2 * j + 1][l], f01[l], h[j][l]);
            }
            slot = slot + 1 == kStages ? 0 : slot + 1;
        }
        cp_async_wait<0>();
    }
    __syncthreads();  // the ring is reused as the reduction's scratch (sums below 2^32 are
                      // added as they are: the finisher reduces the 64-bit totals)
    reduce_group<2 * R>(acc, g, t.active, red, 0,
                        ClaimFin{red, evals_out, claim, {0u, 0u, 0u}, g.N, (uint32_t)R});
}

// ---------------------------------------------------------------- phase one, round 1
// Round 1 with hg rebuilt rather than read: for each output pair i the four source rows
// x = 4i..4i+3 get hg_j[x] = a_j[x] + sum over mul gates (x, y, k) of v[y] w_j[k] again,
// already folded (the fold is linear: the gate weights come scaled by 1 - r_j for even x and
// r_j for odd x, so one sum over both rows' gates is the folded hg),
// and hg_j and the layer input are folded at r_j into rows 2i, 2i+1 of hdst_j / fdst_j
// (what receive_challenge of round 0 would have left, sumcheck_helper.hpp:104-133), which
// are stored and summed into the round-1 evaluations.  All repetitions in one thread, as in
// k_hg_round0: each gathered v[y] row serves the R weights.  When neither source row of an
// output row has mul gates, its hg is the same for every copy: fold(a_j[x0], a_j[x1], r_j)
// is computed once.  The sums are those of k_hg_round0, p0 and p2raw with mac_lazy (p1 is
// the claim, round 0's polynomial at r_j, less p0); after the first row of a pair only its
// f and h are kept, for p2raw.
template <int R>
__global__ void __launch_bounds__(256, 2) k_hg_round1(const uint32_t* __restrict__ v, uint64_t npairs,
                                                   const uint32_t* __restrict__ quads,
                                                   const uint32_t* __restrict__ mx_off, const uint4* __restrict__ mx_g,
                                                   const uint4* __restrict__ a4, const uint4* __restrict__ w4r,
                                                   RoundPtrs p, Geo g, RedScratch red, uint32_t* evals_out) {
    const TileIdx t = tile_idx(g);
    uint32_t acc[2 * R][4];  // 2j: p0, 2j + 1: p2raw
#pragma unroll
    for (int c = 0; c < 2 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = 0u;
    if (t.active) {
        // iteration ii works on output pair i = group_at(quads, ii) (source rows 4i .. 4i+3)
        const uint64_t step = (uint64_t)gridDim.x * g.rps;
        uint64_t ii = (uint64_t)blockIdx.x * g.rps + t.rs;
        uint64_t next_i = ii < npairs ? group_at(quads, ii) : 0;
        for (; ii < npairs; ii += step) {
            const uint64_t i = next_i;
            next_i = ii + step < npairs ? group_at(quads, ii + step) : 0;
            const uint4 o4 = __ldg(reinterpret_cast<const uint4*>(mx_off + 4 * i));  // off(4i .. 4i+3)
            const uint32_t o_end = __ldg(mx_off + 4 * i + 4);
            const uint32_t off[5] = {o4.x, o4.y, o4.z, o4.w, o_end};
            uint32_t fe[R][4], he[R][4];
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const uint64_t x0 = 4 * i + 2 * s;
                const uint4 v0 = ld4(v, x0, g.N, t.lane0), v1 = ld4(v, x0 + 1, g.N, t.lane0);
                const uint4 a0 = __ldg(a4 + x0), a1 = __ldg(a4 + x0 + 1);
                // fold(hg(x0), hg(x1), r_j) = fold(a_j(x0), a_j(x1), r_j) plus the gate terms of
                // rows x0 and x1 (gates off(x0) .. off(x0 + 2), contiguous) with their weights
                // scaled by 1 - r_j and r_j (w4r, k_scale_weights)
                uint32_t h[R][4];
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const uint32_t hs = m31::lerp(comp(a0, j), comp(a1, j), p.c[j]);
#pragma unroll
                    for (int l = 0; l < 4; l++) h[j][l] = hs;
                }
                if (off[2 * s] != off[2 * s + 2]) {
                    gate_terms<R, kHg1Gates>(v, mx_g, w4r, off[2 * s], off[2 * s + 2], g.N, t.lane0, h);
#pragma unroll
                    for (int j = 0; j < R; j++)
#pragma unroll
                        for (int l = 0; l < 4; l++) h[j][l] = m31::from_u32(h[j][l]);
                }
#pragma unroll
                for (int j = 0; j < R; j++) {
                    uint32_t f[4];
#pragma unroll
                    for (int l = 0; l < 4; l++) f[l] = m31::lerp(comp(v0, l), comp(v1, l), p.c[j]);
                    // null: round 2 refolds the layer input instead of reading stored copies
                    if (p.fdst[0]) st4(p.fdst[j], 2 * i + s, g.N, t.lane0, mk4(f));
                    // a copy-independent hg row is recomputed by round 2 (k_round with H1)
                    if (off[2 * s] != off[2 * s + 2]) st4(p.hdst[j], 2 * i + s, g.N, t.lane0, mk4(h[j]));
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        if (s == 0) {
                            acc[2 * j][l] = m31::mac_lazy(acc[2 * j][l], f[l], h[j][l]);
                            fe[j][l] = f[l];
                            he[j][l] = h[j][l];
                        } else {
                            acc[2 * j + 1][l] =
                                m31::mac_lazy(acc[2 * j + 1][l], add(fe[j][l], f[l]), add(he[j][l], h[j][l]));
                        }
                    }
                }
            }
        }
    }
    reduce_group<2 * R>(acc, g, t.active, red, 0,
                        ClaimFin{red, evals_out, nullptr, {p.r[0], p.r[1], p.r[2]}, g.N, (uint32_t)R});
}

// ---------------------------------------------------------------- fold + reduce round
// FOLD: the inputs hold 4*npairs rows; rows (4i, 4i+1) and (4i+2, 4i+3) are folded at the
// previous round's challenge r_j into rows 2i and 2i+1 of the outputs, which are stored
// for the next round and summed into this round's evaluations.  Without FOLD the inputs
// hold 2*npairs rows and are summed directly (first round of phase two).
// SHARED: every repetition folds the same source table (the layer input at round 1).
// LANE_HG: hg is a per-copy table (phase one); otherwise it is a copy-independent scalar
// table s_j (phase two) and the finisher multiplies the sums by vx_j.
// HR (phase-one rounds 2 and 3, HR = round - 1): a source hg row q covers the 2^HR input
// rows q 2^HR .. (q+1) 2^HR - 1; where none of them has mul gates the previous round did
// not store it, and it is recomputed by folding their add weights a_j at the challenges of
// rounds 0 .. HR-1.  Round 2 (HR = 1) does not store its own output rows of that kind.
template <bool SHARED, bool LANE_HG, bool FOLD, int HR = 0>
__global__ void __launch_bounds__(256, 4) k_round(RoundPtrs p, uint64_t npairs, const uint32_t* __restrict__ vx, Geo g,
                                               uint32_t reps, RedScratch red, uint32_t* evals_out) {
    const TileIdx t = tile_idx(g);
    const uint32_t j = blockIdx.x % reps, cx = blockIdx.x / reps, nx = gridDim.x / reps;
    // selects instead of p.x[j]: a dynamic index into kernel parameters would copy them to the stack
    const uint32_t* __restrict__ fs = (SHARED || j == 0) ? p.fsrc[0] : (j == 1 ? p.fsrc[1] : p.fsrc[2]);
    const uint32_t* __restrict__ hs = j == 0 ? p.hsrc[0] : (j == 1 ? p.hsrc[1] : p.hsrc[2]);
    uint32_t* __restrict__ fd = j == 0 ? p.fdst[0] : (j == 1 ? p.fdst[1] : p.fdst[2]);
    uint32_t* __restrict__ hd = j == 0 ? p.hdst[0] : (j == 1 ? p.hdst[1] : p.hdst[2]);
    const m31::Lerp c = j == 0 ? p.c[0] : (j == 1 ? p.c[1] : p.c[2]);
    uint32_t acc[2][4] = {};  // p0, p2raw, below 2^32 (64-bit sums cost the registers of a fourth CTA)
    auto accum = [&](const uint32_t (&f0)[4], const uint32_t (&f1)[4], const uint32_t (&h0)[4], const uint32_t (&h1)[4]) {
#pragma unroll
        for (int l = 0; l < 4; l++) {
            acc[0][l] = m31::mac_lazy(acc[0][l], f0[l], h0[l]);
            acc[1][l] = m31::mac_lazy(acc[1][l], add(f0[l], f1[l]), add(h0[l], h1[l]));
        }
    };
    if (t.active) {
        uint64_t i = (uint64_t)cx * g.rps + t.rs;
        const uint64_t step = (uint64_t)nx * g.rps;
        if (FOLD && !LANE_HG) {
            // scalar-h folds: two pairs per iteration, their eight row loads issued together
            auto fold_pair = [&](const uint4 (&a)[4], const uint4& sv, uint64_t ii) {
                const uint32_t s0 = m31::lerp(sv.x, sv.y, c), s1 = m31::lerp(sv.z, sv.w, c);
                if (t.q == 0 && blockIdx.y == 0) *reinterpret_cast<uint2*>(hd + 2 * ii) = make_uint2(s0, s1);
                uint32_t f0[4], f1[4], h0[4], h1[4];
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    f0[l] = m31::lerp(comp(a[0], l), comp(a[1], l), c);
                    f1[l] = m31::lerp(comp(a[2], l), comp(a[3], l), c);
                    h0[l] = s0;
                    h1[l] = s1;
                }
                st4(fd, 2 * ii, g.N, t.lane0, mk4(f0));
                st4(fd, 2 * ii + 1, g.N, t.lane0, mk4(f1));
                accum(f0, f1, h0, h1);
            };
            for (; i + step < npairs; i += 2 * step) {
                uint4 a[4], b[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    a[k] = ld4(fs, 4 * i + k, g.N, t.lane0);
                    b[k] = ld4(fs, 4 * (i + step) + k, g.N, t.lane0);
                }
                const uint4 sa = __ldg(reinterpret_cast<const uint4*>(hs) + i);
                const uint4 sb = __ldg(reinterpret_cast<const uint4*>(hs) + i + step);
                fold_pair(a, sa, i);
                fold_pair(b, sb, i + step);
            }
        }
        for (; i < npairs; i += step) {
            uint32_t f0[4], f1[4], h0[4], h1[4];
            if (FOLD) {
                uint4 a[4];
#pragma unroll
                for (int k = 0; k < 4; k++) a[k] = ld4(fs, 4 * i + k, g.N, t.lane0);
                if (LANE_HG) {
                    uint4 b[4];
                    bool keep0 = true, keep1 = true;  // store output rows 2i, 2i+1
                    if (HR > 0) {
                        constexpr int SPAN = 1 << HR;  // input rows per source row
                        // offsets of input rows 4i SPAN .. 4(i+1) SPAN at the source rows' ends
                        uint32_t off[5];
                        const uint32_t* o = p.hoff + 4 * SPAN * i;
#pragma unroll
                        for (int k = 0; k <= 4; k++) off[k] = __ldg(o + k * SPAN);
                        const m31::Lerp c0 = j == 0 ? p.c0[0] : (j == 1 ? p.c0[1] : p.c0[2]);
                        const m31::Lerp2 c01 = j == 0 ? p.c01[0] : (j == 1 ? p.c01[1] : p.c01[2]);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            if (off[k] == off[k + 1]) {
                                const uint32_t* a = reinterpret_cast<const uint32_t*>(p.ha + (4 * i + k) * SPAN) + j;
                                const uint32_t hv = HR == 2
                                                        ? m31::lerp2(__ldg(a), __ldg(a + 4), __ldg(a + 8), __ldg(a + 12), c01)
                                                        : m31::lerp(__ldg(a), __ldg(a + 4), c0);
                                b[k] = make_uint4(hv, hv, hv, hv);
                            } else {
                                b[k] = ld4(hs, 4 * i + k, g.N, t.lane0);
                            }
                        }
                        if (HR == 1) {
                            keep0 = off[0] != off[2];
                            keep1 = off[2] != off[4];
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; k++) b[k] = ld4(hs, 4 * i + k, g.N, t.lane0);
                    }
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        h0[l] = m31::lerp(comp(b[0], l), comp(b[1], l), c);
                        h1[l] = m31::lerp(comp(b[2], l), comp(b[3], l), c);
                    }
                    if (keep0) st4(hd, 2 * i, g.N, t.lane0, mk4(h0));
                    if (keep1) st4(hd, 2 * i + 1, g.N, t.lane0, mk4(h1));
                } else {
                    const uint4 s = __ldg(reinterpret_cast<const uint4*>(hs) + i);
                    const uint32_t s0 = m31::lerp(s.x, s.y, c), s1 = m31::lerp(s.z, s.w, c);
                    if (t.q == 0 && blockIdx.y == 0) *reinterpret_cast<uint2*>(hd + 2 * i) = make_uint2(s0, s1);
#pragma unroll
                    for (int l = 0; l < 4; l++) { h0[l] = s0; h1[l] = s1; }
                }
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    f0[l] = m31::lerp(comp(a[0], l), comp(a[1], l), c);
                    f1[l] = m31::lerp(comp(a[2], l), comp(a[3], l), c);
                }
                st4(fd, 2 * i, g.N, t.lane0, mk4(f0));
                st4(fd, 2 * i + 1, g.N, t.lane0, mk4(f1));
            } else {
                const uint4 a0 = ld4(fs, 2 * i, g.N, t.lane0), a1 = ld4(fs, 2 * i + 1, g.N, t.lane0);
#pragma unroll
                for (int l = 0; l < 4; l++) { f0[l] = comp(a0, l); f1[l] = comp(a1, l); }
                if (LANE_HG) {
                    const uint4 b0 = ld4(hs, 2 * i, g.N, t.lane0), b1 = ld4(hs, 2 * i + 1, g.N, t.lane0);
#pragma unroll
                    for (int l = 0; l < 4; l++) { h0[l] = comp(b0, l); h1[l] = comp(b1, l); }
                } else {
                    const uint2 s = __ldg(reinterpret_cast<const uint2*>(hs) + i);
#pragma unroll
                    for (int l = 0; l < 4; l++) { h0[l] = s.x; h1[l] = s.y; }
                }
            }
            accum(f0, f1, h0, h1);
        }
    }
    reduce_group<2>(acc, g, t.active, red, 2 * j,
                    ClaimFin{red, evals_out, nullptr, {p.r[0], p.r[1], p.r[2]}, g.N, reps,
                             LANE_HG ? nullptr : vx});
}

// Phase-one round 2 after a round 1 that stored no folded copies of the layer input, with
// every repetition in one thread (each input row is loaded once for the R repetitions):
// output row 2i + s (s = 0, 1) of f folds input rows 8i + 4s .. 8i + 4s + 3 in pairs at the
// round-0 challenge r0_j (p.hr[0]) and then at the round-1 challenge r_j (p.r), and output
// row 2i + s of hg folds round 1's hg rows 4i + 2s, 4i + 2s + 1 at r_j, a row round 1 did not
// store (both its input rows without mul gates) being recomputed from the add weights at
// r0_j (receive_challenge twice, sumcheck_helper.hpp:104-133).  Output hg rows whose four
// input rows have no mul gates are not stored (round 3 recomputes them), as in
// k_round<.., HR = 1>.
template <int R>
__global__ void __launch_bounds__(256, 2) k_p1_round2(RoundPtrs p, uint64_t npairs, Geo g, RedScratch red,
                                                   uint32_t* evals_out) {
    const TileIdx t = tile_idx(g);
    const uint32_t* __restrict__ v = p.fsrc[0];
    uint32_t acc[2 * R][4];  // 2j: p0, 2j + 1: p2raw
#pragma unroll
    for (int c = 0; c < 2 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = 0u;
    if (t.active) {
        for (uint64_t i = (uint64_t)blockIdx.x * g.rps + t.rs; i < npairs; i += (uint64_t)gridDim.x * g.rps) {
            // offsets of input rows 8i, 8i+2, .., 8i+8: round-1 hg row 4i + k covers input rows
            // 8i + 2k, 8i + 2k + 1
            uint32_t off[5];
#pragma unroll
            for (int k = 0; k <= 4; k++) off[k] = __ldg(p.hoff + 8 * i + 2 * k);
            uint32_t fe[R][4], he[R][4];
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const uint64_t q = 8 * i + 4 * s;
                const uint4 x0 = ld4(v, q, g.N, t.lane0), x1 = ld4(v, q + 1, g.N, t.lane0);
                const uint4 x2 = ld4(v, q + 2, g.N, t.lane0), x3 = ld4(v, q + 3, g.N, t.lane0);
                const bool keep = off[2 * s] != off[2 * s + 2];
#pragma unroll
                for (int j = 0; j < R; j++) {
                    uint4 b[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int k = 2 * s + e;
                        if (off[k] == off[k + 1]) {
                            const uint32_t* a = reinterpret_cast<const uint32_t*>(p.ha + (4 * i + k) * 2) + j;
                            const uint32_t hv = m31::lerp(__ldg(a), __ldg(a + 4), p.c0[j]);
                            b[e] = make_uint4(hv, hv, hv, hv);
                        } else {
                            b[e] = ld4(p.hsrc[j], 4 * i + k, g.N, t.lane0);
                        }
                    }
                    uint32_t f[4], h[4];
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        f[l] = m31::lerp2(comp(x0, l), comp(x1, l), comp(x2, l), comp(x3, l), p.c01[j]);
                        h[l] = m31::lerp(comp(b[0], l), comp(b[1], l), p.c[j]);
                    }
                    st4(p.fdst[j], 2 * i + s, g.N, t.lane0, mk4(f));
                    if (keep) st4(p.hdst[j], 2 * i + s, g.N, t.lane0, mk4(h));
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        if (s == 0) {
                            acc[2 * j][l] = m31::mac_lazy(acc[2 * j][l], f[l], h[l]);
                            fe[j][l] = f[l];
                            he[j][l] = h[l];
                        } else {
                            acc[2 * j + 1][l] =
                                m31::mac_lazy(acc[2 * j + 1][l], add(fe[j][l], f[l]), add(he[j][l], h[l]));
                        }
                    }
                }
            }
        }
    }
    reduce_group<2 * R>(acc, g, t.active, red, 0,
                        ClaimFin{red, evals_out, nullptr, {p.r[0], p.r[1], p.r[2]}, g.N, (uint32_t)R});
}

// Rounds k and k + 1 from one pass over the tables: output rows 4i .. 4i+3 (the tables as round
// k has them) are folded from the source at the D challenges since it was stored, stored
// themselves, and summed into what both rounds need.  A round's sums are quadratic in the
// challenge before it: with E over rows 4i, 4i+1 and U over the sums of rows 4i, 4i+2 and
// 4i+1, 4i+3, round k + 1's p0 and p2raw at r are (1-r)^2 X00 + r (1-r) (XQ - X00 - X11) +
// r^2 X11 for X = E and U (k_pair_fin), so round k + 1 reads no table.
// What bounds it: memory, and that is what the pair saves.  From stored tables of T bytes two
// single rounds move T + T/2 + T/2 + T/4, a pair at D = 1 T + T/2, each pair after it (D = 2)
// T + T/4 where single rounds move 9/4 T.
// One repetition a thread as in k_round: 32 sums and an output row's loads in flight; two CTAs
// an SM is the registers' bound.  2^20 rows of 1024 copies: rounds 3 and 4 in phase one 1430 us
// (5.5 TB/s; the add weights' rows are computed), 5 and 6 596 us (6.8 TB/s), rounds 3 to 8 of
// four such layers 2.1 ms less than one by one.
// HR = 2: round 3 in phase one, source hg rows as in k_round<.., HR = 2>.
constexpr int kPairSums = 8;  // E00, E11, EQ, F00 (rows 4i+2, 4i+3), FQ, U00, U11, UQ

// Round k's evaluations from the pair's sums, which stay canonical in `sums` for round k + 1.
struct PairFin {
    RedScratch red;
    uint32_t* out;       // R x 3 x N
    uint32_t* sums;      // kPairSums R x N
    uint32_t r[3];       // challenges of round k - 1
    uint32_t N, reps;
    const uint32_t* vx;  // R x N, or null
    __device__ void operator()(uint32_t lane) const {
        uint32_t* dev = red.evals_dev;
        for (uint32_t j = 0; j < reps; j++) {
            uint32_t m[kPairSums];
#pragma unroll
            for (int e = 0; e < kPairSums; e++) {
                m[e] = take(red, kPairSums * j + e, N, lane);
                sums[(size_t)(kPairSums * j + e) * N + lane] = m[e];
            }
            const uint32_t rj = j == 0 ? r[0] : (j == 1 ? r[1] : r[2]);
            uint32_t* d = dev + (size_t)(3 * j) * N + lane;
            const uint32_t cl = m31::eval_degree2(d[0], d[N], d[2 * (size_t)N], rj);
            uint32_t p0 = add(m[0], m[3]), p2raw = add(m[2], m[4]);
            if (vx) {
                const uint32_t x = vx[(size_t)j * N + lane];
                p0 = mul(p0, x);
                p2raw = mul(p2raw, x);
            }
            const uint32_t p1 = sub(cl, p0), p2 = m31::eval_at_two(p0, p1, p2raw);
            uint32_t* o = out + (size_t)(3 * j) * N + lane;
            o[0] = d[0] = p0;
            o[N] = d[N] = p1;
            o[2 * (size_t)N] = d[2 * (size_t)N] = p2;
        }
    }
};

template <bool LANE_HG, int D, int HR>
__global__ void __launch_bounds__(256, 2) k_round_pair(RoundPtrs p, uint64_t ngroups, const uint32_t* __restrict__ vx,
                                                       Geo g, uint32_t reps, RedScratch red, uint32_t* evals_out,
                                                       uint32_t* sums_out) {
    const TileIdx t = tile_idx(g);
    const uint32_t j = blockIdx.x % reps, cx = blockIdx.x / reps, nx = gridDim.x / reps;
    const uint32_t* __restrict__ fs = j == 0 ? p.fsrc[0] : (j == 1 ? p.fsrc[1] : p.fsrc[2]);
    const uint32_t* __restrict__ hs = j == 0 ? p.hsrc[0] : (j == 1 ? p.hsrc[1] : p.hsrc[2]);
    uint32_t* __restrict__ fd = j == 0 ? p.fdst[0] : (j == 1 ? p.fdst[1] : p.fdst[2]);
    uint32_t* __restrict__ hd = j == 0 ? p.hdst[0] : (j == 1 ? p.hdst[1] : p.hdst[2]);
    const m31::Lerp c = j == 0 ? p.c[0] : (j == 1 ? p.c[1] : p.c[2]);
    const m31::Lerp2 c01 = j == 0 ? p.c01[0] : (j == 1 ? p.c01[1] : p.c01[2]);
    constexpr int S = 1 << D;  // source rows of an output row
    uint32_t acc[kPairSums][4] = {};
    auto mac = [&](int e, int l, uint32_t f, uint32_t h) { acc[e][l] = m31::mac_lazy(acc[e][l], f, h); };
    auto folded = [&](const uint4 (&x)[S], uint32_t (&o)[4]) {
#pragma unroll
        for (int l = 0; l < 4; l++)
            o[l] = D == 2 ? m31::lerp2(comp(x[0], l), comp(x[1], l), comp(x[2 % S], l), comp(x[3 % S], l), c01)
                          : m31::lerp(comp(x[0], l), comp(x[1], l), c);
    };
    if (t.active) {
        for (uint64_t i = (uint64_t)cx * g.rps + t.rs; i < ngroups; i += (uint64_t)nx * g.rps) {
            uint32_t hsc[4];
            if (!LANE_HG) {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (D == 2) {
                        const uint4 x = __ldg(reinterpret_cast<const uint4*>(hs) + 4 * i + e);
                        hsc[e] = m31::lerp2(x.x, x.y, x.z, x.w, c01);
                    } else {
                        const uint2 x = __ldg(reinterpret_cast<const uint2*>(hs) + 4 * i + e);
                        hsc[e] = m31::lerp(x.x, x.y, c);
                    }
                }
                if (t.q == 0 && blockIdx.y == 0)
                    reinterpret_cast<uint4*>(hd)[i] = make_uint4(hsc[0], hsc[1], hsc[2], hsc[3]);
            }
            uint32_t f[4][4], h[4][4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint64_t row = 4 * i + e;
                uint4 x[S];
#pragma unroll
                for (int k = 0; k < S; k++) x[k] = ld4(fs, S * row + k, g.N, t.lane0);
                if (LANE_HG) {
                    uint4 y[S];
#pragma unroll
                    for (int k = 0; k < S; k++) {
                        const uint64_t src = S * row + k;
                        bool stored = true;
                        if (HR == 2) stored = __ldg(p.hoff + 4 * src) != __ldg(p.hoff + 4 * src + 4);
                        if (stored) {
                            y[k] = ld4(hs, src, g.N, t.lane0);
                        } else {
                            const uint32_t* a = reinterpret_cast<const uint32_t*>(p.ha + 4 * src) + j;
                            const uint32_t hv = m31::lerp2(__ldg(a), __ldg(a + 4), __ldg(a + 8), __ldg(a + 12), c01);
                            y[k] = make_uint4(hv, hv, hv, hv);
                        }
                    }
                    folded(y, h[e]);
                    st4(hd, row, g.N, t.lane0, mk4(h[e]));
                } else {
#pragma unroll
                    for (int l = 0; l < 4; l++) h[e][l] = hsc[e];
                }
                folded(x, f[e]);
                st4(fd, row, g.N, t.lane0, mk4(f[e]));
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    if (e < 3) mac(e == 2 ? 3 : e, l, f[e][l], h[e][l]);
                    if (e & 1) mac(e == 1 ? 2 : 4, l, add(f[e - 1][l], f[e][l]), add(h[e - 1][l], h[e][l]));
                }
            }
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint32_t f0 = add(f[0][l], f[2][l]), f1 = add(f[1][l], f[3][l]);
                const uint32_t h0 = add(h[0][l], h[2][l]), h1 = add(h[1][l], h[3][l]);
                mac(5, l, f0, h0);
                mac(6, l, f1, h1);
                mac(7, l, add(f0, f1), add(h0, h1));
            }
        }
    }
    reduce_group<kPairSums>(acc, g, t.active, red, kPairSums * j,
                            PairFin{red, evals_out, sums_out, {p.r[0], p.r[1], p.r[2]}, g.N, reps,
                                    LANE_HG ? nullptr : vx});
}

// Round k + 1 of a pair at round k's challenges p.r from the sums of k_round_pair, a thread a
// copy and repetition.  With rows (4 or 8, of the tables that the pair stored) it also folds
// them at p.r, for the last round or for its rows 0..1: there are only these few then.
template <bool LANE_HG>
__global__ void __launch_bounds__(256) k_pair_fin(RoundPtrs p, const uint32_t* __restrict__ sums,
                                                  const uint32_t* __restrict__ vx, uint32_t rows, uint32_t N,
                                                  uint32_t reps, uint32_t* evals_out, uint32_t* evals_dev,
                                                  unsigned int* done) {
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < reps * N) {
        const uint32_t j = idx / N, lane = idx - j * N;
        const uint32_t r = j == 0 ? p.r[0] : (j == 1 ? p.r[1] : p.r[2]), omr = sub(1u, r);
        const uint32_t c0 = mul(omr, omr), c1 = mul(r, omr), c2 = mul(r, r);
        uint32_t m[kPairSums];
#pragma unroll
        for (int e = 0; e < kPairSums; e++) m[e] = __ldg(sums + (size_t)(kPairSums * j + e) * N + lane);
        uint32_t p0 = add(add(mul(c0, m[0]), mul(c1, sub(sub(m[2], m[0]), m[1]))), mul(c2, m[1]));
        uint32_t p2raw = add(add(mul(c0, m[5]), mul(c1, sub(sub(m[7], m[5]), m[6]))), mul(c2, m[6]));
        if (!LANE_HG) {
            const uint32_t x = __ldg(vx + idx);
            p0 = mul(p0, x);
            p2raw = mul(p2raw, x);
        }
        uint32_t *d = evals_dev + (size_t)(3 * j) * N + lane, *o = evals_out + (size_t)(3 * j) * N + lane;
        const uint32_t p1 = sub(m31::eval_degree2(d[0], d[N], d[2 * (size_t)N], r), p0);
        o[0] = d[0] = p0;
        o[N] = d[N] = p1;
        o[2 * (size_t)N] = d[2 * (size_t)N] = m31::eval_at_two(p0, p1, p2raw);
        const m31::Lerp c = m31::lerp_at(r);
        const uint32_t* fs = j == 0 ? p.fsrc[0] : (j == 1 ? p.fsrc[1] : p.fsrc[2]);
        const uint32_t* hs = j == 0 ? p.hsrc[0] : (j == 1 ? p.hsrc[1] : p.hsrc[2]);
        uint32_t* fd = j == 0 ? p.fdst[0] : (j == 1 ? p.fdst[1] : p.fdst[2]);
        uint32_t* hd = j == 0 ? p.hdst[0] : (j == 1 ? p.hdst[1] : p.hdst[2]);
        for (uint32_t i = 0; i < rows / 2; i++) {
            const size_t s0 = (size_t)(2 * i) * N + lane, to = (size_t)i * N + lane;
            fd[to] = m31::lerp(fs[s0], fs[s0 + N], c);
            if (LANE_HG) hd[to] = m31::lerp(hs[s0], hs[s0 + N], c);
            else if (lane == 0) hd[i] = m31::lerp(hs[2 * i], hs[2 * i + 1], c);
        }
    }
    __threadfence_system();
    __syncthreads();
    if (done && threadIdx.x == 0) atomicAdd_system(done, 1u);
}

// Shared-source rounds (phase-1 round 1, phase-2 rounds 0 and 1) with every repetition in
// one thread: the layer input rows are read once for all R repetitions instead of once per
// repetition-CTA.  Same semantics as k_round<true, LANE_HG, FOLD>.
template <int R, bool LANE_HG, bool FOLD>
__global__ void __launch_bounds__(256) k_round_shared(RoundPtrs p, uint64_t npairs, const uint32_t* __restrict__ vx,
                                                      Geo g, RedScratch red, uint32_t* evals_out) {
    const TileIdx t = tile_idx(g);
    const uint32_t* __restrict__ fs = p.fsrc[0];
    uint32_t acc[2 * R][4] = {};  // 2j: p0, 2j + 1: p2raw
    if (t.active) {
        for (uint64_t i = (uint64_t)blockIdx.x * g.rps + t.rs; i < npairs; i += (uint64_t)gridDim.x * g.rps) {
            uint4 a[4];
            if (FOLD) {
#pragma unroll
                for (int k = 0; k < 4; k++) a[k] = ld4(fs, 4 * i + k, g.N, t.lane0);
            } else {
                a[0] = ld4(fs, 2 * i, g.N, t.lane0);
                a[1] = ld4(fs, 2 * i + 1, g.N, t.lane0);
            }
#pragma unroll
            for (int j = 0; j < R; j++) {
                const m31::Lerp c = p.c[j];
                uint32_t f0[4], f1[4], h0[4], h1[4];
                if (FOLD) {
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        f0[l] = m31::lerp(comp(a[0], l), comp(a[1], l), c);
                        f1[l] = m31::lerp(comp(a[2], l), comp(a[3], l), c);
                    }
                    if (p.fdst[j]) {  // null: the next round refolds the source instead
                        st4(p.fdst[j], 2 * i, g.N, t.lane0, mk4(f0));
                        st4(p.fdst[j], 2 * i + 1, g.N, t.lane0, mk4(f1));
                    }
                } else {
#pragma unroll
                    for (int l = 0; l < 4; l++) { f0[l] = comp(a[0], l); f1[l] = comp(a[1], l); }
                }
                if (LANE_HG) {
                    uint4 b[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) b[k] = ld4(p.hsrc[j], 4 * i + k, g.N, t.lane0);
#pragma unroll
                    for (int l = 0; l < 4; l++) {
                        h0[l] = m31::lerp(comp(b[0], l), comp(b[1], l), c);
                        h1[l] = m31::lerp(comp(b[2], l), comp(b[3], l), c);
                    }
                    st4(p.hdst[j], 2 * i, g.N, t.lane0, mk4(h0));
                    st4(p.hdst[j], 2 * i + 1, g.N, t.lane0, mk4(h1));
                } else if (FOLD) {
                    const uint4 s = __ldg(reinterpret_cast<const uint4*>(p.hsrc[j]) + i);
                    const uint32_t s0 = m31::lerp(s.x, s.y, c), s1 = m31::lerp(s.z, s.w, c);
                    if (t.q == 0 && blockIdx.y == 0) *reinterpret_cast<uint2*>(p.hdst[j] + 2 * i) = make_uint2(s0, s1);
#pragma unroll
                    for (int l = 0; l < 4; l++) { h0[l] = s0; h1[l] = s1; }
                } else {
                    const uint2 s = __ldg(reinterpret_cast<const uint2*>(p.hsrc[j]) + i);
#pragma unroll
                    for (int l = 0; l < 4; l++) { h0[l] = s.x; h1[l] = s.y; }
                }
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    acc[2 * j][l] = add(acc[2 * j][l], mul(f0[l], h0[l]));
                    acc[2 * j + 1][l] = add(acc[2 * j + 1][l], mul(add(f0[l], f1[l]), add(h0[l], h1[l])));
                }
            }
        }
    }
    reduce_group<2 * R>(acc, g, t.active, red, 0,
                        ClaimFin{red, evals_out, nullptr, {p.r[0], p.r[1], p.r[2]}, g.N, (uint32_t)R,
                                 LANE_HG ? nullptr : vx});
}

// Phase-two round 2 from the layer input: round 1 stored only its folded scalar tables, not
// the folded copies f1_j(q) = fold(v(2q), v(2q+1), r0_j), which would be written once and
// read once; here each output pair i refolds the eight input rows 8i..8i+7 at r0_j (p.hr[0])
// and then at r1_j (p.r), stores rows 2i, 2i+1 of f2_j and the folded scalars, and sums the
// round-2 evaluations (receive_challenge + poly_eval_at, sumcheck_helper.hpp:68-133).  All
// repetitions in one thread: the eight rows are read once for the R tables.  The rows of the
// next kRowStages - 1 iterations are staged with cp.async while an iteration computes (each
// thread copies and reads back only its own slots).
constexpr int kRowStages = 3;
constexpr int kRowRingSmem = kRowStages * 8 * 16 * 256;

template <int R>
__global__ void __launch_bounds__(256, 2) k_p2_round2(RoundPtrs p, uint64_t npairs, const uint32_t* __restrict__ vx,
                                                   Geo g, RedScratch red, uint32_t* evals_out) {
    extern __shared__ uint4 rows8[];  // kRowStages x 8 x blockDim.x
    const TileIdx t = tile_idx(g);
    const uint32_t B = blockDim.x, tid = threadIdx.x;
    const uint32_t* __restrict__ fs = p.fsrc[0];
    uint32_t acc[2 * R][4];  // 2j: p0, 2j + 1: p2raw
#pragma unroll
    for (int c = 0; c < 2 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = 0u;
    if (t.active) {
        const uint64_t step = (uint64_t)gridDim.x * g.rps;
        const uint64_t i0 = (uint64_t)blockIdx.x * g.rps + t.rs;
        auto stage = [&](uint64_t i, int slot) {
            if (i < npairs) {
                uint4* st = rows8 + (size_t)slot * 8 * B + tid;
#pragma unroll
                for (int k = 0; k < 8; k++) cp_async16(st + k * B, fs + (8 * i + k) * g.N + t.lane0);
            }
            cp_async_commit();  // one group per iteration, empty past the end
        };
#pragma unroll
        for (int q = 0; q < kRowStages - 1; q++) stage(i0 + q * step, q);
        int slot = 0;
        for (uint64_t i = i0; i < npairs; i += step) {
            // refill the slot read in the previous iteration, then wait for this one
            stage(i + (kRowStages - 1) * step, slot == 0 ? kRowStages - 1 : slot - 1);
            cp_async_wait<kRowStages - 1>();
            const uint4* st = rows8 + (size_t)slot * 8 * B + tid;
            uint4 a[8];
#pragma unroll
            for (int k = 0; k < 8; k++) a[k] = st[k * B];
            slot = slot + 1 == kRowStages ? 0 : slot + 1;
#pragma unroll
            for (int j = 0; j < R; j++) {
                const uint4 sv = __ldg(reinterpret_cast<const uint4*>(p.hsrc[j]) + i);
                const uint32_t s0 = m31::lerp(sv.x, sv.y, p.c[j]), s1 = m31::lerp(sv.z, sv.w, p.c[j]);
                if (t.q == 0 && blockIdx.y == 0) *reinterpret_cast<uint2*>(p.hdst[j] + 2 * i) = make_uint2(s0, s1);
                uint32_t f0[4], f1[4], h0[4], h1[4];
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    f0[l] = m31::lerp2(comp(a[0], l), comp(a[1], l), comp(a[2], l), comp(a[3], l), p.c01[j]);
                    f1[l] = m31::lerp2(comp(a[4], l), comp(a[5], l), comp(a[6], l), comp(a[7], l), p.c01[j]);
                    h0[l] = s0;
                    h1[l] = s1;
                }
                st4(p.fdst[j], 2 * i, g.N, t.lane0, mk4(f0));
                st4(p.fdst[j], 2 * i + 1, g.N, t.lane0, mk4(f1));
                // sums kept below 2^32 without reduction (mac_lazy), canonical at the end
                const uint32_t hs = add(s0, s1);
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    acc[2 * j][l] = m31::mac_lazy(acc[2 * j][l], f0[l], h0[l]);
                    acc[2 * j + 1][l] = m31::mac_lazy(acc[2 * j + 1][l], add(f0[l], f1[l]), hs);
                }
            }
        }
        cp_async_wait<0>();
    }
#pragma unroll
    for (int c = 0; c < 2 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = m31::from_u32(acc[c][l]);
    __syncthreads();  // the ring is reused as the reduction's scratch
    reduce_group<2 * R>(acc, g, t.active, red, 0,
                        ClaimFin{red, evals_out, nullptr, {p.r[0], p.r[1], p.r[2]}, g.N, (uint32_t)R, vx});
}

// Phase-two round 0 (no fold): p0_j = sum f(2i) s_j(2i), p1_j = sum f(2i+1) s_j(2i+1),
// p2raw_j = sum (f(2i) + f(2i+1)) (s_j(2i) + s_j(2i+1)) over the layer input f = v, for
// all R repetitions in one thread so that each row read serves the R scalar tables.  With
// 4 bytes read per copy and row, the products are summed unreduced in 64-bit accumulators
// (one multiply-add each, every factor canonical) and folded every third pair.  The pair's
// two rows and the R scalar pairs are staged by cp.async kP2Stages - 1 iterations ahead.
// (SumcheckMultiLinearProdHelper::poly_eval_at on the first phase-two round,
// sumcheck_helper.hpp:68-102, with hg = v(rx) s: the finisher multiplies by vx.)
constexpr int kP2Stages = 6;
constexpr int kP2Fields = 4;  // v(2i), v(2i+1), (s_0, s_1) pairs, (s_2 pair, unused)
constexpr int kMaxP2Smem = kP2Stages * kP2Fields * 16 * 256;

struct P2Src {
    const uint32_t* f;     // the layer input, 2 npairs rows
    const uint32_t* s[3];  // the repetitions' scalar tables s_j
};

template <int R>
__global__ void __launch_bounds__(256, 2) k_p2_round0(P2Src src, uint64_t npairs, const uint32_t* __restrict__ vx,
                                                      Geo g, RedScratch red, uint32_t* evals_out) {
    extern __shared__ uint4 ring[];  // kP2Stages x kP2Fields x blockDim.x
    const TileIdx t = tile_idx(g);
    const uint32_t B = blockDim.x, tid = threadIdx.x;
    const uint32_t* __restrict__ fs = src.f;
    const uint32_t* hsrc[R];
#pragma unroll
    for (int j = 0; j < R; j++) hsrc[j] = src.s[j];
    uint64_t acc[3 * R][4];
#pragma unroll
    for (int c = 0; c < 3 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = 0ull;
    if (t.active) {
        const uint64_t step = (uint64_t)gridDim.x * g.rps;
        const uint64_t i0 = (uint64_t)blockIdx.x * g.rps + t.rs;
        auto stage = [&](uint64_t i, int slot) {
            if (i < npairs) {
                uint4* st = ring + (size_t)slot * kP2Fields * B + tid;
                cp_async16(st, fs + (2 * i) * g.N + t.lane0);
                cp_async16(st + B, fs + (2 * i + 1) * g.N + t.lane0);
#pragma unroll
                for (int j = 0; j < R; j++)
                    cp_async8(reinterpret_cast<uint2*>(st + (2 + j / 2) * B) + (j & 1), hsrc[j] + 2 * i);
            }
            cp_async_commit();  // one group per iteration, empty past the end
        };
#pragma unroll
        for (int s = 0; s < kP2Stages - 1; s++) stage(i0 + s * step, s);
        int slot = 0;
        uint32_t since_fold = 0;
        for (uint64_t i = i0; i < npairs; i += step) {
            stage(i + (kP2Stages - 1) * step, slot == 0 ? kP2Stages - 1 : slot - 1);
            cp_async_wait<kP2Stages - 1>();
            const uint4* st = ring + (size_t)slot * kP2Fields * B + tid;
            const uint4 f0 = st[0], f1 = st[B];
            uint32_t sa[R], sb[R], sab[R];
#pragma unroll
            for (int j = 0; j < R; j++) {
                const uint2 sj = reinterpret_cast<const uint2*>(st + (2 + j / 2) * B)[j & 1];
                sa[j] = sj.x;
                sb[j] = sj.y;
                sab[j] = add(sj.x, sj.y);
            }
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint32_t a = comp(f0, l), b = comp(f1, l), ab = add(a, b);
#pragma unroll
                for (int j = 0; j < R; j++) {
                    acc[3 * j][l] += (uint64_t)a * sa[j];
                    acc[3 * j + 1][l] += (uint64_t)b * sb[j];
                    acc[3 * j + 2][l] += (uint64_t)ab * sab[j];
                }
            }
            if (++since_fold == 3) {
                since_fold = 0;
#pragma unroll
                for (int c = 0; c < 3 * R; c++)
#pragma unroll
                    for (int l = 0; l < 4; l++) acc[c][l] = fold64(acc[c][l]);
            }
            slot = slot + 1 == kP2Stages ? 0 : slot + 1;
        }
        cp_async_wait<0>();
    }
    uint32_t out[3 * R][4];
#pragma unroll
    for (int c = 0; c < 3 * R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) out[c][l] = reduce64(acc[c][l]);
    __syncthreads();  // the ring is reused as the reduction's scratch
    reduce_group<3 * R>(out, g, t.active, red, 0, RoundFin{red, evals_out, vx, g.N, (uint32_t)R});
}

// ---------------------------------------------------------------- phase two: rounds 0 and 1 in one pass
// Round 1 folds the layer input v and the scalar tables s_j at the round-0 challenge r
// (receive_challenge, sumcheck_helper.hpp:104-133), so its sums are quadratic in r.  Over a
// group of four input rows y = 4i..4i+3 (values v0..v3, scalars s0..s3), round 1's pair is
// f0 = (1-r) v0 + r v1, f1 = (1-r) v2 + r v3 (h0, h1 alike from s), and
//   p0_1    = sum f0 h0             = (1-r)^2 E00 + r(1-r) KE + r^2 E11,
//   p1_1    = sum f1 h1             = (1-r)^2 F22 + r(1-r) KF + r^2 F33,
//   p2raw_1 = sum (f0 + f1)(h0 + h1) = (1-r)^2 U00 + r(1-r) KU + r^2 U11,
// with E00 = sum v0 s0, E11 = sum v1 s1 and the cross sum KE = sum v0 s1 + v1 s0 = QE - E00 - E11,
// QE = sum (v0 + v1)(s0 + s1) (F.. and QF from rows 2, 3), and U.. the same over u0 = v0 + v2,
// u1 = v1 + v3 and t0 = s0 + s2, t1 = s1 + s3.  Round 0's sums (poly_eval_at over the pairs
// (4i, 4i+1), (4i+2, 4i+3), sumcheck_helper.hpp:68-102) are p0_0 = E00 + F22,
// p1_0 = E11 + F33 and p2raw_0 = QE + QF.  One pass over v therefore yields both rounds: the
// finisher writes round 0's evaluations (times v(rx), since h = v(rx) s) for the transcript
// and the 9R canonical sums to `sums`, and k_p2_round1_fin evaluates round 1 from them once r
// is known — round 1 never reads v.
// One copy per thread: nine products per repetition and group, summed unreduced in 64-bit
// sums that fold64 folds every fourth group (below 3 * 2^32 + 4 (p - 1)^2 < 2^64).  A warp
// covers 32 consecutive copies of one row group and stages it kP01Stages - 1 groups ahead
// with one 16-byte cp.async per thread (row wl / 8, copies 4 (wl % 8) ..), plus the group's
// scalars (s0..s3) and (t0, t1, s0 + s1, s2 + s3) of each repetition from lanes 0 .. 2R-1;
// after the wait a __syncwarp makes the whole slot visible and each thread reads its
// copy's four values transposed.
constexpr int kP01Stages = 8;
constexpr int kP01Sums = 9;       // E00, E11, QE, F22, F33, QF, U00, U11, QU
constexpr int kP01WarpSlot = 608;  // bytes per warp and stage: 4 rows x 32 copies x 4 B + 6 x 16 B scalars

struct P01Src {
    const uint32_t* v;     // the layer input, 4 ngroups rows
    const uint32_t* s[3];  // s_j: 4 ngroups scalars (s0..s3 of each group)
    const uint32_t* t[3];  // (t0, t1, s0 + s1, s2 + s3) of each group: 4 ngroups scalars
};

// Round 0's evaluations from the nine sums of each repetition, times v(rx); the sums are
// kept canonical in `sums` for round 1.
struct P01Fin {
    RedScratch red;
    uint32_t* out;       // R x 3 x N
    const uint32_t* vx;  // R x N
    uint32_t* sums;      // 9R x N
    uint32_t N, reps;
    __device__ void operator()(uint32_t lane) const {
        for (uint32_t j = 0; j < reps; j++) {
            uint32_t m[kP01Sums];
#pragma unroll
            for (int k = 0; k < kP01Sums; k++) {
                m[k] = take(red, kP01Sums * j + k, N, lane);
                sums[(size_t)(kP01Sums * j + k) * N + lane] = m[k];
            }
            const uint32_t p0 = add(m[0], m[3]), p1 = add(m[1], m[4]), p2raw = add(m[2], m[5]);
            const uint32_t x = vx[(size_t)j * N + lane];
            out[(size_t)(3 * j) * N + lane] = mul(p0, x);
            out[(size_t)(3 * j + 1) * N + lane] = mul(p1, x);
            out[(size_t)(3 * j + 2) * N + lane] = mul(m31::eval_at_two(p0, p1, p2raw), x);
        }
    }
};

template <int R>
__global__ void __launch_bounds__(256, 2) k_p2_round01(P01Src src, uint64_t ngroups, const uint32_t* __restrict__ quads,
                                                       const uint32_t* __restrict__ vx, Geo g, RedScratch red,
                                                       uint32_t* evals_out, uint32_t* sums_out) {
    extern __shared__ uint4 ring01[];  // kP01Stages x warps x kP01WarpSlot bytes
    const uint32_t tid = threadIdx.x, wl = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const uint32_t L = g.tpr, rs = tid / L;  // L: copies per row slice, a multiple of 32
    const uint64_t N = g.N;
    // this warp's first copy, and the 16 bytes the thread stages: row wl / 8 of the group,
    // copies 4 (wl % 8) .. of the warp's 32 (those below N: the sums of the others are dropped)
    const uint64_t warp_lane0 = (uint64_t)blockIdx.y * L + (tid - rs * L - wl);
    const bool active = rs < g.rps && warp_lane0 < N;  // uniform over a warp
    const bool stages = warp_lane0 + 4 * (wl & 7) < N;
    const uint32_t* __restrict__ vst = src.v + (wl >> 3) * N + warp_lane0 + 4 * (wl & 7);
    const uint32_t* __restrict__ sst = nullptr;
    if (wl < 2 * R) {
        const uint32_t j = wl >> 1;
        sst = (wl & 1) ? (j == 0 ? src.t[0] : (j == 1 ? src.t[1] : src.t[2]))
                       : (j == 0 ? src.s[0] : (j == 1 ? src.s[1] : src.s[2]));
    }
    char* const ring = reinterpret_cast<char*>(ring01);
    uint64_t acc[R * kP01Sums];
#pragma unroll
    for (int c = 0; c < R * kP01Sums; c++) acc[c] = 0ull;
    if (active) {
        const uint64_t step = (uint64_t)gridDim.x * g.rps;
        const uint64_t i0 = (uint64_t)blockIdx.x * g.rps + rs;
        // iteration i works on row group q = group_at(quads, i) (rows 4q .. 4q+3); the list
        // entry of the iteration staged next is loaded one iteration ahead of its staging
        auto stage = [&](uint64_t i, uint64_t q, int slot) {
            if (i < ngroups) {
                char* st = ring + ((size_t)slot * nw + w) * kP01WarpSlot;
                if (stages) cp_async16(st + 16 * wl, vst + 4 * q * N);
                if (sst) cp_async16(st + 512 + 16 * wl, sst + 4 * q);
            }
            cp_async_commit();  // one group per iteration, empty past the end
        };
#pragma unroll
        for (int s = 0; s < kP01Stages - 1; s++) {
            const uint64_t i = i0 + s * step;
            stage(i, i < ngroups ? group_at(quads, i) : 0, s);
        }
        uint64_t next_q = i0 + (kP01Stages - 1) * step < ngroups ? group_at(quads, i0 + (kP01Stages - 1) * step) : 0;
        int slot = 0;
        uint32_t it = 0;
        for (uint64_t i = i0; i < ngroups; i += step, it++) {
            __syncwarp();  // every lane has read the slot refilled next
            const uint64_t is = i + (kP01Stages - 1) * step, q = next_q;
            next_q = is + step < ngroups ? group_at(quads, is + step) : 0;
            stage(is, q, slot == 0 ? kP01Stages - 1 : slot - 1);
            cp_async_wait<kP01Stages - 1>();
            __syncwarp();  // the other lanes' copies of this slot are visible
            const char* st = ring + ((size_t)slot * nw + w) * kP01WarpSlot;
            const uint32_t* rows = reinterpret_cast<const uint32_t*>(st);
            const uint32_t x0 = rows[wl], x1 = rows[32 + wl], x2 = rows[64 + wl], x3 = rows[96 + wl];
            const uint4* sc = reinterpret_cast<const uint4*>(st + 512);
            const uint32_t u0 = add(x0, x2), u1 = add(x1, x3), w01 = add(x0, x1), w23 = add(x2, x3), wu = add(u0, u1);
#pragma unroll
            for (int j = 0; j < R; j++) {
                const uint4 sv = sc[2 * j], tv = sc[2 * j + 1];
                uint64_t* a = acc + kP01Sums * j;
                mad64(a[0], x0, sv.x);
                mad64(a[1], x1, sv.y);
                mad64(a[2], w01, tv.z);
                mad64(a[3], x2, sv.z);
                mad64(a[4], x3, sv.w);
                mad64(a[5], w23, tv.w);
                mad64(a[6], u0, tv.x);
                mad64(a[7], u1, tv.y);
                mad64(a[8], wu, add(tv.x, tv.y));
            }
            if ((it & 3) == 3) {
#pragma unroll
                for (int c = 0; c < R * kP01Sums; c++) acc[c] = fold64(acc[c]);
            }
            slot = slot + 1 == kP01Stages ? 0 : slot + 1;
        }
        cp_async_wait<0>();
    }
    uint32_t out[R * kP01Sums];
#pragma unroll
    for (int c = 0; c < R * kP01Sums; c++) out[c] = reduce64(acc[c]);
    __syncthreads();  // the ring is reused as the reduction's scratch
    reduce_group1<R * kP01Sums>(out, g, active, red, P01Fin{red, evals_out, vx, sums_out, g.N, (uint32_t)R});
}

// Round 1 of phase two at the round-0 challenges r_j from the sums of k_p2_round01: block 0
// evaluates every copy's p0_1, p1_1, p2_1 (times v(rx)) and publishes them like a round
// kernel's finisher; the other blocks fold the scalar tables at r_j for round 2,
// s'_j(2i) = fold(s_j(4i), s_j(4i+1), r_j), s'_j(2i+1) = fold(s_j(4i+2), s_j(4i+3), r_j).
struct P1Fold {
    const uint32_t* s[3];
    uint32_t* sd[3];
    uint32_t r[3];
};

__global__ void __launch_bounds__(256) k_p2_round1_fin(const uint32_t* __restrict__ sums, const uint32_t* __restrict__ vx,
                                                       P1Fold f, uint64_t ngroups, uint32_t N, uint32_t reps,
                                                       uint32_t* evals_out, uint32_t* evals_dev, unsigned int* done) {
    const uint32_t tid = threadIdx.x, B = blockDim.x;
    if (blockIdx.x == 0) {
        for (uint32_t j = 0; j < reps; j++) {
            const uint32_t r = j == 0 ? f.r[0] : (j == 1 ? f.r[1] : f.r[2]);
            const uint32_t omr = sub(1u, r);
            const uint32_t c0 = mul(omr, omr), c1 = mul(r, omr), c2 = mul(r, r);
            for (uint32_t lane = tid; lane < N; lane += B) {
                uint32_t m[kP01Sums];
#pragma unroll
                for (int k = 0; k < kP01Sums; k++) m[k] = __ldg(sums + (size_t)(kP01Sums * j + k) * N + lane);
                // the cross sums KE, KF, KU from QE, QF, QU
#pragma unroll
                for (int k = 2; k < kP01Sums; k += 3) m[k] = sub(sub(m[k], m[k - 2]), m[k - 1]);
                const uint32_t p0 = add(add(mul(c0, m[0]), mul(c1, m[2])), mul(c2, m[1]));
                const uint32_t p1 = add(add(mul(c0, m[3]), mul(c1, m[5])), mul(c2, m[4]));
                const uint32_t p2raw = add(add(mul(c0, m[6]), mul(c1, m[8])), mul(c2, m[7]));
                const uint32_t x = __ldg(vx + (size_t)j * N + lane);
                const uint32_t e0 = mul(p0, x), e1 = mul(p1, x), e2 = mul(m31::eval_at_two(p0, p1, p2raw), x);
                evals_out[(size_t)(3 * j) * N + lane] = e0;
                evals_out[(size_t)(3 * j + 1) * N + lane] = e1;
                evals_out[(size_t)(3 * j + 2) * N + lane] = e2;
                if (evals_dev) {
                    evals_dev[(size_t)(3 * j) * N + lane] = e0;
                    evals_dev[(size_t)(3 * j + 1) * N + lane] = e1;
                    evals_dev[(size_t)(3 * j + 2) * N + lane] = e2;
                }
            }
        }
        if (done) {
            __threadfence_system();
            __syncthreads();
            if (tid == 0) atomicAdd_system(done, 1u);
        }
        return;
    }
    const uint64_t total = (uint64_t)reps * ngroups, stride = (uint64_t)(gridDim.x - 1) * B;
    for (uint64_t idx = (uint64_t)(blockIdx.x - 1) * B + tid; idx < total; idx += stride) {
        const uint32_t j = (uint32_t)(idx / ngroups);
        const uint64_t i = idx - (uint64_t)j * ngroups;
        const uint32_t r = j == 0 ? f.r[0] : (j == 1 ? f.r[1] : f.r[2]);
        const uint32_t* sj = j == 0 ? f.s[0] : (j == 1 ? f.s[1] : f.s[2]);
        uint32_t* dj = j == 0 ? f.sd[0] : (j == 1 ? f.sd[1] : f.sd[2]);
        const uint4 sv = __ldg(reinterpret_cast<const uint4*>(sj) + i);
        reinterpret_cast<uint2*>(dj)[i] = make_uint2(fold(sv.x, sv.y, r), fold(sv.z, sv.w, r));
    }
}

// ---------------------------------------------------------------- phase two: s(y)
// s_j[y] = sum over mul gates (z, x, y, c) of eqc_j(z) * eq(rx_j, x) * c: the
// copy-independent factor of h(y) = v(rx) s(y) (sumcheck_helper.hpp:250-259).  With T4 (I a
// multiple of 4) the threads of four neighbouring rows also write t_j(i) =
// (s_j(4i) + s_j(4i+2), s_j(4i+1) + s_j(4i+3), s_j(4i) + s_j(4i+1), s_j(4i+2) + s_j(4i+3)),
// the scalar pair sums that k_p2_round01 stages with each group.
template <bool T4>
__global__ void __launch_bounds__(256) k_s_build(uint64_t I, const uint32_t* __restrict__ my_off,
                                                 const uint4* __restrict__ my_g, const __grid_constant__ EqArgs eqc,
                                                 const __grid_constant__ EqArgs eqx, uint32_t* __restrict__ s_out,
                                                 uint32_t* __restrict__ t_out, uint64_t s_stride) {
    __shared__ uint32_t tz[2 * kEqWords], tx[kEqWords];
    eq_build(tz, eqc);
    eq_build(tx, eqx);
    __syncthreads();
    const uint32_t ndz = eq_digits(eqc), ndx = eq_digits(eqx), reps = eqc.reps;
    const bool two = eqc.f2 != 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    // whole warps go round together: four neighbouring lanes hold a group's rows
    const uint64_t end = (I + 31) & ~31ull;
    for (uint64_t y = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; y < end; y += stride) {
        uint32_t s[3] = {0u, 0u, 0u};
        const uint32_t k0 = y < I ? __ldg(my_off + y) : 0u, k1 = y < I ? __ldg(my_off + y + 1) : 0u;
        for (uint32_t e = k0; e < k1; e++) {
            const uint4 gt = __ldg(my_g + e);  // (x, z, c, 0)
#pragma unroll
            for (uint32_t j = 0; j < 3; j++)
                if (j < reps)
                    s[j] = add(s[j], mul(mul(eq_at(tz, ndz, two, j, gt.y), eq_at(tx, ndx, false, j, gt.x)), gt.z));
        }
#pragma unroll
        for (uint32_t j = 0; j < 3; j++) {
            if (j >= reps) break;
            if (T4) {
                // lane l of a group: t_l = s_0 + s_2, s_1 + s_3, s_0 + s_1, s_2 + s_3
                const uint32_t l = threadIdx.x & 3;
                const uint32_t u = __shfl_sync(0xffffffffu, s[j], l < 2 ? l : 2 * (l - 2), 4);
                const uint32_t w = __shfl_sync(0xffffffffu, s[j], l < 2 ? l + 2 : 2 * (l - 2) + 1, 4);
                if (y < I) t_out[(uint64_t)j * s_stride + y] = add(u, w);
            }
            if (y < I) s_out[(uint64_t)j * s_stride + y] = s[j];
        }
    }
}

// ---------------------------------------------------------------- weighted row sums
// out[j] = sum_z eq(r_j, z) vals[z]: eval_multilinear at r_j for each point
// (include/poly_commit/poly.hpp:88-104).  The table is read once, so the bound is HBM: 2^18
// rows of 1024 copies at three points take 160 us at the copy peak.  Products are summed
// unreduced in 64 bits and folded every four rows (as separate field operations the sums took
// 430 us, bound by instruction issue); a thread stages its next steps of four consecutive rows
// with cp.async, and their weights, computed per block of rows from the digit tables, come from
// shared memory.  (One point, and narrow rows; the others in k_wsum_mma.)  At three points what
// bounds it is the wide multiply-add, 17 products with their folding per
// clock and SM: 235 us at three CTAs an SM and four stages, 256 at four and two or three.
constexpr uint32_t kWsumRows = 256;  // rows of a CTA's weights at a time, at least
constexpr int kWsumStages = 4;       // steps of four rows a thread has in its cp.async ring

__host__ __device__ inline uint32_t wsum_block(const Geo& g, uint64_t rows, uint32_t ctas) {
    const uint32_t step = 4 * g.rps;
    uint64_t per = rows / ((uint64_t)step * (ctas ? ctas : 1));  // small tables: one step a CTA
    const uint32_t most = (kWsumRows + step - 1) / step;
    if (per > most) per = most;
    return step * (per > 1 ? (uint32_t)per : 1u);
}

template <int R>
__global__ void __launch_bounds__(256, 3) k_wsum(const uint32_t* __restrict__ vals, uint64_t rows, uint32_t rb,
                                                 const __grid_constant__ EqArgs eq, Geo g, RedScratch red, uint32_t* out) {
    extern __shared__ uint4 wring[];  // the ring, then R x rb weights; at the end the reduction's scratch
    __shared__ uint32_t tab[kEqWords];
    const TileIdx t = tile_idx(g);
    const uint32_t B = blockDim.x, tid = threadIdx.x;
    uint32_t* const wt = reinterpret_cast<uint32_t*>(wring + kWsumStages * 4 * B);
    eq_build(tab, eq);
    const uint32_t nd = eq_digits(eq);
    uint64_t acc[R][4];
#pragma unroll
    for (int c = 0; c < R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) acc[c][l] = 0ull;
    // blocks of rb rows, taken in turn by the CTAs; within one, steps of 4 rps rows
    const uint64_t stride = (uint64_t)gridDim.x * rb, base = (uint64_t)blockIdx.x * rb;
    const uint32_t step = 4 * g.rps;
    // the step staged next: block offset sz, row si of the block (a table of fewer than four
    // rows repeats its last, weight 0)
    uint64_t sz = base;
    uint32_t si = 4 * t.rs;
    auto stage = [&](int slot) {
        if (t.active && sz < rows) {
            uint4* st = wring + slot * 4 * B + tid;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint64_t z = sz + si + k < rows ? sz + si + k : rows - 1;
                cp_async16(st + k * B, vals + z * g.N + t.lane0);
            }
            si += step;
            if (si >= rb) {
                si = 4 * t.rs;
                sz += stride;
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int q = 0; q < kWsumStages - 1; q++) stage(q);
    int slot = 0;
    for (uint64_t z0 = base; z0 < rows; z0 += stride) {
        __syncthreads();  // the digit tables, or the last block's weights, are done with
        for (uint32_t i = tid; i < rb; i += B)
#pragma unroll
            for (int j = 0; j < R; j++)
                wt[j * rb + i] = z0 + i < rows ? eq_at(tab, nd, false, j, (uint32_t)(z0 + i)) : 0u;
        __syncthreads();
        for (uint32_t i = 4 * t.rs; i < rb; i += step) {
            stage(slot == 0 ? kWsumStages - 1 : slot - 1);
            cp_async_wait<kWsumStages - 1>();
            if (t.active) {
                const uint4* st = wring + slot * 4 * B + tid;
                const uint4 v[4] = {st[0], st[B], st[2 * B], st[3 * B]};
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const uint4 w = *reinterpret_cast<const uint4*>(wt + j * rb + i);
#pragma unroll
                    for (int l = 0; l < 4; l++) {
#pragma unroll
                        for (int k = 0; k < 4; k++) mad64(acc[j][l], comp(v[k], l), comp(w, k));
                        acc[j][l] = fold64(acc[j][l]);
                    }
                }
            }
            slot = slot + 1 == kWsumStages ? 0 : slot + 1;
        }
    }
    cp_async_wait<0>();
    uint32_t sum[R][4];
#pragma unroll
    for (int c = 0; c < R; c++)
#pragma unroll
        for (int l = 0; l < 4; l++) sum[c][l] = reduce64(acc[c][l]);
    __syncthreads();  // the ring is the reduction's scratch
    reduce_group<R>(sum, g, t.active, red, 0, CopyFin{red, out, g.N, (uint32_t)R});
}

// Two or three points on wide rows: the same sums as a contraction on the tensor cores, exact.
// With v = sum_d 2^(8d) b_d(v) over its four bytes, sum_z v[z] w[z] is the sum over (z, d) of
// b_d(v[z]) times 2^(8d) w[z] mod p (a rotation of w's 31 bits), whose bytes are again 2^(8e)
// apart: for every copy, a sum for each point and byte e over k = (row, digit) of products of two
// bytes.  A byte widened with zeros is the subnormal 16-bit float b 2^-24, the products are
// multiples of 2^-48 in the 32-bit sums, and a sum of the 256 products of 64 rows is at most
// 256 * 255^2 < 2^24 of them: no sum is rounded before it goes on to the integers.
// mma.sync m16n8k16: the k index may be any order of the (row, digit) pairs, so a thread's four
// k are one row's digits, two byte permutes a value; the four copies of its 16 bytes are rows g
// and g + 8 of two tiles.  A value costs a thread one MMA instruction and those two permutes,
// where k_wsum has three wide multiply-adds and their folding: 2^18 rows of 1024 copies at three
// points 235 -> 192 us (5.6 TB/s; without the MMAs 193, so what is left is memory).
// (tcgen05 would need the digits in shared memory first; the tensor cores are a third used.)
constexpr uint32_t kWmmaRows = 128;               // rows of a CTA's weights at a time, at most
constexpr uint32_t kWmmaExact = 64;               // rows between conversions of the sums
constexpr int kWmmaStages = 3;                    // steps of four rows a thread has in its cp.async ring
constexpr uint32_t kWmmaWords = 32;               // words of a row's weights (16 columns x 4 digits)

__device__ __forceinline__ uint32_t rot31(uint32_t x, uint32_t s) {  // 2^s x mod p, 0 <= s < 31
    return ((x << s) & m31::P) | (x >> (31 - s));
}
// Two bytes of x (sel 0x4140: the low ones, 0x4342: the high ones) as 16-bit floats, each b 2^-24:
// a byte widened with zeros is that subnormal number.
__device__ __forceinline__ uint32_t half2_bytes(uint32_t x, uint32_t sel) { return __byte_perm(x, 0u, sel); }
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// wc: groups of 32 copies a CTA takes (a divisor of 8), a warp each; 8 / wc warps share a group's
// rows, 16 at a time.  rb: rows a block, a multiple of 16 * 8 / wc.
template <int R>
__global__ void __launch_bounds__(256, 3) k_wsum_mma(const uint32_t* __restrict__ vals, uint64_t rows, uint32_t rb,
                                                     const __grid_constant__ EqArgs eq, uint32_t N, uint32_t wc,
                                                     RedScratch red, uint32_t* out) {
    constexpr int T = (R + 1) / 2;  // tiles of eight columns, two points each
    extern __shared__ uint4 wmma_sm[];  // rb rows of weights, the ring; at the end partial sums
    __shared__ uint32_t tab[kEqWords];
    uint4* const ring = wmma_sm + rb * (kWmmaWords / 4);
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, row8 = lane >> 2, c = lane & 3;
    const uint32_t cg = w % wc, slice = w / wc, step = 16 * (8 / wc);
    eq_build(tab, eq);
    const uint32_t nd = eq_digits(eq);
    float s[2][T][4] = {};      // [copies 2m, 2m+1 of the four][columns 8t ..]
    uint32_t acc[2][T][4] = {};
    auto convert = [&](bool reduce) {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int t = 0; t < T; t++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    acc[m][t][k] += __float2uint_rn(s[m][t][k] * 281474976710656.0f);  // 2^48
                    if (reduce) acc[m][t][k] = m31::from_u32(acc[m][t][k]);
                    s[m][t][k] = 0.0f;
                }
    };
    const uint64_t stride = (uint64_t)gridDim.x * rb, base = (uint64_t)blockIdx.x * rb;
    // The ring's next step: `step` rows from row si of the block at sz on, a row's copies by
    // neighbouring threads.  (With 128 bytes of four rows a warp, each for itself and without a
    // barrier, memory gave 3.75 TB/s.)  Row r's quad q is at q ^ 2 (r mod 4), which spreads the
    // four rows and two quads that eight threads read over all banks.
    uint64_t sz = base;
    uint32_t si = 0;
    const uint32_t rowq = 8 * wc, first = blockIdx.y * rowq;  // quads a row; the CTA's first
    const uint32_t sr = tid / rowq, sq = tid % rowq, per = 256 / rowq;  // rows sr, sr + per, ..
    const bool stages = 4 * (first + sq) < N;
    const uint32_t* from = vals + base * N + 4 * (first + sq);
    uint32_t off[4];  // words from `from` (a table of less than a step's rows repeats its last, weight 0)
    uint4* to[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t r = sr + k * per;
        off[k] = (r < rows ? r : (uint32_t)rows - 1) * N;
        to[k] = ring + r * rowq + (sq ^ 2 * (r & 3));
    }
    auto stage = [&](int slot) {
        if (sz < rows) {
            if (stages)
#pragma unroll
                for (int k = 0; k < 4; k++) cp_async16(to[k] + slot * 1024, from + off[k]);
            si += step;
            from += (uint64_t)step * N;
            if (si >= rb) {
                si = 0;
                sz += stride;
                from += (stride - rb) * N;
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int q = 0; q < kWmmaStages - 1; q++) stage(q);
    int slot = 0;
    uint32_t since = 0, reduced = 0;
    for (uint64_t z0 = base; z0 < rows; z0 += stride) {
        __syncthreads();  // the digit tables are built, or the last block's weights are done with
        for (uint32_t i = tid; i < rb * 4; i += blockDim.x) {
            const uint32_t z = i >> 2, j = i & 3;  // j >= R: the columns of no point
            uint32_t wd[4];
            wd[0] = j < R && z0 + z < rows ? eq_at(tab, nd, false, j, (uint32_t)(z0 + z)) : 0u;
#pragma unroll
            for (int d = 1; d < 4; d++) wd[d] = rot31(wd[0], 8 * d);
            // 16 bytes per place and row, the four rows of a step that a place's threads read side by side
            uint32_t* to = reinterpret_cast<uint32_t*>(wmma_sm + (z >> 2) * 32 + 16 * (j & 1) + (z & 3)) + 2 * (j >> 1);
#pragma unroll
            for (int e = 0; e < 4; e++) {  // column 4j + e: tile j / 2, place 4 (j % 2) + e
                const uint32_t sel = e | (e + 4) << 4;
                *reinterpret_cast<uint2*>(to + 16 * e) = make_uint2(half2_bytes(__byte_perm(wd[0], wd[1], sel), 0x4140),
                                                                   half2_bytes(__byte_perm(wd[2], wd[3], sel), 0x4140));
            }
        }
        __syncthreads();
        for (uint32_t i = 16 * slice; i < rb; i += step) {
            cp_async_wait<kWmmaStages - 2>();
            __syncthreads();  // the step is there, and every warp is done with the one before
            stage(slot == 0 ? kWmmaStages - 1 : slot - 1);
            uint4 v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) v[k] = ring[slot * 1024 + (16 * slice + 4 * k + c) * rowq + ((8 * cg + row8) ^ 2 * c)];
            slot = slot + 1 == kWmmaStages ? 0 : slot + 1;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint4 b = wmma_sm[(i / 4 + k) * 32 + lane];
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const uint32_t x = comp(v[k], 2 * m), y = comp(v[k], 2 * m + 1);
                    const uint32_t a[4] = {half2_bytes(x, 0x4140), half2_bytes(y, 0x4140), half2_bytes(x, 0x4342),
                                           half2_bytes(y, 0x4342)};
                    mma16816(s[m][0], a, b.x, b.y);
                    if (T > 1) mma16816(s[m][T - 1], a, b.z, b.w);
                }
            }
            since += 16;
            if (since == kWmmaExact) {
                since = 0;
                convert((++reduced & 63) == 0);  // 64 x 2^24 + 2^31 < 2^32
            }
        }
    }
    cp_async_wait<0>();
    convert(true);
    // 2^(8e) shares of a copy and point are in two neighbouring threads
    uint32_t* const part = reinterpret_cast<uint32_t*>(wmma_sm);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int t = 0; t < T; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t e = 16 * (c & 1), j = 2 * t + (c >> 1);
                uint32_t x = add(rot31(acc[m][t][2 * h], e), rot31(acc[m][t][2 * h + 1], e + 8));
                x = add(x, __shfl_xor_sync(0xffffffffu, x, 1));
                if (!(c & 1) && j < R) part[j * 256 + 32 * w + 4 * row8 + 2 * m + h] = x;
            }
    __syncthreads();
    uint32_t sum[R];
#pragma unroll
    for (int j = 0; j < R; j++) sum[j] = part[256 * j + tid];
    __syncthreads();
    Geo g;
    g.N = N;
    g.tpr = 32 * wc;
    g.rps = 8 / wc;
    reduce_group1<R>(sum, g, true, red, CopyFin{red, out, N, (uint32_t)R});
}

// k_p2_round01 on the tensor cores, exact in the same way.  Row 4q + e of a group meets four
// coefficients of each repetition: its own s and its neighbour's (s_e, s_(e^1)), which make E or F
// and their cross sums, and the two pair sums t0 = s0 + s2, t1 = s1 + s3, which make U and its
// cross sum: [s_e, s_(e^1), t_(e&1), t_(1-(e&1))], each with four bytes.  A warp takes the rows of
// one e for 32 copies, an MMA step four of its groups (k = group and digit), so a group costs it
// twelve MMAs for three repetitions where a thread a copy had 27 wide multiply-adds, their folding
// and the coefficients' loads, 224 instructions a group and warp.
// The CTA stages the next steps' rows (64 copies) and coefficients with cp.async, and turns the
// next step's coefficients into bytes while it multiplies this one's.  The integer sums are in
// shared memory (a conversion every 64 groups), since with the float sums they would not leave
// two CTAs their registers.  Three repetitions of 2^17 rows of 1024 copies, 14.8 thousand groups
// with gates: 197 -> 114 us, four layers of 2^20 rows 3.6 -> 2.3 ms; the tensor cores are active
// 39% of it, the rest is the barrier a step and the conversions.
constexpr int kP01mStages = 4;
constexpr uint32_t kP01mGroups = 8;  // groups of a step
constexpr uint32_t kP01mCopies = 64;
template <int R>
constexpr uint32_t p01m_smem() {
    return 2 * R * 8 * 256 * 4 + 2 * 2 * 6 * R * 16 * 8 + kP01mStages * (512 + 16 * R) * 16;
}

template <int R>
__global__ void __launch_bounds__(256, 2) k_p2_round01_mma(P01Src src, uint32_t ngroups, const uint32_t* __restrict__ quads,
                                                           const uint32_t* __restrict__ vx, uint32_t N, RedScratch red,
                                                           uint32_t* evals_out, uint32_t* sums_out) {
    constexpr int U = 4 * R, T = 2 * R;                // units of four columns (coefficient, repetition); tiles of two
    constexpr uint32_t kSub = 6 * R * 16, kSlot = 512 + 16 * R;
    extern __shared__ uint4 p01m[];
    uint32_t* const sums = reinterpret_cast<uint32_t*>(p01m) + threadIdx.x;     // T * 8 words a thread
    uint2* const bytes = reinterpret_cast<uint2*>(p01m + T * 8 * 64);            // [2][2 steps of four groups][kSub]
    uint4* const ring = reinterpret_cast<uint4*>(bytes + 4 * kSub);
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, row8 = lane >> 2, c = lane & 3;
    const uint32_t e = w & 3, cg = w >> 2, copy0 = blockIdx.y * kP01mCopies;
#pragma unroll
    for (int k = 0; k < T * 8; k++) sums[256 * k] = 0u;
    float s[2][T][4] = {};
    uint32_t since = 0, reduced = 0;
    auto convert = [&](bool reduce) {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int t = 0; t < T; t++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    uint32_t* p = sums + 256 * ((m * T + t) * 4 + k);
                    const uint32_t x = *p + __float2uint_rn(s[m][t][k] * 281474976710656.0f);  // 2^48
                    *p = reduce ? m31::from_u32(x) : x;
                    s[m][t][k] = 0.0f;
                }
    };
    // what a thread stages of a step: 16 bytes of row (tid / 16) % 4 of two groups, and of one
    // repetition's s or t of a group
    const uint32_t vg = tid >> 6, ve = (tid >> 4) & 3, piece = tid & 15, sg = tid / (2 * R), sr = tid % (2 * R);
    const bool any = ngroups > 0, stages = any && copy0 + 4 * piece < N, scalars = any && tid < 16 * R;
    const uint32_t* const vfrom = src.v + (uint64_t)ve * N + copy0 + 4 * piece;
    const uint32_t sj = sr >> 1;
    const uint32_t* const sfrom = (sr & 1) ? (sj == 0 ? src.t[0] : (sj == 1 ? src.t[1] : src.t[2]))
                                           : (sj == 0 ? src.s[0] : (sj == 1 ? src.s[1] : src.s[2]));
    // the first group of the step staged next, and those of its groups in the list (past the
    // last group the last one's data are staged again, with no coefficients: build)
    const uint32_t stride = gridDim.x * kP01mGroups, last = ngroups - 1;
    uint32_t is = blockIdx.x * kP01mGroups, ga = 0, gb = 0, gs = 0;
    auto look = [&] {
        if (!any) return;
        ga = (uint32_t)group_at(quads, min(is + vg, last));
        gb = (uint32_t)group_at(quads, min(is + vg + 4, last));
        if (scalars) gs = (uint32_t)group_at(quads, min(is + sg, last));
        is = is < ngroups ? is + stride : is;
    };
    uint4* const vto = ring + (vg * 4 + ve) * 16 + (piece ^ 2 * vg);
    auto stage = [&](int slot) {
        if (stages) {
            cp_async16(vto + slot * kSlot, vfrom + (uint64_t)ga * (4 * N));
            cp_async16(vto + slot * kSlot + 256, vfrom + (uint64_t)gb * (4 * N));
        }
        if (scalars) cp_async16(ring + slot * kSlot + 512 + tid, sfrom + (uint64_t)gs * 4);
        cp_async_commit();
        look();
    };
    // the bytes of the coefficients of the step at group i (slot) into buffer `buf`; none past the last group
    const uint32_t bg = tid & 7, bc = tid >> 3;  // group, coefficient x repetition
    const uint32_t kappa = bc / R;
    const uint32_t* const bfrom =
        reinterpret_cast<const uint32_t*>(ring + 512 + bg * 2 * R + 2 * (bc % R) + (kappa >> 2)) + (kappa & 3);
    uint2* const bto = bytes + (bg >> 2) * kSub + bc * 16 + (bg & 3);
    auto build = [&](uint32_t i, int slot, uint32_t buf) {
        if (bc >= 6 * R) return;
        uint32_t wd[4];
        wd[0] = i + bg < ngroups ? bfrom[slot * (4 * kSlot)] : 0u;
#pragma unroll
        for (int d = 1; d < 4; d++) wd[d] = rot31(wd[0], 8 * d);
        uint2* const to = bto + buf * 2 * kSub;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint32_t sel = b | (b + 4) << 4;
            to[4 * b] = make_uint2(half2_bytes(__byte_perm(wd[0], wd[1], sel), 0x4140),
                                   half2_bytes(__byte_perm(wd[2], wd[3], sel), 0x4140));
        }
    };
    uint32_t ko[T];  // this thread's bytes of each tile
#pragma unroll
    for (int t = 0; t < T; t++) {
        const uint32_t u = 2 * t + (row8 >> 2), f = u / R, j = u % R;
        const uint32_t x = f < 2 ? e ^ f : 4 + ((f ^ e) & 1);
        ko[t] = ((x * R + j) * 4 + (row8 & 3)) * 4 + c;
    }
    look();
#pragma unroll
    for (int q = 0; q < kP01mStages - 1; q++) stage(q);
    cp_async_wait<kP01mStages - 2>();
    __syncthreads();
    build(blockIdx.x * kP01mGroups, 0, 0);
    int slot = 0;
    uint32_t buf = 0;
    for (uint32_t i = blockIdx.x * kP01mGroups; i < ngroups; i += stride) {
        const int after = slot + 1 == kP01mStages ? 0 : slot + 1;
        cp_async_wait<kP01mStages - 3>();
        __syncthreads();  // this step's bytes and the next step's data are there, the last one is done with
        stage(slot == 0 ? kP01mStages - 1 : slot - 1);
        build(i + stride, after, buf ^ 1);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint4 v = ring[slot * kSlot + ((4 * h + c) * 4 + e) * 16 + ((8 * cg + row8) ^ 2 * c)];
            uint32_t a[2][4];
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const uint32_t x = comp(v, 2 * m), y = comp(v, 2 * m + 1);
                a[m][0] = half2_bytes(x, 0x4140);
                a[m][1] = half2_bytes(y, 0x4140);
                a[m][2] = half2_bytes(x, 0x4342);
                a[m][3] = half2_bytes(y, 0x4342);
            }
#pragma unroll
            for (int t = 0; t < T; t++) {
                const uint2 b = bytes[(buf * 2 + h) * kSub + ko[t]];
                mma16816(s[0][t], a[0], b.x, b.y);
                mma16816(s[1][t], a[1], b.x, b.y);
            }
        }
        since += kP01mGroups;
        if (since == 64) {
            since = 0;
            convert((++reduced & 63) == 0);
        }
        slot = after;
        buf ^= 1;
    }
    cp_async_wait<0>();
    convert(true);
    __syncthreads();  // the ring takes every (e, unit, copy)'s total
    uint32_t* const part = reinterpret_cast<uint32_t*>(ring);
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int t = 0; t < T; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t* p = sums + 256 * ((m * T + t) * 4 + 2 * h), sh = 16 * (c & 1);
                uint32_t x = add(rot31(p[0], sh), rot31(p[256], sh + 8));
                x = add(x, __shfl_xor_sync(0xffffffffu, x, 1));
                if (!(c & 1)) part[(e * U + 2 * t + (c >> 1)) * kP01mCopies + 32 * cg + 4 * row8 + 2 * m + h] = x;
            }
    __syncthreads();
    // the nine sums: coefficients (row e, place f) whose totals they add
    constexpr uint16_t kAdds[kP01Sums] = {0x0001, 0x0010, 0x0033, 0x0100, 0x1000, 0x3300, 0x0404, 0x4040, 0xcccc};
    for (uint32_t o = tid; o < kP01Sums * R * kP01mCopies; o += 256) {
        const uint32_t q = o & (kP01mCopies - 1), kj = o / kP01mCopies, k = kj / R, j = kj - k * R;
        uint32_t adds = 0;
#pragma unroll
        for (int i = 0; i < kP01Sums; i++)
            if (i == (int)k) adds = kAdds[i];
        unsigned long long total = 0;
        for (uint32_t i = 0; i < 16; i++)
            if (adds >> i & 1) total += part[((i >> 2) * U + (i & 3) * R + j) * kP01mCopies + q];
        if (copy0 + q < N) atomicAdd(&red.acc[(size_t)(kP01Sums * j + k) * N + copy0 + q], total);
    }
    P01Fin fin{red, evals_out, vx, sums_out, N, (uint32_t)R};
    finish_group(red, copy0, kP01mCopies, N, fin);
}

// CTAs of 256 threads for n threads of a kernel that builds digit tables: one wave at most, a
// CTA more costs another build.
uint32_t grid_eq(uint64_t n) {
    const uint64_t b = (n + 255) / 256;
    return (uint32_t)(b < 1 ? 1 : b < 152 * 8 ? b : 152 * 8);
}

uint32_t grid_1d(uint64_t n, uint32_t block) {
    uint64_t b = (n + block - 1) / block;
    if (b < 1) b = 1;
    if (b > 152ull * 16) b = 152ull * 16;
    return (uint32_t)b;
}

// Row tile with repetition-split CTAs: gridDim.x = reps x row chunks.
LaunchShape rep_shape(const Geo& g, uint64_t rows, uint32_t block, uint32_t ctas_cap, uint32_t reps,
                      uint32_t smem_components = 2) {
    LaunchShape s = row_shape(g, rows, block, ctas_cap / reps, smem_components);
    s.grid.x *= reps;
    return s;
}

}  // namespace

// Row iterations a thread of a reducing kernel makes at least (when the table has that many
// rows): each CTA ends with a reduction epilogue (shared-memory sums, one 64-bit atomic per
// component and copy, the last-CTA finisher), which small grids pay less often.
constexpr uint32_t kMinRowIters = 4;

LaunchShape row_shape(const Geo& g, uint64_t rows, uint32_t block, uint32_t ctas_cap, uint32_t smem_components) {
    LaunchShape s;
    const uint32_t groups = lane_groups(g);
    uint64_t need = (rows + (uint64_t)g.rps * kMinRowIters - 1) / ((uint64_t)g.rps * kMinRowIters);
    uint64_t cap = ctas_cap / groups;
    if (cap < 1) cap = 1;
    if (need < 1) need = 1;
    s.grid = dim3((uint32_t)(need < cap ? need : cap), groups, 1);
    s.block = dim3(block, 1, 1);
    s.smem = (size_t)smem_components * 4 * block * sizeof(uint32_t);
    return s;
}

cudaError_t launch_check_canonical(const uint32_t* v, uint64_t n, unsigned int* flag, cudaStream_t s) {
    k_check_canonical<<<grid_1d(n / 4, 256), 256, 0, s>>>(v, n, flag);
    return cudaGetLastError();
}

cudaError_t launch_evaluate(const uint32_t* in, uint32_t* out, uint64_t O, const uint4* ev, const uint32_t* mo_off,
                            const uint4* mo_g, const uint32_t* ao_off, const uint2* ao_g, const Geo& g, uint32_t block,
                            uint32_t ctas, cudaStream_t s) {
    LaunchShape sh = row_shape(g, O, block, ctas, 0);
    k_evaluate<<<sh.grid, sh.block, 0, s>>>(in, out, O, ev, mo_off, mo_g, ao_off, ao_g, g);
    return cudaGetLastError();
}

cudaError_t launch_canonicalize(uint32_t* v, uint64_t n, cudaStream_t s) {
    k_canonicalize<<<grid_1d(n, 256), 256, 0, s>>>(v, n);
    return cudaGetLastError();
}
cudaError_t launch_gate_sums(bool mul_gates, uint64_t O, const uint32_t* off, const uint32_t* gates, const GateEq& eq,
                             unsigned long long* acc, unsigned int* ticket, uint32_t* out, cudaStream_t s) {
    if (eq.z.reps < 1 || eq.z.reps > 3) return cudaErrorInvalidValue;
    const uint32_t grid = grid_eq(O);
    if (mul_gates)
        k_gate_sums<true><<<grid, 256, 0, s>>>(O, off, gates, eq, acc, ticket, out);
    else
        k_gate_sums<false><<<grid, 256, 0, s>>>(O, off, gates, eq, acc, ticket, out);
    return cudaGetLastError();
}

cudaError_t launch_scale_weights(uint64_t I, const uint32_t* mx_off, const uint4* w4, uint4* w4r, const uint32_t r[3],
                                 int reps, cudaStream_t s) {
    if (reps < 1 || reps > 3) return cudaErrorInvalidValue;
    const uint4 rr = make_uint4(r[0], reps > 1 ? r[1] : 0u, reps > 2 ? r[2] : 0u, 0u);
    k_scale_weights<<<grid_1d(I, 256), 256, 0, s>>>(I, mx_off, w4, w4r, rr);
    return cudaGetLastError();
}

cudaError_t launch_weights(uint64_t I, uint64_t Gm, const EqArgs& eqc, const uint4* mx_g, const uint32_t* ax_off,
                           const uint2* ax_g, uint4* a_out, uint4* w_out, cudaStream_t s) {
    k_weights<<<grid_eq(I > Gm ? I : Gm), 256, 0, s>>>(I, Gm, eqc, mx_g, ax_off, ax_g, a_out, w_out);
    return cudaGetLastError();
}

cudaError_t launch_hg_build(const uint32_t* v, uint32_t I, uint32_t N, uint32_t tpr, const EqArgs& eqc,
                            const uint32_t* mx_off, const uint4* mx_g, const uint32_t* ax_off, const uint2* ax_g,
                            const uint4* a4, const uint4* w4, uint4* priv, size_t priv_stride, cudaStream_t s) {
    const uint32_t grid = grid_eq((uint64_t)I * (N / 4));
    if (a4)
        k_hg_build<true><<<grid, 256, 0, s>>>(v, I, N, tpr, eqc, mx_off, mx_g, ax_off, ax_g, a4, w4, priv, priv_stride);
    else
        k_hg_build<false><<<grid, 256, 0, s>>>(v, I, N, tpr, eqc, mx_off, mx_g, ax_off, ax_g, a4, w4, priv, priv_stride);
    return cudaGetLastError();
}

// p with its fold weights; `both` when hr[0] (round 0's challenges), `r1` when hr[1] rather than
// r follows it.
static RoundPtrs with_weights(const RoundPtrs& p, int reps, bool both, bool r1 = false) {
    RoundPtrs q = p;
    for (int j = 0; j < reps; j++) {
        q.c[j] = m31::lerp_at(p.r[j]);
        if (!both) continue;
        q.c0[j] = m31::lerp_at(p.hr[0][j]);
        q.c01[j] = m31::lerp2_at(p.hr[0][j], r1 ? p.hr[1][j] : p.r[j]);
    }
    return q;
}

// Dynamic shared memory of k_hg_round0: the cp.async ring, or the reduction's scratch where
// that is larger (they share the allocation).  Above 48 KiB less the kernel's static shared
// memory a launch needs the opt-in, which is set once per device and instantiation to the
// largest size any launch asks for (block <= 256).
template <int R>
static size_t hg0_smem(size_t ring_bytes, size_t red_bytes) {
    static std::atomic<uint64_t> opted{0};  // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(opted.load(std::memory_order_relaxed) & bit)) {
        cudaFuncSetAttribute(k_hg_round0<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxStagedSmem);
        opted.fetch_or(bit);
    }
    return ring_bytes > red_bytes ? ring_bytes : red_bytes;
}

// Dynamic shared memory of a kernel with a row ring (kRowRingSmem at most): the opt-in above
// 48 KiB is set once per device and kernel (one instance of this function per kernel).
template <auto Kernel>
static size_t ring_smem(size_t bytes) {
    static std::atomic<uint64_t> opted{0};  // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(opted.load(std::memory_order_relaxed) & bit)) {
        cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowRingSmem);
        opted.fetch_or(bit);
    }
    return bytes;
}

uint32_t launch_stage_words(uint32_t* dst, const uint32_t* const* srcs, uint32_t nsrc, uint64_t n, unsigned int* done,
                            cudaStream_t s, cudaError_t* err) {
    const uint64_t total = n * nsrc;
    uint64_t ctas = (total + 256 * 16 - 1) / (256 * 16);
    if (ctas < 1) ctas = 1;
    if (ctas > 64) ctas = 64;
    k_stage_words<<<(uint32_t)ctas, 256, 0, s>>>(dst, srcs[0], nsrc > 1 ? srcs[1] : nullptr,
                                                 nsrc > 2 ? srcs[2] : nullptr, nsrc, n, done);
    *err = cudaGetLastError();
    return (uint32_t)ctas;
}

cudaError_t launch_hg_round0(int reps, const uint32_t* v, uint64_t npairs, const uint32_t* pairs,
                             const uint32_t* mx_off, const uint4* mx_g, const uint4* a4, const uint4* w4, const Geo& g,
                             uint32_t block, uint32_t ctas, RedScratch red, const uint32_t* claim,
                             uint32_t* evals_out, cudaStream_t s) {
    if (!claim) return cudaErrorInvalidValue;
    // the kernel's launch bound is 256 threads: wider tiles are narrowed to it
    Geo gb = g;
    if (block > 256) block = 256;
    while (gb.tpr > block && gb.tpr % 2 == 0) gb.tpr /= 2;
    if (gb.tpr > block) return cudaErrorInvalidValue;
    gb.rps = block / gb.tpr;
    LaunchShape sh = row_shape(gb, npairs, block, ctas, 2 * reps);
    const size_t ring = (size_t)kStages * kStageFields * sizeof(uint4) * block;
#define GKR_HG0(RR)                                                                                                \
    k_hg_round0<RR><<<sh.grid, sh.block, hg0_smem<RR>(ring, sh.smem), s>>>(v, npairs, pairs, mx_off, mx_g, a4, w4, \
                                                                          gb, red, claim, evals_out)
    switch (reps) {
        case 1: GKR_HG0(1); break;
        case 2: GKR_HG0(2); break;
        case 3: GKR_HG0(3); break;
        default: return cudaErrorInvalidValue;
    }
#undef GKR_HG0
    return cudaGetLastError();
}

cudaError_t launch_hg_round1(int reps, const uint32_t* v, uint64_t npairs, const uint32_t* quads,
                             const uint32_t* mx_off, const uint4* mx_g, const uint4* a4, const uint4* w4r,
                             const RoundPtrs& p, const Geo& g, uint32_t block, uint32_t ctas, RedScratch red,
                             uint32_t* evals_out, cudaStream_t s) {
    if (quads && p.fdst[0]) return cudaErrorInvalidValue;  // stored folded copies need every pair
    if (!red.evals_dev) return cudaErrorInvalidValue;       // the claim is round 0's polynomial
    if (reps < 1 || reps > 3) return cudaErrorInvalidValue;
    const RoundPtrs q = with_weights(p, reps, false);
    LaunchShape sh = row_shape(g, npairs, block, ctas, 2 * reps);
#define GKR_HG1(RR) \
    k_hg_round1<RR><<<sh.grid, sh.block, sh.smem, s>>>(v, npairs, quads, mx_off, mx_g, a4, w4r, q, g, red, evals_out)
    switch (reps) {
        case 1: GKR_HG1(1); break;
        case 2: GKR_HG1(2); break;
        case 3: GKR_HG1(3); break;
        default: return cudaErrorInvalidValue;
    }
#undef GKR_HG1
    return cudaGetLastError();
}

// Shared-memory opt-in of k_p2_round0 (as hg0_smem): once per device and instantiation.
template <int R>
static size_t p2_smem(size_t bytes) {
    static std::atomic<uint64_t> opted{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(opted.load(std::memory_order_relaxed) & bit)) {
        cudaFuncSetAttribute(k_p2_round0<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxP2Smem);
        opted.fetch_or(bit);
    }
    return bytes;
}

cudaError_t launch_round(int reps, bool shared_src, bool lane_hg, bool fold_, const RoundPtrs& p, uint64_t npairs,
                         const uint32_t* vx, const Geo& g, uint32_t block, uint32_t ctas, RedScratch red,
                         uint32_t* evals_out, cudaStream_t s) {
    if (reps < 1 || reps > 3) return cudaErrorInvalidValue;
    if (lane_hg && !fold_) return cudaErrorInvalidValue;  // phase-one round 0 lives in k_hg_round0
    if (!fold_ && !shared_src) return cudaErrorInvalidValue;
    if (!fold_) {
        // phase-two round 0 (k_p2_round0): launch bound 256 threads, wider tiles narrowed
        Geo gb = g;
        uint32_t b = block > 256 ? 256 : block;
        while (gb.tpr > b && gb.tpr % 2 == 0) gb.tpr /= 2;
        if (gb.tpr > b) return cudaErrorInvalidValue;
        gb.rps = b / gb.tpr;
        const LaunchShape sh = row_shape(gb, npairs, b, ctas, 3 * reps);
        const size_t ring = (size_t)kP2Stages * kP2Fields * sizeof(uint4) * b;
        const size_t smem = ring > sh.smem ? ring : sh.smem;
        const P2Src src{p.fsrc[0], {p.hsrc[0], p.hsrc[1], p.hsrc[2]}};
        switch (reps) {
            case 1: k_p2_round0<1><<<sh.grid, sh.block, p2_smem<1>(smem), s>>>(src, npairs, vx, gb, red, evals_out); break;
            case 2: k_p2_round0<2><<<sh.grid, sh.block, p2_smem<2>(smem), s>>>(src, npairs, vx, gb, red, evals_out); break;
            default: k_p2_round0<3><<<sh.grid, sh.block, p2_smem<3>(smem), s>>>(src, npairs, vx, gb, red, evals_out); break;
        }
        return cudaGetLastError();
    }
    const RoundPtrs pw = with_weights(p, reps, false);
    if (!red.evals_dev) return cudaErrorInvalidValue;  // fold rounds take their claim from it
    if (shared_src) {
        // one read of the shared layer input for all repetitions
        LaunchShape sh = row_shape(g, npairs, block, ctas, 2 * reps);
#define GKR_SHARED(RR, LH, FO) k_round_shared<RR, LH, FO><<<sh.grid, sh.block, sh.smem, s>>>(pw, npairs, vx, g, red, evals_out)
#define GKR_SHARED_R(RR)                                  \
    if (lane_hg) GKR_SHARED(RR, true, true);              \
    else GKR_SHARED(RR, false, true);
        switch (reps) {
            case 1: GKR_SHARED_R(1) break;
            case 2: GKR_SHARED_R(2) break;
            default: GKR_SHARED_R(3) break;
        }
#undef GKR_SHARED_R
#undef GKR_SHARED
        return cudaGetLastError();
    }
    LaunchShape sh = rep_shape(g, npairs, block, ctas, reps);
#define GKR_ROUND(SH, LH, FO) k_round<SH, LH, FO><<<sh.grid, sh.block, sh.smem, s>>>(pw, npairs, vx, g, reps, red, evals_out)
    if (lane_hg) GKR_ROUND(false, true, true);
    else GKR_ROUND(false, false, true);
#undef GKR_ROUND
    return cudaGetLastError();
}

cudaError_t launch_round_hr(int round, int reps, const RoundPtrs& p, uint64_t npairs, const Geo& g, uint32_t block,
                            uint32_t ctas, RedScratch red, uint32_t* evals_out, cudaStream_t s) {
    if (reps < 1 || reps > 3 || !p.hoff || !p.ha || (round != 2 && round != 3) || !red.evals_dev)
        return cudaErrorInvalidValue;
    const RoundPtrs q = with_weights(p, reps, true, true);
    LaunchShape sh = rep_shape(g, npairs, block, ctas, reps);
    if (round == 2)
        k_round<false, true, true, 1><<<sh.grid, sh.block, sh.smem, s>>>(q, npairs, nullptr, g, reps, red, evals_out);
    else
        k_round<false, true, true, 2><<<sh.grid, sh.block, sh.smem, s>>>(q, npairs, nullptr, g, reps, red, evals_out);
    return cudaGetLastError();
}

cudaError_t launch_round_pair(int reps, bool lane_hg, int depth, const RoundPtrs& p, uint64_t ngroups,
                              const uint32_t* vx, const Geo& g, uint32_t block, uint32_t ctas, RedScratch red,
                              uint32_t* evals_out, uint32_t* sums_out, cudaStream_t s) {
    if (reps < 1 || reps > 3 || block > 256 || !red.evals_dev || !sums_out || ngroups < 1 || (!lane_hg && !vx) ||
        (lane_hg && depth == 1 && (!p.hoff || !p.ha)))
        return cudaErrorInvalidValue;
    const RoundPtrs q = with_weights(p, reps, lane_hg || depth == 2, depth == 1);
    const LaunchShape sh = rep_shape(g, ngroups, block, ctas, reps, kPairSums);
#define GKR_PAIR(LH, D, HR) \
    k_round_pair<LH, D, HR><<<sh.grid, sh.block, sh.smem, s>>>(q, ngroups, vx, g, reps, red, evals_out, sums_out)
    if (depth == 1 && lane_hg) GKR_PAIR(true, 1, 2);
    else if (depth == 1) GKR_PAIR(false, 1, 0);
    else if (depth == 2 && lane_hg) GKR_PAIR(true, 2, 0);
    else if (depth == 2) GKR_PAIR(false, 2, 0);
    else return cudaErrorInvalidValue;
#undef GKR_PAIR
    return cudaGetLastError();
}

uint32_t pair_fin_ctas(int reps, uint32_t N) { return (uint32_t)(((uint64_t)reps * N + 255) / 256); }

cudaError_t launch_pair_fin(int reps, bool lane_hg, const RoundPtrs& p, const uint32_t* sums, const uint32_t* vx,
                            uint32_t rows, uint32_t N, uint32_t* evals_out, uint32_t* evals_dev, unsigned int* done,
                            cudaStream_t s) {
    if (reps < 1 || reps > 3 || !evals_dev || (!lane_hg && !vx)) return cudaErrorInvalidValue;
    const uint32_t ctas = pair_fin_ctas(reps, N);
    if (lane_hg)
        k_pair_fin<true><<<ctas, 256, 0, s>>>(p, sums, vx, rows, N, (uint32_t)reps, evals_out, evals_dev, done);
    else
        k_pair_fin<false><<<ctas, 256, 0, s>>>(p, sums, vx, rows, N, (uint32_t)reps, evals_out, evals_dev, done);
    return cudaGetLastError();
}

cudaError_t launch_p1_round2(int reps, const RoundPtrs& p, uint64_t npairs, const Geo& g, uint32_t block,
                             uint32_t ctas, RedScratch red, uint32_t* evals_out, cudaStream_t s) {
    if (!p.hoff || !p.ha || !red.evals_dev) return cudaErrorInvalidValue;
    if (reps < 1 || reps > 3) return cudaErrorInvalidValue;
    const RoundPtrs q = with_weights(p, reps, true);
    LaunchShape sh = row_shape(g, npairs, block, ctas, 2 * reps);
    switch (reps) {
        case 1: k_p1_round2<1><<<sh.grid, sh.block, sh.smem, s>>>(q, npairs, g, red, evals_out); break;
        case 2: k_p1_round2<2><<<sh.grid, sh.block, sh.smem, s>>>(q, npairs, g, red, evals_out); break;
        case 3: k_p1_round2<3><<<sh.grid, sh.block, sh.smem, s>>>(q, npairs, g, red, evals_out); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_p2_round2(int reps, const RoundPtrs& p, uint64_t npairs, const uint32_t* vx, const Geo& g,
                             uint32_t block, uint32_t ctas, RedScratch red, uint32_t* evals_out, cudaStream_t s) {
    if (!red.evals_dev || block > 256) return cudaErrorInvalidValue;
    if (reps < 1 || reps > 3) return cudaErrorInvalidValue;
    const RoundPtrs q = with_weights(p, reps, true);
    LaunchShape sh = row_shape(g, npairs, block, ctas, 2 * reps);
    const size_t ring = (size_t)kRowStages * 8 * sizeof(uint4) * block;
    const size_t smem = ring > sh.smem ? ring : sh.smem;
    switch (reps) {
        case 1: k_p2_round2<1><<<sh.grid, sh.block, ring_smem<k_p2_round2<1>>(smem), s>>>(q, npairs, vx, g, red, evals_out); break;
        case 2: k_p2_round2<2><<<sh.grid, sh.block, ring_smem<k_p2_round2<2>>(smem), s>>>(q, npairs, vx, g, red, evals_out); break;
        case 3: k_p2_round2<3><<<sh.grid, sh.block, ring_smem<k_p2_round2<3>>(smem), s>>>(q, npairs, vx, g, red, evals_out); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Copies per row slice of the one-copy-per-thread kernel: the multiple of 32 up to 256 that
// keeps most of the threads at work (the last slice of a row, and the threads of a CTA that
// make no whole slice, stay idle), the widest of those; 0 where less than half would work.
static uint32_t one_copy_slice(uint32_t N) {
    uint32_t best = 0;
    uint64_t best_used = 0;  // of 256 x slices threads, N copies are of use
    for (uint32_t L = 32; L <= 256; L += 32) {
        const uint32_t slices = (N + L - 1) / L;
        const uint64_t used = (uint64_t)N * (256 / L) * 65536 / ((uint64_t)slices * 256);
        if (slices <= 1024 && used >= best_used) best = L, best_used = used;  // a ticket per slice
    }
    return best_used * 2 >= 65536 ? best : 0;
}

// Groups of copies of k_p2_round01_mma; 0 where more than an eighth of a CTA's would be past the end.
static uint32_t p01m_groups(uint32_t N) {
    const uint32_t ny = (N + kP01mCopies - 1) / kP01mCopies;
    return (uint64_t)N * 8 >= (uint64_t)ny * kP01mCopies * 7 && ny <= 1024 ? ny : 0;
}

uint32_t p2_round01_groups(uint32_t N) {
    if (const uint32_t ny = p01m_groups(N)) return ny;
    const uint32_t L = one_copy_slice(N);
    return L ? (N + L - 1) / L : 0;
}

cudaError_t launch_p2_round01(int reps, const uint32_t* v, const uint32_t* const* s, const uint32_t* const* t,
                              uint64_t ngroups, const uint32_t* quads, const uint32_t* vx, uint32_t N, uint32_t ctas,
                              RedScratch red, uint32_t* evals_out, uint32_t* sums_out, cudaStream_t st) {
    if (reps < 1 || reps > 3 || p2_round01_groups(N) == 0) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(v) & 15) != 0) return cudaErrorInvalidValue;  // 16-byte cp.async
    P01Src src;
    src.v = v;
    for (int j = 0; j < 3; j++) {
        src.s[j] = j < reps ? s[j] : nullptr;
        src.t[j] = j < reps ? t[j] : nullptr;
    }
    if (const uint32_t ny = p01m_groups(N)) {
        const uint64_t nsteps = (ngroups + kP01mGroups - 1) / kP01mGroups, cap2 = ctas / 2 / ny ? ctas / 2 / ny : 1;
        const dim3 gm((uint32_t)(nsteps < 1 ? 1 : nsteps < cap2 ? nsteps : cap2), ny);
#define GKR_P01M(RR) \
    k_p2_round01_mma<RR><<<gm, 256, ring_smem<k_p2_round01_mma<RR>>(p01m_smem<RR>()), st>>>(src, (uint32_t)ngroups, quads, vx, N, red, \
                                                                                           evals_out, sums_out)
        switch (reps) {
            case 1: GKR_P01M(1); break;
            case 2: GKR_P01M(2); break;
            default: GKR_P01M(3); break;
        }
#undef GKR_P01M
        return cudaGetLastError();
    }
    Geo g;
    g.N = N;
    g.tpr = one_copy_slice(N);
    g.rps = 256 / g.tpr;
    const uint32_t groups = p2_round01_groups(N);
    uint64_t need = (ngroups + (uint64_t)g.rps * kMinRowIters - 1) / ((uint64_t)g.rps * kMinRowIters), cap = ctas / groups;
    if (cap < 1) cap = 1;
    if (need < 1) need = 1;
    const dim3 grid((uint32_t)(need < cap ? need : cap), groups, 1);
    const size_t ring = (size_t)kP01Stages * 8 * kP01WarpSlot, red_b = (size_t)3 * kP01Sums * 4 * 256;
    const size_t smem = ring > red_b ? ring : red_b;
    switch (reps) {
        case 1: k_p2_round01<1><<<grid, 256, smem, st>>>(src, ngroups, quads, vx, g, red, evals_out, sums_out); break;
        case 2: k_p2_round01<2><<<grid, 256, smem, st>>>(src, ngroups, quads, vx, g, red, evals_out, sums_out); break;
        default: k_p2_round01<3><<<grid, 256, smem, st>>>(src, ngroups, quads, vx, g, red, evals_out, sums_out); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_p2_round1_fin(int reps, const uint32_t* sums, const uint32_t* vx, const uint32_t* const* s,
                                 uint32_t* const* sd, const uint32_t* r, uint64_t ngroups, uint32_t N,
                                 uint32_t* evals_out, uint32_t* evals_dev, unsigned int* done, cudaStream_t st) {
    if (reps < 1 || reps > 3) return cudaErrorInvalidValue;
    P1Fold f;
    for (int j = 0; j < 3; j++) {
        f.s[j] = j < reps ? s[j] : nullptr;
        f.sd[j] = j < reps ? sd[j] : nullptr;
        f.r[j] = j < reps ? r[j] : 0u;
    }
    const uint32_t fold_blocks = grid_1d((uint64_t)reps * ngroups, 256);
    k_p2_round1_fin<<<1 + fold_blocks, 256, 0, st>>>(sums, vx, f, ngroups, N, (uint32_t)reps, evals_out, evals_dev,
                                                      done);
    return cudaGetLastError();
}

cudaError_t launch_s_build(uint64_t I, const uint32_t* my_off, const uint4* my_g, const EqArgs& eqc, const EqArgs& eqx,
                           uint32_t* s_out, uint32_t* t_out, uint64_t s_stride, cudaStream_t s) {
    if (t_out && (I % 4 || s_stride % 4)) return cudaErrorInvalidValue;
    if (t_out)
        k_s_build<true><<<grid_eq(I), 256, 0, s>>>(I, my_off, my_g, eqc, eqx, s_out, t_out, s_stride);
    else
        k_s_build<false><<<grid_eq(I), 256, 0, s>>>(I, my_off, my_g, eqc, eqx, s_out, nullptr, s_stride);
    return cudaGetLastError();
}

// Groups of 32 copies a CTA of k_wsum_mma takes; 0: k_wsum.  From two points on, where its
// copies are a kilobyte or the whole of a row (128 bytes of each of 2^18 rows of 200 copies took
// 93 us against 72) and at most an eighth of its threads' are past the end.  One point is memory
// bound either way (2^18 rows of 1024 copies: 189 us both) and smaller tables are faster with the
// narrow kernel's shorter blocks (2^14 rows 28 against 32 us).
static uint32_t wmma_groups(uint32_t reps, uint32_t N) {
    if (reps < 2) return 0;
    const uint32_t cgs = (N + 31) / 32;
    for (uint32_t wc = 8; wc > 1; wc /= 2) {
        const uint32_t ny = (cgs + wc - 1) / wc;
        if ((wc == 8 || ny == 1) && (uint64_t)N * 8 >= (uint64_t)ny * wc * 32 * 7 && ny <= 1024) return wc;
    }
    return 0;
}

uint32_t wsum_groups(const EqArgs& eq, const Geo& g) {
    const uint32_t wc = wmma_groups(eq.reps, g.N);
    return wc ? (g.N + 32 * wc - 1) / (32 * wc) : lane_groups(g);
}

cudaError_t launch_wsum(const uint32_t* vals, const EqArgs& eq, const Geo& g, uint32_t block, uint32_t ctas,
                        RedScratch red, uint32_t* out, cudaStream_t s) {
    const uint64_t rows = 1ull << eq.nvars;
    if (const uint32_t wc = wmma_groups(eq.reps, g.N)) {
        const uint32_t ny = (g.N + 32 * wc - 1) / (32 * wc), step = 16 * (8 / wc), cap2 = ctas / ny ? ctas / ny : 1;
        uint32_t rbm = step;  // a power of two, as the rows are
        while (2 * rbm <= kWmmaRows && (uint64_t)2 * rbm * cap2 <= rows) rbm *= 2;
        const uint64_t nb = (rows + rbm - 1) / rbm;
        // (the partial sums and the reduction's scratch, 3 KB, are less than the ring)
        const size_t sm = (size_t)rbm * kWmmaWords * 4 + (size_t)kWmmaStages * 4 * 16 * 256;
        const dim3 gm((uint32_t)(nb < cap2 ? nb : cap2), ny);
        switch (eq.reps) {
            case 2: k_wsum_mma<2><<<gm, 256, ring_smem<k_wsum_mma<2>>(sm), s>>>(vals, rows, rbm, eq, g.N, wc, red, out); break;
            default: k_wsum_mma<3><<<gm, 256, ring_smem<k_wsum_mma<3>>(sm), s>>>(vals, rows, rbm, eq, g.N, wc, red, out); break;
        }
        return cudaGetLastError();
    }
    const uint32_t groups = lane_groups(g), cap = ctas / groups ? ctas / groups : 1, rb = wsum_block(g, rows, cap);
    const uint64_t need = (rows + rb - 1) / rb;
    const dim3 grid((uint32_t)(need < cap ? need : cap), groups, 1);
    if (block > 256 || eq.reps < 1 || eq.reps > 3) return cudaErrorInvalidValue;
    // (the reduction's scratch, 16 reps bytes a thread, is less than the ring)
    const size_t smem = (size_t)kWsumStages * 4 * 16 * block + 4 * (size_t)eq.reps * rb;
    switch (eq.reps) {
        case 1: k_wsum<1><<<grid, block, ring_smem<k_wsum<1>>(smem), s>>>(vals, rows, rb, eq, g, red, out); break;
        case 2: k_wsum<2><<<grid, block, ring_smem<k_wsum<2>>(smem), s>>>(vals, rows, rb, eq, g, red, out); break;
        case 3: k_wsum<3><<<grid, block, ring_smem<k_wsum<3>>(smem), s>>>(vals, rows, rb, eq, g, red, out); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace gkrgpu
