// GPU-assisted verifier (M31: Verifier, BN254: BnVerifier): Verifier::verify (include/LinearGKR/LinearGKR.hpp:
// 105-149), gkr_verify (include/LinearGKR/gkr.hpp:75-122) and sumcheck_verify_gkr_layer
// (include/LinearGKR/sumcheck.hpp:113-176).  Part of prover.cu's translation unit (included
// inside its anonymous namespace after the provers, whose lanes and circuit it uses).
//
// The host replays the transcript (the same SHA-256 schedule as the prover) and does the
// per-lane round checks; the device does what scales with the circuit and the input: the
// gate sums of eval_sparse_circuit_connect_poly
// (include/LinearGKR/sumcheck_verifier_utils.hpp:22-56) per layer, and RawPC::verify's
// eval_multilinear of the whole committed input at rz1_j and rz2_j (include/poly_commit/
// raw.hpp:75-78, include/poly_commit/poly.hpp:88-104).
//
// Decisions follow the reference: proof values are read with from_bytes (reduced mod p), the
// proof's grinding bytes are skipped rather than compared (LinearGKR.hpp:121-124), bytes
// after the last claim are ignored, and a proof that runs out is rejected.
#pragma once

struct Verifier {
    gkrgpu_ctx& X;
    Lane& c;
    const gkrgpu_circuit& C;
    uint32_t N;
    int R;
    char* block = nullptr;
    uint32_t* com = nullptr;
    unsigned long long *gacc = nullptr, *wacc = nullptr;
    unsigned int *gticket = nullptr, *wticket = nullptr;

    Verifier(gkrgpu_ctx& ctx, Lane& lane, const gkrgpu_circuit& circ, uint32_t n, int reps)
        : X(ctx), c(lane), C(circ), N(n), R(reps) {}
    ~Verifier() {
        if (block) cudaFreeAsync(block, c.stream);
    }

    void reserve() {
        size_t o = 0;
        std::vector<std::pair<void**, size_t>> parts = {
            {(void**)&com, C.in_rows(0) * N * 4}, {(void**)&gacc, 3 * 8}, {(void**)&gticket, 16},
            {(void**)&wacc, 9ull * N * 8},        {(void**)&wticket, 4096},
        };
        size_t zero_from = 0;
        for (auto& p : parts) {
            if (p.first == (void**)&gacc) zero_from = o;
            o += align_up(std::max<size_t>(p.second, 16), 256);
        }
        void* base = nullptr;
        ck(cudaMallocFromPoolAsync(&base, o, X.pool, c.stream), "verifier workspace allocation");
        block = static_cast<char*>(base);
        o = 0;
        for (auto& p : parts) {
            *p.first = block + o;
            o += align_up(std::max<size_t>(p.second, 16), 256);
        }
        ck(cudaMemsetAsync(block + zero_from, 0, o - zero_from, c.stream), "cudaMemsetAsync");
        c.ensure_mapped(0, 4 * (claims_word() + 6ull * N));
    }

    // Results in the lane's mapped extra area (words): each layer's add and mul gate sums (4
    // each), then the input's evaluations at rz1_j and rz2_j (3N each).
    uint64_t claims_word() const { return align_up(8ull * C.layers.size(), 64); }
    uint32_t* mapped(bool dev, uint64_t word) const {
        return reinterpret_cast<uint32_t*>(dev ? c.extra_d() : c.extra_h()) + word;
    }
    uint64_t sums_word(size_t li, bool mul_part) const { return 8ull * li + (mul_part ? 4 : 0); }

    // eval_sparse_circuit_connect_poly of layer li for every repetition: the add part (needs
    // rx) or the mul part (needs rx and ry).  No challenge depends on it, so it is only launched
    // here; the checks that use it are made at the end, after one wait for the device.
    void gate_sums(size_t li, bool mul_part, uint32_t (*rz1)[32], uint32_t (*rz2)[32], uint32_t alpha, uint32_t beta,
                   uint32_t (*rx)[32], uint32_t (*ry)[32]) {
        const DevLayer& Ly = C.layers[li];
        const uint64_t O = 1ull << Ly.nout;
        GateEq eq;
        eq.z = eq_args(R, rz1, rz2, alpha, beta, Ly.nout);
        eq.x = eq_args(R, rx, nullptr, 1u, 0u, Ly.nin);
        eq.y = mul_part ? eq_args(R, ry, nullptr, 1u, 0u, Ly.nin) : eq.x;
        const double gates = mul_part ? (double)Ly.nmul : (double)Ly.nadd;
        c.launch(K_GATE_SUMS, (mul_part ? 16.0 : 8.0) * gates + 4.0 * (O + 1), [&] {
            return launch_gate_sums(mul_part, O, mul_part ? Ly.mo_off : Ly.ao_off,
                                    mul_part ? reinterpret_cast<const uint32_t*>(Ly.mo_g)
                                             : reinterpret_cast<const uint32_t*>(Ly.ao_g),
                                    eq, gacc, gticket, mapped(true, sums_word(li, mul_part)), c.stream);
        });
    }

    // eval_multilinear of the committed input at the R points r[j], into the claims area.
    void raw_pc_eval(uint32_t (*r)[32], int which) {
        const uint32_t n0 = C.layers[0].nin;
        c.launch(K_WSUM, 4.0 * N * (double)(1ull << n0), [&] {
            return launch_wsum(com, eq_args(R, r, nullptr, 1u, 0u, n0), X.geo(N, K_WSUM), X.block,
                               X.cta_budget(K_WSUM), RedScratch{wacc, wticket},
                               mapped(true, claims_word() + 3ull * N * which), c.stream);
        });
    }

    // What a layer's checks need once its gate sums are known, R x N each: the running sum
    // less p(0) + p(1) at phase two's first round, which must be vx * add sum, and the last
    // running sum, which must be vx * vy * mul sum.
    struct Pending {
        std::vector<uint32_t> first, last, vx, vy;
    };

    bool run(int grinding_bits, const uint8_t* proof, uint64_t len, const uint32_t* claimed_v) {
        const uint64_t rowb = (uint64_t)N * 4;
        const uint64_t com_bytes = C.in_rows(0) * rowb;
        if (len < com_bytes + 32) return false;
        reserve();
        c.copy(com, proof, com_bytes, cudaMemcpyHostToDevice, "commitment upload");
        c.launch(K_CANONICAL, 8.0 * C.in_rows(0) * N, [&] { return launch_canonicalize(com, C.in_rows(0) * N, c.stream); });

        // transcript: the commitment bytes (hashed in place), grinding
        std::unique_ptr<uint8_t[]> tbuf(new uint8_t[len]);  // each row at its own place in the proof
        Transcript t(tbuf.get(), len, X.fs_hash);
        uint8_t d[32];
        fs_hash(X.fs_hash, proof, com_bytes, d);
        t.appended_prehashed(com_bytes, d);
        grind(t, grinding_bits);
        uint64_t pos = com_bytes + 32;
        // Proof::get_next_and_step of one row (N lanes), reduced, to the transcript's tail + at;
        // false, with nothing written, when the proof has run out
        auto next_row = [&](uint64_t at) {
            if (len - pos < rowb) return false;
            uint32_t* out = reinterpret_cast<uint32_t*>(t.tail() + at);
            memcpy(out, proof + pos, rowb);
            for (uint32_t k = 0; k < N; k++) out[k] = m31::from_u32(out[k]);
            pos += rowb;
            return true;
        };
        // The rejection of a proof that has run out, made at once: what was launched is waited for,
        // since it reads the proof and writes the lane's mapped area.
        auto ran_out = [&] {
            c.sync();
            c.resolve_events();
            return false;
        };

        const size_t L = C.layers.size();
        uint32_t rz1[3][32], rz2[3][32], rx[3][32], ry[3][32];
        memset(rz1, 0, sizeof(rz1));
        memset(rz2, 0, sizeof(rz2));
        const uint32_t nz = C.layers[L - 1].nout;
        for (uint32_t i = 0; i < nz; i++)
            for (int j = 0; j < R; j++) rz1[j][i] = t.challenge();
        uint32_t alpha = 1, beta = 0;
        const size_t RN = (size_t)R * N;
        std::vector<uint32_t> cv1(RN), cv2(RN, 0u), sum(RN);
        for (size_t i = 0; i < RN; i++) cv1[i] = m31::from_u32(claimed_v[i]);
        std::vector<Pending> pending(L);
        bool ok = true;

        for (int li = (int)L - 1; li >= 0; li--) {
            const uint32_t n = C.layers[li].nin;
            Pending& pd = pending[li];
            pd.first.resize(RN);
            pd.vx.resize(RN);
            pd.vy.resize(RN);
            for (size_t i = 0; i < RN; i++) sum[i] = m31::add(m31::mul(cv1[i], alpha), m31::mul(cv2[i], beta));
            for (uint32_t i_var = 0; i_var < 2 * n; i_var++) {
                // the rounds' rows, and vx after each repetition's challenge in phase one's last
                const bool vx_round = i_var == n - 1;
                uint32_t rs[3];
                const uint8_t* ev0 = t.tail();
                if (!vx_round) {
                    for (int q = 0; q < 3 * R; q++)
                        if (!next_row(q * rowb)) return ran_out();
                    t.challenge_each(3 * rowb, R, rs);
                } else {
                    for (int j = 0; j < R; j++) {
                        for (int q = 0; q < 3; q++)
                            if (!next_row(q * rowb)) return ran_out();
                        t.appended(3 * rowb);
                        rs[j] = t.challenge();
                        if (!next_row(0)) return ran_out();
                        memcpy(pd.vx.data() + (size_t)j * N, t.tail(), rowb);
                        t.appended(rowb);
                    }
                }
                for (int j = 0; j < R; j++) {
                    const uint32_t* ev = reinterpret_cast<const uint32_t*>(ev0 + (vx_round ? 4 : 3) * j * rowb);
                    const uint32_t r = rs[j];
                    (i_var < n ? rx[j][i_var] : ry[j][i_var - n]) = r;
                    uint32_t* s = sum.data() + (size_t)j * N;
                    uint32_t off = 0;
                    for (uint32_t k = 0; k < N; k++) {
                        const uint32_t left = m31::sub(s[k], m31::add(ev[k], ev[N + k]));
                        if (i_var == n) pd.first[(size_t)j * N + k] = left;
                        else off |= left;
                        s[k] = m31::eval_degree2(ev[k], ev[N + k], ev[2 * N + k], r);
                    }
                    if (off) ok = false;
                }
                if (vx_round) gate_sums((size_t)li, false, rz1, rz2, alpha, beta, rx, ry);
            }
            for (int j = 0; j < R; j++) {
                if (!next_row(0)) return ran_out();
                memcpy(pd.vy.data() + (size_t)j * N, t.tail(), rowb);
                t.appended(rowb);
            }
            gate_sums((size_t)li, true, rz1, rz2, alpha, beta, rx, ry);
            pd.last = sum;
            alpha = t.challenge();
            beta = t.challenge();
            for (int j = 0; j < R; j++) {
                memcpy(rz1[j], rx[j], 4 * n);
                memcpy(rz2[j], ry[j], 4 * n);
            }
            cv1 = pd.vx;
            cv2 = pd.vy;
        }
        // RawPC::verify against the commitment, at rz1_j and rz2_j
        raw_pc_eval(rz1, 0);
        raw_pc_eval(rz2, 1);
        c.sync();
        std::atomic_thread_fence(std::memory_order_acquire);
        c.came_back(4ull * R * (2 * L + 2ull * N));
        for (size_t li = 0; li < L && ok; li++) {
            const uint32_t *a = mapped(false, sums_word(li, false)), *m = mapped(false, sums_word(li, true));
            const Pending& pd = pending[li];
            for (size_t i = 0; i < RN; i++) {
                const size_t j = i / N;
                if (pd.first[i] != m31::mul(pd.vx[i], a[j])) ok = false;
                if (pd.last[i] != m31::mul(m31::mul(pd.vx[i], pd.vy[i]), m[j])) ok = false;
            }
        }
        const uint32_t* ev = mapped(false, claims_word());
        if (ok) ok = memcmp(ev, cv1.data(), RN * 4) == 0 && memcmp(ev + 3ull * N, cv2.data(), RN * 4) == 0;
        c.resolve_events();
        return ok;
    }
};

// The same verifier for BN254 circuits (one repetition; field operations of fr_host.hpp on
// canonical values on the host, Montgomery tables on the device).
struct BnVerifier {
    gkrgpu_ctx& X;
    Lane& c;
    const gkrgpu_circuit& C;
    uint32_t N;
    char* block = nullptr;
    uint32_t *raw = nullptr, *com = nullptr, *sums = nullptr, *cv = nullptr;
    unsigned long long *gacc = nullptr, *wacc = nullptr;
    unsigned int *gticket = nullptr, *wticket = nullptr;

    BnVerifier(gkrgpu_ctx& ctx, Lane& lane, const gkrgpu_circuit& circ, uint32_t n) : X(ctx), c(lane), C(circ), N(n) {}
    ~BnVerifier() {
        if (block) cudaFreeAsync(block, c.stream);
    }

    void reserve() {
        const uint64_t I0 = C.in_rows(0);
        std::vector<std::pair<void**, size_t>> parts = {
            {(void**)&raw, I0 * N * 32},   {(void**)&com, I0 * N * 32}, {(void**)&sums, 32},
            {(void**)&cv, (size_t)N * 32}, {(void**)&gacc, 8 * 8},      {(void**)&gticket, 16},
            {(void**)&wacc, 3ull * N * 8 * 8}, {(void**)&wticket, 4096},
        };
        size_t o = 0, zero_from = 0;
        for (auto& p : parts) {
            if (p.first == (void**)&gacc) zero_from = o;
            o += align_up(std::max<size_t>(p.second, 16), 256);
        }
        void* base = nullptr;
        ck(cudaMallocFromPoolAsync(&base, o, X.pool, c.stream), "verifier workspace allocation");
        block = static_cast<char*>(base);
        o = 0;
        for (auto& p : parts) {
            *p.first = block + o;
            o += align_up(std::max<size_t>(p.second, 16), 256);
        }
        ck(cudaMemsetAsync(block + zero_from, 0, o - zero_from, c.stream), "cudaMemsetAsync");
        c.h_cv.ensure((size_t)N * 32 + 64, "pinned verifier results");
    }

    frh::Fr gate_sums(size_t li, bool mul_part, const frh::Fr* rz1, const frh::Fr* rz2, const frh::Fr& alpha,
                      const frh::Fr& beta, const frh::Fr* rx, const frh::Fr* ry) {
        const DevLayer& Ly = C.layers[li];
        const uint64_t O = 1ull << Ly.nout;
        const frh::Fr one = frh::from_u32(1), zero = frh::zero();
        bn::GateEqBn eq;
        eq.z = eq_args_bn(rz1, rz2, alpha, beta, Ly.nout);
        eq.x = eq_args_bn(rx, nullptr, one, zero, Ly.nin);
        eq.y = mul_part ? eq_args_bn(ry, nullptr, one, zero, Ly.nin) : eq.x;
        const double gates = mul_part ? (double)Ly.nmul : (double)Ly.nadd;
        c.launch(K_GATE_SUMS, (mul_part ? 48.0 : 40.0) * gates + 4.0 * (O + 1) + 32.0 * O, [&] {
            return bn::launch_gate_sums(mul_part, O, mul_part ? Ly.mo_off : Ly.ao_off,
                                        mul_part ? reinterpret_cast<const uint32_t*>(Ly.mo_g)
                                                 : reinterpret_cast<const uint32_t*>(Ly.ao_g),
                                        mul_part ? Ly.mo_c : Ly.ao_c, eq, gacc, gticket, sums, c.stream);
        });
        c.copy(c.h_cv.p, sums, 32, cudaMemcpyDeviceToHost, "gate sums readback");
        c.sync();
        return frh::load(c.h_cv.as<uint32_t>());
    }

    bool raw_pc_verify(const frh::Fr* r, const std::vector<uint32_t>& claims) {
        const uint32_t n0 = C.layers[0].nin;
        const uint64_t rows = 1ull << n0;
        const bn::EqArgsBn eq = eq_args_bn(r, nullptr, frh::from_u32(1), frh::zero(), n0);
        const bn::GeoBn g = geo_bn(X, N, K_BN_WSUM);
        c.launch(K_BN_WSUM, 32.0 * N * rows, [&] {
            return bn::launch_wsum(com, eq, g, X.cta_budget(K_BN_WSUM), bn::RedBn{wacc, wticket}, cv, c.stream);
        });
        c.copy(c.h_cv.p, cv, (size_t)N * 32, cudaMemcpyDeviceToHost, "multilinear evaluation readback");
        c.sync();
        return memcmp(c.h_cv.p, claims.data(), (size_t)N * 32) == 0;
    }

    bool run(int grinding_bits, const uint8_t* proof, uint64_t len, const uint32_t* claimed_v) {
        const uint64_t rowb = (uint64_t)N * 32, rowl = (uint64_t)N * 8;
        const uint64_t com_bytes = C.in_rows(0) * rowb;
        if (len < com_bytes + 32) return false;
        reserve();
        c.copy(raw, proof, com_bytes, cudaMemcpyHostToDevice, "commitment upload");
        c.launch(K_BN_LOAD, 64.0 * C.in_rows(0) * N,
                 [&] { return bn::launch_load(raw, com, C.in_rows(0) * N, nullptr, c.stream); });

        std::unique_ptr<uint8_t[]> tbuf(new uint8_t[len]);  // each row at its own place in the proof
        Transcript t(tbuf.get(), len, X.fs_hash);
        uint8_t d[32];
        fs_hash(X.fs_hash, proof, com_bytes, d);
        t.appended_prehashed(com_bytes, d);
        grind_bn254(t, grinding_bits);
        uint64_t pos = com_bytes + 32;
        // one row of N canonical elements (from_bytes reduces each 32-byte word); false when the
        // proof has run out, which is rejected at once, as above
        auto next_row = [&](uint32_t* out) {
            if (len - pos < rowb) return false;
            for (uint32_t k = 0; k < N; k++) frh::store(frh::from_bytes(proof + pos + 32ull * k), out + 8ull * k);
            pos += rowb;
            return true;
        };
        auto ran_out = [&] {
            c.sync();
            c.resolve_events();
            return false;
        };
        auto el = [](const std::vector<uint32_t>& v, uint64_t row, uint32_t N_, uint32_t k) {
            return frh::load(v.data() + (row * N_ + k) * 8);
        };

        const size_t L = C.layers.size();
        frh::Fr rz1[32], rz2[32], rx[32], ry[32];
        const uint32_t nz = C.layers[L - 1].nout;
        for (uint32_t i = 0; i < nz; i++) rz1[i] = t.challenge_bn254();
        frh::Fr alpha = frh::from_u32(1), beta = frh::zero();
        bool have_rz2 = false;
        std::vector<uint32_t> cv1(rowl), cv2(rowl, 0u), vx(rowl), vy(rowl), ev(3 * rowl);
        std::vector<frh::Fr> sum(N);
        for (uint32_t k = 0; k < N; k++) {
            uint8_t b[32];
            memcpy(b, claimed_v + 8ull * k, 32);
            frh::store(frh::from_bytes(b), cv1.data() + 8ull * k);
        }
        const frh::Fr inv2{{frh::kInv2[0], frh::kInv2[1], frh::kInv2[2], frh::kInv2[3]}};
        bool ok = true;

        for (int li = (int)L - 1; li >= 0; li--) {
            const uint32_t n = C.layers[li].nin;
            for (uint32_t k = 0; k < N; k++)
                sum[k] = frh::add(frh::mul(el(cv1, 0, N, k), alpha), frh::mul(el(cv2, 0, N, k), beta));
            for (uint32_t i_var = 0; i_var < 2 * n; i_var++) {
                for (int q = 0; q < 3; q++)
                    if (!next_row(ev.data() + q * rowl)) return ran_out();
                t.append(ev.data(), 3 * rowb);
                const frh::Fr r = t.challenge_bn254();
                (i_var < n ? rx[i_var] : ry[i_var - n]) = r;
                for (uint32_t k = 0; k < N; k++) {
                    // degree_2_eval (sumcheck_verifier_utils.hpp:10-18)
                    const frh::Fr c0 = el(ev, 0, N, k), v1 = el(ev, 1, N, k), v2 = el(ev, 2, N, k);
                    if (!frh::eq(frh::add(c0, v1), sum[k])) ok = false;
                    const frh::Fr c2 = frh::mul(inv2, frh::add(frh::sub(v2, frh::add(v1, v1)), c0));
                    const frh::Fr c1 = frh::sub(frh::sub(v1, c0), c2);
                    sum[k] = frh::add(c0, frh::mul(frh::add(frh::mul(c2, r), c1), r));
                }
                if (i_var == n - 1) {
                    if (!next_row(vx.data())) return ran_out();
                    t.append(vx.data(), rowb);
                    const frh::Fr a = gate_sums((size_t)li, false, rz1, have_rz2 ? rz2 : nullptr, alpha, beta, rx, ry);
                    for (uint32_t k = 0; k < N; k++) sum[k] = frh::sub(sum[k], frh::mul(el(vx, 0, N, k), a));
                }
            }
            if (!next_row(vy.data())) return ran_out();
            t.append(vy.data(), rowb);
            const frh::Fr m = gate_sums((size_t)li, true, rz1, have_rz2 ? rz2 : nullptr, alpha, beta, rx, ry);
            for (uint32_t k = 0; k < N; k++)
                if (!frh::eq(sum[k], frh::mul(frh::mul(el(vx, 0, N, k), el(vy, 0, N, k)), m))) ok = false;
            alpha = t.challenge_bn254();
            beta = t.challenge_bn254();
            for (uint32_t i = 0; i < n; i++) {
                rz1[i] = rx[i];
                rz2[i] = ry[i];
            }
            have_rz2 = true;
            cv1 = vx;
            cv2 = vy;
        }
        if (!raw_pc_verify(rz1, cv1)) ok = false;
        if (!raw_pc_verify(rz2, cv2)) ok = false;
        c.resolve_events();
        return ok;
    }
};
