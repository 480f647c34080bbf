// M31 field arithmetic (p = 2^31 - 1) for host and device.
//
// Every function maps canonical inputs in [0, p) to the canonical result, which is the
// value the reference's scalar and packed operators produce (include/field/M31.hpp:64-93,
// include/field/M31_avx.tcc:97-176): field results are unique, so the proof bytes do
// not depend on how a sum is ordered or split across threads.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define GKR_HD __host__ __device__ __forceinline__
#else
#define GKR_HD inline
#endif

namespace m31 {

static constexpr uint32_t P = 2147483647u;

GKR_HD uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }

// a + b: the sum is < 2^32; min(s, s - p) picks s - p exactly when s >= p.
GKR_HD uint32_t add(uint32_t a, uint32_t b) {
    uint32_t s = a + b;
    return umin(s, s - P);
}

// a - b: d wraps to a value > p when a < b, and then d + p (mod 2^32) is the smaller one.
GKR_HD uint32_t sub(uint32_t a, uint32_t b) {
    uint32_t d = a - b;
    return umin(d, d + P);
}

// Mersenne reduction of a 62-bit product: x = hi * 2^31 + lo == hi + lo (mod p).
// lo + hi <= p + 2^31 - 2 < 2p, so one conditional subtraction finishes it.
GKR_HD uint32_t reduce62(uint64_t x) {
    uint32_t s = (uint32_t)(x & P) + (uint32_t)(x >> 31);
    return umin(s, s - P);
}

// a * b, formed as a * 2b: the product's high word is then (a b) >> 31 and half its low word
// (a b) mod 2^31, one shift-and-add apart (reduce62 of the plain product takes a mask, a
// 64-bit shift and an add).
GKR_HD uint32_t mul(uint32_t a, uint32_t b) {
    const uint64_t t = (uint64_t)a * (b + b);
    const uint32_t s = (uint32_t)(t >> 32) + ((uint32_t)t >> 1);
    return umin(s, s - P);
}

// Canonical form of an arbitrary u32 (M31::from_bytes, include/field/M31.hpp:111-116).
GKR_HD uint32_t from_u32(uint32_t x) {
    uint32_t s = (x & P) + (x >> 31);
    return umin(s, s - P);
}

// acc + a * b (mod p) for any acc < 2^32 and canonical a, b, left unreduced below 2^32:
// a * b <= (p - 1)^2 = 2^62 - 2^33 + 4, so t = acc + a * b < 2^62, t >> 31 < 2^31 and
// (t & p) + (t >> 31) <= 2^32 - 2.  Chains of these stay below 2^32; from_u32 finishes.
GKR_HD uint32_t mac_lazy(uint32_t acc, uint32_t a, uint32_t b) {
    const uint64_t t = (uint64_t)a * b + acc;
    return (uint32_t)(t & P) + (uint32_t)(t >> 31);
}

// a + (b - a) * r: the fold of a multilinear table at challenge r
// (SumcheckMultiLinearProdHelper::receive_challenge, sumcheck_helper.hpp:115,124-125).
GKR_HD uint32_t fold(uint32_t a, uint32_t b, uint32_t r) { return add(a, mul(sub(b, a), r)); }

// The fold at challenge r as a weighted sum: lerp(a, b, lerp_at(r)) = a (1 - r) + b r, the same
// field element as fold(a, b, r).  The weights are kept doubled, 2 (p + 1 - r) and 2 r (2 and 0
// for r = 0), so that t = a c0 + b c1 <= (p - 1) 2^32 holds twice the sum S: t >> 32 is S >> 31,
// at most p - 1, and (uint32_t)t >> 1 is S mod 2^31, at most p.  Two wide multiply-adds, one
// shift-and-add and one conditional subtraction, where fold takes three field operations.
struct Lerp {
    uint32_t c0, c1;
};
GKR_HD Lerp lerp_at(uint32_t r) {
    Lerp c;
    c.c1 = r + r;
    c.c0 = r ? 0u - c.c1 : 2u;
    return c;
}
GKR_HD uint32_t lerp(uint32_t a, uint32_t b, const Lerp& c) {
    const uint64_t t = (uint64_t)a * c.c0 + (uint64_t)b * c.c1;
    const uint32_t s = (uint32_t)(t >> 32) + ((uint32_t)t >> 1);
    return umin(s, s - P);
}

// Two folds in one, at challenges r0 and then r1, as a weighted sum of four rows with weights
// (1 - r0)(1 - r1), r0 (1 - r1), (1 - r0) r1, r0 r1 (canonical).  t = sum x_e c_e <= 4 (p - 1)^2 <
// 2^64; its bits 0..30, 31..61 and 62..63 weigh 1, 2^31 == 1 and 2^62 == 1 (mod p).  The upper two
// parts are at most p and 3, so one conditional subtraction brings their sum below p, and a
// second one the total of it and the lowest part, at most 2p - 1.  (The total of all three
// reaches 2p + 2.)  Four wide multiply-adds where three lerps take six.
struct Lerp2 {
    uint32_t c[4];
};
GKR_HD Lerp2 lerp2_at(uint32_t r0, uint32_t r1) {
    const uint32_t s0 = sub(1u, r0), s1 = sub(1u, r1);
    Lerp2 w;
    w.c[0] = mul(s0, s1);
    w.c[1] = mul(r0, s1);
    w.c[2] = mul(s0, r1);
    w.c[3] = mul(r0, r1);
    return w;
}
GKR_HD uint32_t lerp2(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, const Lerp2& w) {
    const uint64_t t = (uint64_t)x0 * w.c[0] + (uint64_t)x1 * w.c[1] + (uint64_t)x2 * w.c[2] + (uint64_t)x3 * w.c[3];
    const uint32_t u = ((uint32_t)(t >> 31) & P) + (uint32_t)(t >> 62);
    const uint32_t s = ((uint32_t)t & P) + umin(u, u - P);
    return umin(s, s - P);
}

// Evaluation at 2 of the degree-2 round polynomial from p0 = h(0), p1 = h(1) and
// p2raw = sum (f0+f1)(g0+g1) = 4 h(1/2): 6 p1 + 3 p0 - 2 p2raw (sumcheck_helper.hpp:100).
GKR_HD uint32_t eval_at_two(uint32_t p0, uint32_t p1, uint32_t p2raw) {
    return sub(add(mul(p1, 6), mul(p0, 3)), mul(p2raw, 2));
}

// The degree-2 polynomial through (0, v0), (1, v1), (2, v2) evaluated at x: the claim the
// next sumcheck round must meet (degree_2_eval, sumcheck_verifier_utils.hpp:10-18).  2^30 is
// the inverse of 2 (2 * 2^30 = p + 1).
GKR_HD uint32_t eval_degree2(uint32_t v0, uint32_t v1, uint32_t v2, uint32_t x) {
    const uint32_t c2 = mul(1u << 30, add(sub(v2, add(v1, v1)), v0));
    const uint32_t c1 = sub(sub(v1, v0), c2);
    return add(v0, mul(add(mul(c2, x), c1), x));
}

}  // namespace m31
