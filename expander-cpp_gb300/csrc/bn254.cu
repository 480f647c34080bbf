// BN254 scalar-field kernels (see bn254.cuh).  Same algorithms as the M31 kernels in
// kernels.cu, for one repetition (R = 1 for BN254, include/configuration/config.hpp:61-65),
// with 256-bit elements: one thread per element of a row, Montgomery multiplication on
// 8 x 32-bit limbs (CIOS as PTX multiply-add carry chains).
#include "bn254.cuh"

#include <algorithm>
#include <atomic>

namespace gkrgpu {
namespace bn {

namespace {

// r = 0x30644e72e131a029b85045b68181585d2833e84879b9709143e1f593f0000001 (little-endian
// limbs 0xf0000001, 0x43e1f593, ... appear as immediates in the PTX below), -r^-1 mod 2^32 =
// 0xefffffff.
__constant__ uint32_t kOne[8] = {0x4ffffffbu, 0xac96341cu, 0x9f60cd29u, 0x36fc7695u,
                                 0x7879462eu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};  // 2^256 mod r
__constant__ uint32_t kR2[8] = {0xae216da7u, 0x1bb8e645u, 0xe35c59e3u, 0x53fe3ab1u,
                                0x53bb8085u, 0x8c49833du, 0x7f4e44a5u, 0x0216d0b1u};  // 2^512 mod r
__constant__ uint32_t kInv2M[8] = {0x1ffffffeu, 0x783c14d8u, 0x0c8d1eddu, 0xaf982f6fu,
                                   0xfcfd4f45u, 0x8f5f7492u, 0x3d9cbfacu, 0x1f37631au};  // (r + 1) / 2 * 2^256 mod r

__device__ __forceinline__ Fr zero() {
    Fr z;
#pragma unroll
    for (int i = 0; i < 8; i++) z.l[i] = 0u;
    return z;
}
__device__ __forceinline__ Fr one() {
    Fr z;
#pragma unroll
    for (int i = 0; i < 8; i++) z.l[i] = kOne[i];
    return z;
}
// Field operations on canonical Montgomery forms (< r) as PTX carry chains (add.cc/addc,
// mad.lo.cc/madc.hi.cc); each asm block holds a whole chain, so no carry flag crosses
// statements.  The modulus limbs are immediates.

// x - r with a borrow chain; returns the borrow-out word (0xffffffff when x < r).
__device__ __forceinline__ uint32_t minus_r(const uint32_t* x, uint32_t* d) {
    uint32_t bw;
    asm("sub.cc.u32 %0, %9, 0xf0000001;\n\t"
        "subc.cc.u32 %1, %10, 0x43e1f593;\n\t"
        "subc.cc.u32 %2, %11, 0x79b97091;\n\t"
        "subc.cc.u32 %3, %12, 0x2833e848;\n\t"
        "subc.cc.u32 %4, %13, 0x8181585d;\n\t"
        "subc.cc.u32 %5, %14, 0xb85045b6;\n\t"
        "subc.cc.u32 %6, %15, 0xe131a029;\n\t"
        "subc.cc.u32 %7, %16, 0x30644e72;\n\t"
        "subc.u32 %8, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(bw)
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]));
    return bw;
}

__device__ __forceinline__ Fr add(const Fr& a, const Fr& b) {
    uint32_t s[8], d[8];
    // a + b < 2r < 2^255: no carry out of the top limb
    asm("add.cc.u32 %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32 %7, %15, %23;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
        : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(a.l[3]), "r"(a.l[4]), "r"(a.l[5]), "r"(a.l[6]), "r"(a.l[7]),
          "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]), "r"(b.l[3]), "r"(b.l[4]), "r"(b.l[5]), "r"(b.l[6]), "r"(b.l[7]));
    const bool below = minus_r(s, d) != 0u;
    Fr o;
#pragma unroll
    for (int i = 0; i < 8; i++) o.l[i] = below ? s[i] : d[i];
    return o;
}
__device__ __forceinline__ Fr sub(const Fr& a, const Fr& b) {
    uint32_t d[8], bw;
    asm("sub.cc.u32 %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32 %8, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(bw)
        : "r"(a.l[0]), "r"(a.l[1]), "r"(a.l[2]), "r"(a.l[3]), "r"(a.l[4]), "r"(a.l[5]), "r"(a.l[6]), "r"(a.l[7]),
          "r"(b.l[0]), "r"(b.l[1]), "r"(b.l[2]), "r"(b.l[3]), "r"(b.l[4]), "r"(b.l[5]), "r"(b.l[6]), "r"(b.l[7]));
    // a < b: add r back (bw is all ones, masking r's limbs)
    Fr o;
    asm("{\n\t.reg .u32 m0, m1, m2, m3, m4, m5, m6, m7;\n\t"
        "and.b32 m0, %16, 0xf0000001;\n\t"
        "and.b32 m1, %16, 0x43e1f593;\n\t"
        "and.b32 m2, %16, 0x79b97091;\n\t"
        "and.b32 m3, %16, 0x2833e848;\n\t"
        "and.b32 m4, %16, 0x8181585d;\n\t"
        "and.b32 m5, %16, 0xb85045b6;\n\t"
        "and.b32 m6, %16, 0xe131a029;\n\t"
        "and.b32 m7, %16, 0x30644e72;\n\t"
        "add.cc.u32 %0, %8, m0;\n\t"
        "addc.cc.u32 %1, %9, m1;\n\t"
        "addc.cc.u32 %2, %10, m2;\n\t"
        "addc.cc.u32 %3, %11, m3;\n\t"
        "addc.cc.u32 %4, %12, m4;\n\t"
        "addc.cc.u32 %5, %13, m5;\n\t"
        "addc.cc.u32 %6, %14, m6;\n\t"
        "addc.u32 %7, %15, m7;\n\t"
        "}"
        : "=r"(o.l[0]), "=r"(o.l[1]), "=r"(o.l[2]), "=r"(o.l[3]), "=r"(o.l[4]), "=r"(o.l[5]), "=r"(o.l[6]),
          "=r"(o.l[7])
        : "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]), "r"(bw));
    return o;
}

// Montgomery product a * b * 2^-256 mod r (inputs < r, output < r): CIOS (Koc, Acar, Kaliski
// 1996) with the running sum T = x + 2^32 y in two accumulators of eight words, x collecting
// the products of a's and r's even words and y those of the odd ones.  Every product's low and
// high word then land on neighbouring words of one accumulator, a 32 x 32 + 64 -> 64-bit
// multiply-add with carry, where a chain over all low words and another over all high words
// needs two multiplications a product, the high one at half the rate (30.9 per clock and SM
// against 61.6; the 64-bit form runs at about the low word's rate).  T < 2^288 as r < 2^254, so
// x carries out of its top word into y's and y never does.
// A step: T += a * bi, then T += m * r with m = T * (-r^-1) mod 2^32, which clears x0, then
// T /= 2^32: y becomes the accumulator at position 0 (its word 0 takes x1, whose carry enters
// the odd chain of the next step) and x from word 2 on the one at position 1.
__device__ __forceinline__ Fr mul(const Fr& a, const Fr& b) {
    uint32_t x[8], y[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t bi = b.l[i];
        if (i == 0) {
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const uint64_t e = (uint64_t)a.l[k] * bi, o = (uint64_t)a.l[k + 1] * bi;
                x[k] = (uint32_t)e;
                x[k + 1] = (uint32_t)(e >> 32);
                y[k] = (uint32_t)o;
                y[k + 1] = (uint32_t)(o >> 32);
            }
        } else {
            uint32_t z6, z7;
            // y0 += x1, then the odd products onto x2.. (the next y)
            asm("add.cc.u32 %0, %0, %9;\n\t"
                "madc.lo.cc.u32 %1, %10, %14, %1;\n\t"
                "madc.hi.cc.u32 %2, %10, %14, %2;\n\t"
                "madc.lo.cc.u32 %3, %11, %14, %3;\n\t"
                "madc.hi.cc.u32 %4, %11, %14, %4;\n\t"
                "madc.lo.cc.u32 %5, %12, %14, %5;\n\t"
                "madc.hi.cc.u32 %6, %12, %14, %6;\n\t"
                "madc.lo.cc.u32 %7, %13, %14, 0;\n\t"
                "madc.hi.u32 %8, %13, %14, 0;"
                : "+r"(y[0]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "=&r"(z6), "=&r"(z7)
                : "r"(x[1]), "r"(a.l[1]), "r"(a.l[3]), "r"(a.l[5]), "r"(a.l[7]), "r"(bi));
            const uint32_t z[8] = {x[2], x[3], x[4], x[5], x[6], x[7], z6, z7};
#pragma unroll
            for (int k = 0; k < 8; k++) {
                x[k] = y[k];
                y[k] = z[k];
            }
            // the even products onto x
            asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
                "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
                "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
                "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
                "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
                "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
                "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
                "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
                "addc.u32 %8, %8, 0;"
                : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "+r"(y[7])
                : "r"(a.l[0]), "r"(a.l[2]), "r"(a.l[4]), "r"(a.l[6]), "r"(bi));
        }
        const uint32_t m = x[0] * 0xefffffffu;
        asm("mad.lo.cc.u32 %0, %8, 0x43e1f593, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, 0x43e1f593, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, 0x2833e848, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, 0x2833e848, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, 0xb85045b6, %4;\n\t"
            "madc.hi.cc.u32 %5, %8, 0xb85045b6, %5;\n\t"
            "madc.lo.cc.u32 %6, %8, 0x30644e72, %6;\n\t"
            "madc.hi.u32 %7, %8, 0x30644e72, %7;"
            : "+r"(y[0]), "+r"(y[1]), "+r"(y[2]), "+r"(y[3]), "+r"(y[4]), "+r"(y[5]), "+r"(y[6]), "+r"(y[7])
            : "r"(m));
        asm("mad.lo.cc.u32 %0, %9, 0xf0000001, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, 0xf0000001, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, 0x79b97091, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, 0x79b97091, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, 0x8181585d, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, 0x8181585d, %5;\n\t"
            "madc.lo.cc.u32 %6, %9, 0xe131a029, %6;\n\t"
            "madc.hi.cc.u32 %7, %9, 0xe131a029, %7;\n\t"
            "addc.u32 %8, %8, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "+r"(y[7])
            : "r"(m));
    }
    // T / 2^32 < 2r < 2^255: one conditional subtraction of r
    uint32_t t[8], d[8];
    asm("add.cc.u32 %0, %8, %15;\n\t"
        "addc.cc.u32 %1, %9, %16;\n\t"
        "addc.cc.u32 %2, %10, %17;\n\t"
        "addc.cc.u32 %3, %11, %18;\n\t"
        "addc.cc.u32 %4, %12, %19;\n\t"
        "addc.cc.u32 %5, %13, %20;\n\t"
        "addc.cc.u32 %6, %14, %21;\n\t"
        "addc.u32 %7, %22, 0;"
        : "=&r"(t[0]), "=&r"(t[1]), "=&r"(t[2]), "=&r"(t[3]), "=&r"(t[4]), "=&r"(t[5]), "=&r"(t[6]), "=&r"(t[7])
        : "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(y[0]), "r"(y[1]), "r"(y[2]),
          "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
    const bool below = minus_r(t, d) != 0u;
    Fr o;
#pragma unroll
    for (int i = 0; i < 8; i++) o.l[i] = below ? t[i] : d[i];
    return o;
}
__device__ __forceinline__ Fr from_mont(const Fr& a) {
    Fr u = zero();
    u.l[0] = 1u;
    return mul(a, u);
}
__device__ __forceinline__ Fr to_mont(const Fr& a) {
    Fr r2;
#pragma unroll
    for (int i = 0; i < 8; i++) r2.l[i] = kR2[i];
    return mul(a, r2);
}
__device__ __forceinline__ Fr fold(const Fr& a, const Fr& b, const Fr& r) { return add(a, mul(sub(b, a), r)); }

// Sums of products before their Montgomery reduction, below 16 r^2 < 2^512 - 2^510: a product
// alone is 64 of mul's 136 multiplications, and a sum is reduced once for kWideTerms of them.
// The round kernels are bound by the multiply pipe: on 2^16 rows of 64 copies phase two's round 0
// (three sums a pair) went from 122 to 84 us, the first fold rounds (two sums and four or
// two folds) from 127 to 114 and 111 to 100.
struct Wide {
    uint32_t w[16];
};
// Products that may be added to zero or to a lifted sum (lift(x) < 2^256 r < 5.3 r^2).
constexpr uint32_t kWideTerms = 10;

__device__ __forceinline__ Wide lift(const Fr& x) {
    Wide s;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        s.w[i] = 0u;
        s.w[8 + i] = x.l[i];
    }
    return s;
}

// s += a b.  As in mul, the product is formed in two accumulators whose 64-bit pairs start at
// the even words (e) and at the odd ones (o).  Row i adds four products to four neighbouring
// pairs of each: to e from word i + (i & 1) on, to o from word i + 1 - (i & 1) on.  The rows that
// end on a pair not used before leave no carry; the others' carry starts the next pair.
__device__ __forceinline__ void mac(Wide& s, const Fr& a, const Fr& b) {
    uint32_t e[16], o[18];  // a word at its own index (o[0] unused, o[16] and o[17] zero)
#pragma unroll
    for (int k = 0; k < 16; k++) e[k] = 0u;
#pragma unroll
    for (int k = 0; k < 18; k++) o[k] = 0u;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t bi = b.l[i];
        const int odd = i & 1;
        // products of the words of a with i's parity meet e, the others o
        const int pe = i + odd, po = i + 1 - odd;
        if (i == 0) {
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const uint64_t x = (uint64_t)a.l[k] * bi, y = (uint64_t)a.l[k + 1] * bi;
                e[k] = (uint32_t)x;
                e[k + 1] = (uint32_t)(x >> 32);
                o[k + 1] = (uint32_t)y;
                o[k + 2] = (uint32_t)(y >> 32);
            }
            continue;
        }
        const uint32_t e0 = a.l[odd], e1 = a.l[2 + odd], e2 = a.l[4 + odd], e3 = a.l[6 + odd];
        const uint32_t o0 = a.l[1 - odd], o1 = a.l[3 - odd], o2 = a.l[5 - odd], o3 = a.l[7 - odd];
        if (odd) {
            asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
                "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
                "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
                "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
                "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
                "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
                "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
                "madc.hi.u32 %7, %11, %12, %7;"
                : "+r"(e[pe]), "+r"(e[pe + 1]), "+r"(e[pe + 2]), "+r"(e[pe + 3]), "+r"(e[pe + 4]), "+r"(e[pe + 5]),
                  "+r"(e[pe + 6]), "+r"(e[pe + 7])
                : "r"(e0), "r"(e1), "r"(e2), "r"(e3), "r"(bi));
            asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
                "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
                "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
                "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
                "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
                "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
                "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
                "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
                "addc.u32 %8, 0, 0;"
                : "+r"(o[po]), "+r"(o[po + 1]), "+r"(o[po + 2]), "+r"(o[po + 3]), "+r"(o[po + 4]), "+r"(o[po + 5]),
                  "+r"(o[po + 6]), "+r"(o[po + 7]), "=r"(o[po + 8])
                : "r"(o0), "r"(o1), "r"(o2), "r"(o3), "r"(bi));
        } else {
            asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
                "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
                "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
                "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
                "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
                "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
                "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
                "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
                "addc.u32 %8, 0, 0;"
                : "+r"(e[pe]), "+r"(e[pe + 1]), "+r"(e[pe + 2]), "+r"(e[pe + 3]), "+r"(e[pe + 4]), "+r"(e[pe + 5]),
                  "+r"(e[pe + 6]), "+r"(e[pe + 7]), "=r"(e[pe + 8])
                : "r"(e0), "r"(e1), "r"(e2), "r"(e3), "r"(bi));
            asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
                "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
                "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
                "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
                "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
                "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
                "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
                "madc.hi.u32 %7, %11, %12, %7;"
                : "+r"(o[po]), "+r"(o[po + 1]), "+r"(o[po + 2]), "+r"(o[po + 3]), "+r"(o[po + 4]), "+r"(o[po + 5]),
                  "+r"(o[po + 6]), "+r"(o[po + 7])
                : "r"(o0), "r"(o1), "r"(o2), "r"(o3), "r"(bi));
        }
    }
    auto add8 = [](uint32_t* d, const uint32_t* x, uint32_t carry) {  // d[0..7] += x[0..7] + carry
        uint32_t out;
        asm("add.cc.u32 %8, %17, 0xffffffff;\n\t"
            "addc.cc.u32 %0, %0, %9;\n\t"
            "addc.cc.u32 %1, %1, %10;\n\t"
            "addc.cc.u32 %2, %2, %11;\n\t"
            "addc.cc.u32 %3, %3, %12;\n\t"
            "addc.cc.u32 %4, %4, %13;\n\t"
            "addc.cc.u32 %5, %5, %14;\n\t"
            "addc.cc.u32 %6, %6, %15;\n\t"
            "addc.cc.u32 %7, %7, %16;\n\t"
            "addc.u32 %8, 0, 0;"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7]), "=&r"(out)
            : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(carry));
        return out;
    };
    add8(s.w + 8, e + 8, add8(s.w, e, 0u));
    add8(s.w + 8, o + 8, add8(s.w, o, 0u));
}

// s 2^-256 mod r: the low half's Montgomery reduction (mul's steps without its products), at
// most r, plus the high half, below 2.9 r (s < 15.3 r^2, and r < 0.19 2^256): below 4 r together.
__device__ __forceinline__ Fr reduce(const Wide& s) {
    uint32_t x[8], y[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        x[k] = s.w[k];
        y[k] = 0u;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        if (i > 0) {
            uint32_t z6;
            asm("add.cc.u32 %0, %0, %8;\n\t"
                "addc.cc.u32 %1, %1, 0;\n\t"
                "addc.cc.u32 %2, %2, 0;\n\t"
                "addc.cc.u32 %3, %3, 0;\n\t"
                "addc.cc.u32 %4, %4, 0;\n\t"
                "addc.cc.u32 %5, %5, 0;\n\t"
                "addc.cc.u32 %6, %6, 0;\n\t"
                "addc.u32 %7, 0, 0;"
                : "+r"(y[0]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "=r"(z6)
                : "r"(x[1]));
            const uint32_t z[8] = {x[2], x[3], x[4], x[5], x[6], x[7], z6, 0u};
#pragma unroll
            for (int k = 0; k < 8; k++) {
                x[k] = y[k];
                y[k] = z[k];
            }
        }
        const uint32_t m = x[0] * 0xefffffffu;
        asm("mad.lo.cc.u32 %0, %8, 0x43e1f593, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, 0x43e1f593, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, 0x2833e848, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, 0x2833e848, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, 0xb85045b6, %4;\n\t"
            "madc.hi.cc.u32 %5, %8, 0xb85045b6, %5;\n\t"
            "madc.lo.cc.u32 %6, %8, 0x30644e72, %6;\n\t"
            "madc.hi.u32 %7, %8, 0x30644e72, %7;"
            : "+r"(y[0]), "+r"(y[1]), "+r"(y[2]), "+r"(y[3]), "+r"(y[4]), "+r"(y[5]), "+r"(y[6]), "+r"(y[7])
            : "r"(m));
        asm("mad.lo.cc.u32 %0, %9, 0xf0000001, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, 0xf0000001, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, 0x79b97091, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, 0x79b97091, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, 0x8181585d, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, 0x8181585d, %5;\n\t"
            "madc.lo.cc.u32 %6, %9, 0xe131a029, %6;\n\t"
            "madc.hi.cc.u32 %7, %9, 0xe131a029, %7;\n\t"
            "addc.u32 %8, %8, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "+r"(y[7])
            : "r"(m));
    }
    // x[1..7] + y + the high half
    uint32_t t[8], d[8];
    asm("add.cc.u32 %0, %8, %15;\n\t"
        "addc.cc.u32 %1, %9, %16;\n\t"
        "addc.cc.u32 %2, %10, %17;\n\t"
        "addc.cc.u32 %3, %11, %18;\n\t"
        "addc.cc.u32 %4, %12, %19;\n\t"
        "addc.cc.u32 %5, %13, %20;\n\t"
        "addc.cc.u32 %6, %14, %21;\n\t"
        "addc.u32 %7, %22, 0;"
        : "=&r"(t[0]), "=&r"(t[1]), "=&r"(t[2]), "=&r"(t[3]), "=&r"(t[4]), "=&r"(t[5]), "=&r"(t[6]), "=&r"(t[7])
        : "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(y[0]), "r"(y[1]), "r"(y[2]),
          "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
    asm("add.cc.u32 %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, %9;\n\t"
        "addc.cc.u32 %2, %2, %10;\n\t"
        "addc.cc.u32 %3, %3, %11;\n\t"
        "addc.cc.u32 %4, %4, %12;\n\t"
        "addc.cc.u32 %5, %5, %13;\n\t"
        "addc.cc.u32 %6, %6, %14;\n\t"
        "addc.u32 %7, %7, %15;"
        : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7])
        : "r"(s.w[8]), "r"(s.w[9]), "r"(s.w[10]), "r"(s.w[11]), "r"(s.w[12]), "r"(s.w[13]), "r"(s.w[14]), "r"(s.w[15]));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const bool below = minus_r(t, d) != 0u;
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = below ? t[i] : d[i];
    }
    Fr o;
#pragma unroll
    for (int i = 0; i < 8; i++) o.l[i] = t[i];
    return o;
}

// The canonical value of a sum of Montgomery forms given as 64-bit limb sums:
// T = sum_k s[k] 2^(32k) is the sum of the x_i R (R = 2^256), so REDC(T) = T R^-1 mod r is
// sum x_i, already canonical after one conditional subtraction (T < 2^266 keeps
// REDC(T) < 2r).  Eight reduction steps of CIOS on a ten-word window.
__device__ __forceinline__ Fr redc_sums(const unsigned long long* s) {
    uint32_t t0, t1, t2, t3, t4, t5, t6, t7, t8, t9;
    {
        uint32_t w[10];
        unsigned long long c = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const unsigned long long lo = c + (s[k] & 0xffffffffull);
            w[k] = (uint32_t)lo;
            c = (lo >> 32) + (s[k] >> 32);
        }
        w[8] = (uint32_t)c;
        w[9] = (uint32_t)(c >> 32);
        t0 = w[0]; t1 = w[1]; t2 = w[2]; t3 = w[3]; t4 = w[4];
        t5 = w[5]; t6 = w[6]; t7 = w[7]; t8 = w[8]; t9 = w[9];
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        asm("{\n\t.reg .u32 m;\n\t"
            "mul.lo.u32 m, %0, 0xefffffff;\n\t"
            "mad.lo.cc.u32 %0, m, 0xf0000001, %0;\n\t"
            "madc.lo.cc.u32 %1, m, 0x43e1f593, %1;\n\t"
            "madc.lo.cc.u32 %2, m, 0x79b97091, %2;\n\t"
            "madc.lo.cc.u32 %3, m, 0x2833e848, %3;\n\t"
            "madc.lo.cc.u32 %4, m, 0x8181585d, %4;\n\t"
            "madc.lo.cc.u32 %5, m, 0xb85045b6, %5;\n\t"
            "madc.lo.cc.u32 %6, m, 0xe131a029, %6;\n\t"
            "madc.lo.cc.u32 %7, m, 0x30644e72, %7;\n\t"
            "addc.cc.u32 %8, %8, 0;\n\t"
            "addc.u32 %9, %9, 0;\n\t"
            "mad.hi.cc.u32 %1, m, 0xf0000001, %1;\n\t"
            "madc.hi.cc.u32 %2, m, 0x43e1f593, %2;\n\t"
            "madc.hi.cc.u32 %3, m, 0x79b97091, %3;\n\t"
            "madc.hi.cc.u32 %4, m, 0x2833e848, %4;\n\t"
            "madc.hi.cc.u32 %5, m, 0x8181585d, %5;\n\t"
            "madc.hi.cc.u32 %6, m, 0xb85045b6, %6;\n\t"
            "madc.hi.cc.u32 %7, m, 0xe131a029, %7;\n\t"
            "madc.hi.cc.u32 %8, m, 0x30644e72, %8;\n\t"
            "addc.u32 %9, %9, 0;\n\t"
            "}"
            : "+r"(t0), "+r"(t1), "+r"(t2), "+r"(t3), "+r"(t4), "+r"(t5), "+r"(t6), "+r"(t7), "+r"(t8), "+r"(t9));
        t0 = t1; t1 = t2; t2 = t3; t3 = t4; t4 = t5; t5 = t6; t6 = t7; t7 = t8; t8 = t9; t9 = 0;
    }
    const uint32_t t[8] = {t0, t1, t2, t3, t4, t5, t6, t7};
    uint32_t d[8];
    const bool below = minus_r(t, d) != 0u;
    Fr o;
#pragma unroll
    for (int i = 0; i < 8; i++) o.l[i] = below ? t[i] : d[i];
    return o;
}

__device__ __forceinline__ Fr ldf(const uint32_t* __restrict__ base, uint64_t row, uint32_t N, uint32_t lane) {
    const uint4* p = reinterpret_cast<const uint4*>(base + (row * N + lane) * 8);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    Fr f;
    f.l[0] = a.x; f.l[1] = a.y; f.l[2] = a.z; f.l[3] = a.w;
    f.l[4] = b.x; f.l[5] = b.y; f.l[6] = b.z; f.l[7] = b.w;
    return f;
}
__device__ __forceinline__ void stf(uint32_t* base, uint64_t row, uint32_t N, uint32_t lane, const Fr& f) {
    uint4* p = reinterpret_cast<uint4*>(base + (row * N + lane) * 8);
    p[0] = make_uint4(f.l[0], f.l[1], f.l[2], f.l[3]);
    p[1] = make_uint4(f.l[4], f.l[5], f.l[6], f.l[7]);
}
__device__ __forceinline__ Fr lds(const Fr* __restrict__ t, uint64_t i) {
    const uint4* p = reinterpret_cast<const uint4*>(t + i);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    Fr f;
    f.l[0] = a.x; f.l[1] = a.y; f.l[2] = a.z; f.l[3] = a.w;
    f.l[4] = b.x; f.l[5] = b.y; f.l[6] = b.z; f.l[7] = b.w;
    return f;
}
__device__ __forceinline__ void sts(Fr* t, uint64_t i, const Fr& f) {
    uint4* p = reinterpret_cast<uint4*>(t + i);
    p[0] = make_uint4(f.l[0], f.l[1], f.l[2], f.l[3]);
    p[1] = make_uint4(f.l[4], f.l[5], f.l[6], f.l[7]);
}

struct Tile {
    uint32_t q, rs;
    bool active;
};
__device__ __forceinline__ Tile tile(const GeoBn& g) {
    Tile t;
    t.q = blockIdx.y * g.tpr + threadIdx.x % g.tpr;  // lane
    t.rs = threadIdx.x / g.tpr;
    t.active = t.rs < g.rps;
    return t;
}

// Canonical total of component c of one lane; leaves its accumulators zeroed.
__device__ __noinline__ Fr take(const RedBn& red, uint32_t c, uint32_t N, uint32_t lane) {
    unsigned long long s[8];
    unsigned long long* p = &red.acc[((size_t)c * N + lane) * 8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        s[k] = __ldcg(p + k);
        p[k] = 0ull;
    }
    return redc_sums(s);
}

// C components per thread -> shared-memory sum over the CTA's row slices -> 64-bit
// atomic adds per limb -> the last CTA of the lane group finishes its lanes: one thread per
// (component, lane) total, then fin(c, lane, totals of the lane, tpr) per output value.
template <int C, class Fin>
__device__ __forceinline__ void reduce_bn(Fr (&acc)[C], const GeoBn& g, bool active, RedBn red, Fin fin) {
    extern __shared__ uint32_t smem[];
    const uint32_t tid = threadIdx.x, B = blockDim.x;
    uint32_t rows = g.rps;
    if (g.tpr < 32 && (g.tpr & (g.tpr - 1)) == 0) {
        // power-of-two tile below a warp (every thread active): first fold the warp's row
        // slices together with shuffles, leaving one row per warp
        for (uint32_t off = g.tpr; off < 32; off <<= 1)
#pragma unroll
            for (int c = 0; c < C; c++) {
                Fr o;
#pragma unroll
                for (int k = 0; k < 8; k++) o.l[k] = __shfl_xor_sync(0xffffffffu, acc[c].l[k], off);
                acc[c] = add(acc[c], o);
            }
        rows = B / 32;
        if ((tid & 31) < g.tpr)
#pragma unroll
            for (int c = 0; c < C; c++)
#pragma unroll
                for (int k = 0; k < 8; k++) smem[(c * 8 + k) * B + (tid >> 5) * g.tpr + (tid & 31)] = acc[c].l[k];
    } else {
#pragma unroll
        for (int c = 0; c < C; c++)
#pragma unroll
            for (int k = 0; k < 8; k++) smem[(c * 8 + k) * B + tid] = active ? acc[c].l[k] : 0u;
    }
    __syncthreads();
    for (uint32_t o = tid; o < (uint32_t)C * g.tpr; o += B) {
        const uint32_t c = o / g.tpr, q = o - c * g.tpr;
        Fr s = zero();
        for (uint32_t r = 0; r < rows; r++) {
            Fr x;
#pragma unroll
            for (int k = 0; k < 8; k++) x.l[k] = smem[(c * 8 + k) * B + r * g.tpr + q];
            s = add(s, x);
        }
        const uint32_t lane = blockIdx.y * g.tpr + q;
#pragma unroll
        for (int k = 0; k < 8; k++) atomicAdd(&red.acc[((size_t)c * g.N + lane) * 8 + k], (unsigned long long)s.l[k]);
    }
    __threadfence();
    __syncthreads();
    __shared__ unsigned int is_last;
    if (tid == 0) is_last = (atomicAdd(&red.ticket[blockIdx.y], 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // the last CTA: every (component, lane) total is reduced by its own thread, then each
    // output value is finished by its own thread (the finisher's chains run in parallel)
    Fr* tot = reinterpret_cast<Fr*>(smem);
    for (uint32_t o = tid; o < (uint32_t)C * g.tpr; o += B) {
        const uint32_t c = o / g.tpr, li = o - c * g.tpr;
        tot[o] = take(red, c, g.N, blockIdx.y * g.tpr + li);
    }
    __syncthreads();
    for (uint32_t o = tid; o < (uint32_t)C * g.tpr; o += B) {
        const uint32_t c = o / g.tpr, li = o - c * g.tpr;
        fin(c, blockIdx.y * g.tpr + li, tot + li, g.tpr);
    }
    if (tid == 0) red.ticket[blockIdx.y] = 0u;
    if (red.done) {
        __threadfence_system();
        __syncthreads();
        if (tid == 0) atomicAdd_system(red.done, 1u);
    }
}

// Output c of one lane from the canonical totals t[0], t[tpr], t[2 tpr] (components 0..2 of
// that lane): the evaluations at 0, 1 and 2 (6 p1 + 3 p0 - 2 p2raw).  Phase two multiplies
// by vx: a Montgomery product of a canonical value with vx's Montgomery form is the
// canonical product.
struct RoundFinBn {
    uint32_t* out;  // 3 x N x 8 limbs, canonical
    const uint32_t* vx;
    uint32_t N;
    uint32_t* dev = nullptr;  // device copy of out, or null
    __device__ __noinline__ void operator()(uint32_t c, uint32_t lane, const Fr* t, uint32_t tpr) const {
        Fr v;
        if (c < 2) {
            v = t[c * tpr];
        } else {
            const Fr p0 = t[0], p1 = t[tpr], p2r = t[2 * tpr];
            const Fr p1x2 = add(p1, p1);
            v = add(add(p1x2, p1x2), p1x2);       // 6 p1
            v = add(v, add(add(p0, p0), p0));    // + 3 p0
            v = sub(v, add(p2r, p2r));            // - 2 p2raw
        }
        if (vx) v = mul(v, ldf(vx, 0, N, lane));
        stf(out, c, N, lane, v);
        if (dev) stf(dev, c, N, lane, v);
    }
};

// Element of a host-written table read past the caches (each limb fetched again).
__device__ __forceinline__ Fr ldf_cv(const uint32_t* base, uint32_t N, uint32_t lane) {
    Fr f;
#pragma unroll
    for (int k = 0; k < 8; k++) f.l[k] = __ldcv(base + (size_t)lane * 8 + k);
    return f;
}

// The round's evaluations from two components per lane, p0 (t[0]) and p2raw (t[tpr]): p1 is
// the round's claim less p0 (an honest prover's round polynomial meets p0 + p1 = claim, the
// verifier's check in sumcheck.hpp:152).  The claim is `claim` (N x 8 words, host-written),
// or the previous round's polynomial at its challenge r (Montgomery form), degree_2_eval
// (sumcheck_verifier_utils.hpp:10-18) of its evaluations in `prev`.  Component 0 writes the
// evaluations at 0 and 1, component 1 the one at 2; with vx (phase two) the sums are
// multiplied by v(rx) first.  Canonical values times Montgomery forms give canonical values.
struct ClaimFinBn {
    uint32_t* out;          // 3 x N x 8 limbs, canonical
    uint32_t* dev;          // device copy of out, or null
    const uint32_t* claim;  // N x 8, or null
    const uint32_t* prev;   // 3 x N x 8, or null
    const uint32_t* vx;
    Fr r;
    uint32_t N;
    __device__ __noinline__ void operator()(uint32_t c, uint32_t lane, const Fr* t, uint32_t tpr) const {
        Fr cl;
        if (claim) {
            cl = ldf_cv(claim, N, lane);
        } else {
            const Fr v0 = ldf(prev, 0, N, lane), v1 = ldf(prev, 1, N, lane), v2 = ldf(prev, 2, N, lane);
            Fr inv2;
#pragma unroll
            for (int k = 0; k < 8; k++) inv2.l[k] = kInv2M[k];
            const Fr c2 = mul(add(sub(v2, add(v1, v1)), v0), inv2);
            const Fr c1 = sub(sub(v1, v0), c2);
            cl = add(v0, mul(add(mul(c2, r), c1), r));
        }
        Fr x = zero();
        if (vx) x = ldf(vx, 0, N, lane);
        Fr p0 = t[0];
        if (vx) p0 = mul(p0, x);
        const Fr p1 = sub(cl, p0);
        if (c == 0) {
            stf(out, 0, N, lane, p0);
            stf(out, 1, N, lane, p1);
            if (dev) {
                stf(dev, 0, N, lane, p0);
                stf(dev, 1, N, lane, p1);
            }
            return;
        }
        Fr p2r = t[tpr];
        if (vx) p2r = mul(p2r, x);
        const Fr p1x2 = add(p1, p1);
        Fr v = add(add(p1x2, p1x2), p1x2);    // 6 p1
        v = add(v, add(add(p0, p0), p0));     // + 3 p0
        v = sub(v, add(p2r, p2r));            // - 2 p2raw
        stf(out, 2, N, lane, v);
        if (dev) stf(dev, 2, N, lane, v);
    }
};

struct CopyFinBn {
    uint32_t* out;  // N x 8 limbs, canonical
    uint32_t N;
    __device__ void operator()(uint32_t, uint32_t lane, const Fr* t, uint32_t) const { stf(out, 0, N, lane, t[0]); }
};

__device__ __forceinline__ void accum(Wide (&acc)[3], const Fr& f0, const Fr& f1, const Fr& h0, const Fr& h1) {
    mac(acc[0], f0, h0);
    mac(acc[1], f1, h1);
    mac(acc[2], add(f0, f1), add(h0, h1));
}
// p0 and p2raw only (the round's p1 comes from its claim: ClaimFinBn)
__device__ __forceinline__ void accum(Wide (&acc)[2], const Fr& f0, const Fr& f1, const Fr& h0, const Fr& h1) {
    mac(acc[0], f0, h0);
    mac(acc[1], add(f0, f1), add(h0, h1));
}
// Sums of up to kWideTerms accumulations each: the totals so far, which the next ones go on from.
template <int C>
__device__ __forceinline__ void settle(Wide (&acc)[C], Fr (&total)[C]) {
#pragma unroll
    for (int c = 0; c < C; c++) {
        total[c] = reduce(acc[c]);
        acc[c] = lift(total[c]);
    }
}

// ---------------------------------------------------------------- kernels
// Input -> Montgomery table.  Canonical input (bad != null): an element >= r raises *bad
// and is stored as 0.  Otherwise every element is first reduced mod r (from_bytes of
// arbitrary 32-byte words: 2^256 < 6r, so at most five subtractions).
__global__ void k_load(const uint32_t* __restrict__ canon, uint32_t* __restrict__ mont, uint64_t n, unsigned int* bad) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Fr x = lds(reinterpret_cast<const Fr*>(canon), i);
        uint32_t d[8];
        if (bad) {
            if (minus_r(x.l, d) == 0u) {  // no borrow: x >= r
                *reinterpret_cast<volatile unsigned int*>(bad) = 1u;  // every writer stores 1 (device or mapped flag)
                x = zero();
            }
        } else {
            for (int k = 0; k < 5 && minus_r(x.l, d) == 0u; k++)
#pragma unroll
                for (int q = 0; q < 8; q++) x.l[q] = d[q];
        }
        sts(reinterpret_cast<Fr*>(mont), i, to_mont(x));
    }
}

// Montgomery -> canonical, in place.
__global__ void k_unload(uint32_t* v, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    Fr* t = reinterpret_cast<Fr*>(v);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint4* p = reinterpret_cast<const uint4*>(t + i);
        const uint4 a = p[0], b = p[1];
        Fr x;
        x.l[0] = a.x; x.l[1] = a.y; x.l[2] = a.z; x.l[3] = a.w;
        x.l[4] = b.x; x.l[5] = b.y; x.l[6] = b.z; x.l[7] = b.w;
        sts(t, i, from_mont(x));
    }
}

__global__ void __launch_bounds__(256) k_evaluate(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint64_t O,
                                                  const uint32_t* __restrict__ mo_off, const uint4* __restrict__ mo_g,
                                                  const Fr* __restrict__ mo_c, const uint32_t* __restrict__ ao_off,
                                                  const uint2* __restrict__ ao_g, const Fr* __restrict__ ao_c, GeoBn g) {
    const Tile t = tile(g);
    if (!t.active) return;
    for (uint64_t o = (uint64_t)blockIdx.x * g.rps + t.rs; o < O; o += (uint64_t)gridDim.x * g.rps) {
        Fr acc = zero();
        const uint32_t m0 = __ldg(mo_off + o), m1 = __ldg(mo_off + o + 1);
        for (uint32_t k = m0; k < m1; k++) {
            const uint4 gt = __ldg(mo_g + k);
            acc = add(acc, mul(mul(ldf(in, gt.x, g.N, t.q), ldf(in, gt.y, g.N, t.q)), lds(mo_c, k)));
        }
        const uint32_t a0 = __ldg(ao_off + o), a1 = __ldg(ao_off + o + 1);
        for (uint32_t k = a0; k < a1; k++) {
            const uint2 gt = __ldg(ao_g + k);
            acc = add(acc, mul(ldf(in, gt.x, g.N, t.q), lds(ao_c, k)));
        }
        stf(out, o, g.N, t.q, acc);
    }
}

// ---------------------------------------------------------------- eq factors
// f1 eq(r1, z) + f2 eq(r2, z), eq(r, z) = prod over bits t of z of (bit ? r_t : 1 - r_t), from
// tables of 256 entries per eight bits that a CTA builds in shared memory: one product a point
// where the factor is used (up to 2^16), where a table over z was a launch of its own (15 us at
// 2^9 entries, 25 at 2^16) in front of every user.  They are built from tables of 16 entries
// per four bits, a chain of three products.  (Tables of 32 entries straight from the
// bits, as for M31, took 21 us of a 2^9 layer's weights and 63 of a 2^16 layer's.)
constexpr uint32_t kEqBits = 8, kEqEntries = 1u << kEqBits;

__host__ __device__ inline uint32_t eq_tables(const EqArgsBn& a) {
    return a.nvars > kEqBits ? (a.nvars + kEqBits - 1) / kEqBits : 1u;
}
__host__ __device__ inline uint32_t eq_points(const EqArgsBn& a) { return a.has_r2 ? 2u : 1u; }
// Elements of shared memory: the tables, then the building scratch (shared by several args).
__host__ __device__ inline uint32_t eq_elems(const EqArgsBn& a) { return eq_points(a) * eq_tables(a) * kEqEntries; }
__host__ __device__ inline uint32_t eq_scratch(const EqArgsBn& a) { return eq_points(a) * eq_tables(a) * 32; }

// Fills t (eq_elems entries) with the help of u (eq_scratch); the whole CTA calls it, and
// synchronises before it uses either again.
__device__ __forceinline__ void eq_build(Fr* t, Fr* u, const EqArgsBn& a) {
    const uint32_t nt = eq_tables(a), pts = eq_points(a);
    for (uint32_t i = threadIdx.x; i < pts * nt * 32; i += blockDim.x) {
        const uint32_t p = i / (nt * 32), d = (i - p * nt * 32) >> 4, x = i & 15;
        const uint32_t(*r)[8] = p ? a.r2 : a.r1;
        auto factor = [&](uint32_t b) {
            Fr f;
            const bool bit = (x >> b) & 1;
            const uint32_t v = 4 * d + b;
            if (v == 0) {  // with the point's factor
#pragma unroll
                for (int l = 0; l < 8; l++) f.l[l] = p ? a.first2[bit][l] : a.first1[bit][l];
                return f;
            }
#pragma unroll
            for (int l = 0; l < 8; l++) f.l[l] = r[v][l];
            return bit ? f : sub(one(), f);
        };
        const uint32_t left = a.nvars > 4 * d ? a.nvars - 4 * d : 0;
        if (left == 0) {
            if (d == 0) u[i] = factor(0);  // no variables at all: the point's factor
            continue;
        }
        Fr e = factor(0);
        if (left > 1) e = mul(e, factor(1));
        if (left > 2) {
            Fr g = factor(2);
            if (left > 3) g = mul(g, factor(3));
            e = mul(e, g);
        }
        u[i] = e;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < pts * nt * kEqEntries; i += blockDim.x) {
        const uint32_t pd = i >> kEqBits, x = i & (kEqEntries - 1);  // pd = p nt + d
        const uint32_t bits = a.nvars - (pd % nt) * kEqBits;
        if (x >> (bits < kEqBits ? bits : kEqBits)) continue;
        const Fr lo = u[pd * 32 + (x & 15)];
        t[i] = bits > 4 ? mul(lo, u[pd * 32 + 16 + (x >> 4)]) : lo;
    }
}
__device__ __forceinline__ Fr eq_at(const Fr* t, uint32_t nt, bool two, uint32_t z) {
    Fr e = t[z & (kEqEntries - 1)];
    Fr f = two ? t[nt * kEqEntries + (z & (kEqEntries - 1))] : zero();
#pragma unroll 1
    for (uint32_t d = 1; d < nt; d++) {
        const uint32_t x = d * kEqEntries + ((z >> (kEqBits * d)) & (kEqEntries - 1));
        e = mul(e, t[x]);
        if (two) f = mul(f, t[nt * kEqEntries + x]);
    }
    return two ? add(e, f) : e;
}
extern __shared__ uint4 eqsm_raw[];

// Lanes that share a row's gates (about one a row, but four in the longest row of a warp, each a
// chain of three products), and their sums' total in the first of them.
constexpr uint32_t kRowLanes = 4;
__device__ __forceinline__ Fr row_sum(Fr s, uint32_t gates) {
    const uint32_t m = 0xfu << (threadIdx.x & 28);  // the row's lanes
    if (gates < 2) return s;                        // (in the first lane already)
#pragma unroll
    for (uint32_t off = 2; off > 0; off >>= 1) {
        Fr o;
#pragma unroll
        for (int l = 0; l < 8; l++) o.l[l] = __shfl_xor_sync(m, s.l[l], off);
        s = add(s, o);
    }
    return s;
}

__global__ void __launch_bounds__(256) k_weights(uint64_t I, uint64_t Gm, const __grid_constant__ EqArgsBn eqc,
                                                 const uint4* __restrict__ mx_g, const Fr* __restrict__ mx_c,
                                                 const uint32_t* __restrict__ ax_off, const uint2* __restrict__ ax_g,
                                                 const Fr* __restrict__ ax_c, Fr* __restrict__ a_out, Fr* __restrict__ w_out) {
    Fr* const t = reinterpret_cast<Fr*>(eqsm_raw);
    eq_build(t, t + eq_elems(eqc), eqc);
    __syncthreads();
    const uint32_t nd = eq_tables(eqc);
    const bool two = eqc.has_r2;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n = kRowLanes * I > Gm ? kRowLanes * I : Gm;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (i < Gm) sts(w_out, i, mul(lds(mx_c, i), eq_at(t, nd, two, __ldg(&mx_g[i].y))));
        const uint64_t x = i / kRowLanes;
        if (x < I) {
            const uint32_t l = (uint32_t)i % kRowLanes, k0 = __ldg(ax_off + x), k1 = __ldg(ax_off + x + 1);
            Fr s = zero();
            for (uint32_t k = k0 + l; k < k1; k += kRowLanes)
                s = add(s, mul(lds(ax_c, k), eq_at(t, nd, two, __ldg(&ax_g[k].x))));
            s = row_sum(s, k1 - k0);
            if (l == 0) sts(a_out, x, s);
        }
    }
}

// Verifier gate sums (eval_sparse_circuit_connect_poly, one repetition): over the mul gates
// sum c eqz[o] eqx[i0] eqy[i1], or over the add gates sum c eqz[o] eqx[i0], walked by output
// (the evaluate CSR with Montgomery coefficients).  Thread sums -> warp shuffles -> shared
// memory -> 64-bit limb sums; the last block writes the canonical total (one REDC).
template <bool MUL>
__global__ void __launch_bounds__(256) k_gate_sums(uint64_t O, const uint32_t* __restrict__ off,
                                                   const uint32_t* __restrict__ gates, const Fr* __restrict__ coef,
                                                   const __grid_constant__ GateEqBn eq, unsigned long long* acc,
                                                   unsigned int* ticket, uint32_t* out) {
    Fr* const tz = reinterpret_cast<Fr*>(eqsm_raw);
    Fr* const tx = tz + eq_elems(eq.z);
    Fr* const ty = tx + eq_elems(eq.x);
    Fr* const u = ty + (MUL ? eq_elems(eq.y) : 0);
    eq_build(tz, u, eq.z);
    __syncthreads();
    eq_build(tx, u, eq.x);
    __syncthreads();
    if (MUL) eq_build(ty, u, eq.y);
    __syncthreads();
    const uint32_t ndz = eq_tables(eq.z), ndx = eq_tables(eq.x);
    Fr s = zero();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; o < O; o += stride) {
        const uint32_t k0 = __ldg(off + o), k1 = __ldg(off + o + 1);
        if (k0 == k1) continue;
        const Fr ez = eq_at(tz, ndz, eq.z.has_r2, (uint32_t)o);
        for (uint32_t k = k0; k < k1; k++) {
            Fr t;
            if (MUL) {
                const uint4 g = __ldg(reinterpret_cast<const uint4*>(gates) + k);  // (i0, i1, c, 0)
                t = mul(mul(eq_at(tx, ndx, false, g.x), eq_at(ty, ndx, false, g.y)), lds(coef, k));
            } else {
                const uint2 g = __ldg(reinterpret_cast<const uint2*>(gates) + k);  // (i0, c)
                t = mul(eq_at(tx, ndx, false, g.x), lds(coef, k));
            }
            s = add(s, mul(t, ez));
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        Fr o;
#pragma unroll
        for (int k = 0; k < 8; k++) o.l[k] = __shfl_xor_sync(0xffffffffu, s.l[k], d);
        s = add(s, o);
    }
    __shared__ Fr part[8];
    const uint32_t w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) part[w] = s;
    __syncthreads();
    if (threadIdx.x < 8) {
        unsigned long long limb = 0;
        for (uint32_t q = 0; q < nw; q++) limb += part[q].l[threadIdx.x];
        atomicAdd(&acc[threadIdx.x], limb);
    }
    __threadfence();
    __syncthreads();
    __shared__ unsigned int is_last;
    if (threadIdx.x == 0) is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (threadIdx.x == 0) {
        unsigned long long t[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            t[k] = __ldcg(acc + k);
            acc[k] = 0ull;
        }
        const Fr r = redc_sums(t);
#pragma unroll
        for (int k = 0; k < 8; k++) out[k] = r.l[k];
        *ticket = 0u;
    }
}

__global__ void __launch_bounds__(256, 2) k_hg_round0(const uint32_t* __restrict__ v, uint64_t I,
                                                   const uint32_t* __restrict__ mx_off, const uint4* __restrict__ mx_g,
                                                   const Fr* __restrict__ a, const Fr* __restrict__ w, uint32_t* hg,
                                                   GeoBn g, RedBn red, const uint32_t* claim, uint32_t* evals_out) {
    const Tile t = tile(g);
    Fr total[2] = {zero(), zero()};  // p0, p2raw
    Wide acc[2] = {lift(zero()), lift(zero())};
    uint64_t i = (uint64_t)blockIdx.x * g.rps + t.rs;
    while (t.active && i < (I >> 1)) {
        for (uint32_t n = 0; n < kWideTerms && i < (I >> 1); n++, i += (uint64_t)gridDim.x * g.rps) {
            Fr h0, h1;
            // not unrolled: each copy of the gate loop inlines a 256-bit product, and two of
            // them left this kernel waiting on instruction fetch (ncu: no_instruction stalls)
#pragma unroll 1
            for (int s = 0; s < 2; s++) {
                const uint64_t x = 2 * i + s;
                Fr h = lds(a, x);
                const uint32_t k0 = __ldg(mx_off + x), k1 = __ldg(mx_off + x + 1);
                for (uint32_t k = k0; k < k1; k++) h = add(h, mul(ldf(v, __ldg(&mx_g[k].x), g.N, t.q), lds(w, k)));
                stf(hg, x, g.N, t.q, h);
                if (s == 0) h0 = h;
                else h1 = h;
            }
            accum(acc, ldf(v, 2 * i, g.N, t.q), ldf(v, 2 * i + 1, g.N, t.q), h0, h1);
        }
        settle(acc, total);
    }
    reduce_bn<2>(total, g, t.active, red, ClaimFinBn{evals_out, red.evals_dev, claim, nullptr, nullptr, zero(), g.N});
}

template <bool LANE_HG, bool FOLD>
__global__ void __launch_bounds__(256, 2) k_round(RoundPtrsBn p, uint64_t npairs, const uint32_t* __restrict__ vx, GeoBn g,
                                               RedBn red, uint32_t* evals_out) {
    const Tile t = tile(g);
    Fr r;
#pragma unroll
    for (int k = 0; k < 8; k++) r.l[k] = p.r[k];
    // fold rounds sum p0 and p2raw (p1 from the claim), phase two's round 0 all three
    constexpr int C = FOLD ? 2 : 3;
    Fr total[C];
    Wide acc[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
        total[c] = zero();
        acc[c] = lift(total[c]);
    }
    const Fr* hs = reinterpret_cast<const Fr*>(p.hsrc);
    Fr* hd = reinterpret_cast<Fr*>(p.hdst);
    // Phase two folds the lane-independent scalar table: with a power-of-two row tile of at
    // least 2, the threads of a row slice within a warp share it (two of them fold, the
    // others take the results by shuffle), so the loop runs warp-uniformly.
    const bool share = !LANE_HG && FOLD && g.tpr >= 2 && (g.tpr & (g.tpr - 1)) == 0;
    const uint32_t grp = g.tpr < 32 ? g.tpr : 32;
    const uint32_t gq = threadIdx.x & (grp - 1);
    const uint32_t q = threadIdx.x % g.tpr;
    const uint64_t stride = (uint64_t)gridDim.x * g.rps;
    uint64_t i = (uint64_t)blockIdx.x * g.rps + t.rs;
    for (bool more = true; more;) {
        for (uint32_t n = 0; n < kWideTerms; n++, i += stride) {
            const bool valid = t.active && i < npairs;
            more = share ? __any_sync(0xffffffffu, valid) : valid;
            if (!more) break;
            Fr f0 = zero(), f1 = zero(), h0, h1;
            if (FOLD) {
                if (valid) {
                    f0 = fold(ldf(p.fsrc, 4 * i, g.N, t.q), ldf(p.fsrc, 4 * i + 1, g.N, t.q), r);
                    f1 = fold(ldf(p.fsrc, 4 * i + 2, g.N, t.q), ldf(p.fsrc, 4 * i + 3, g.N, t.q), r);
                    stf(p.fdst, 2 * i, g.N, t.q, f0);
                    stf(p.fdst, 2 * i + 1, g.N, t.q, f1);
                }
                if (LANE_HG) {
                    h0 = fold(ldf(p.hsrc, 4 * i, g.N, t.q), ldf(p.hsrc, 4 * i + 1, g.N, t.q), r);
                    h1 = fold(ldf(p.hsrc, 4 * i + 2, g.N, t.q), ldf(p.hsrc, 4 * i + 3, g.N, t.q), r);
                    stf(p.hdst, 2 * i, g.N, t.q, h0);
                    stf(p.hdst, 2 * i + 1, g.N, t.q, h1);
                } else if (share) {
                    Fr mine = zero();
                    if (valid && gq < 2) mine = fold(lds(hs, 4 * i + 2 * gq), lds(hs, 4 * i + 2 * gq + 1), r);
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        h0.l[k] = __shfl_sync(0xffffffffu, mine.l[k], 0, grp);
                        h1.l[k] = __shfl_sync(0xffffffffu, mine.l[k], 1, grp);
                    }
                } else {
                    h0 = fold(lds(hs, 4 * i), lds(hs, 4 * i + 1), r);
                    h1 = fold(lds(hs, 4 * i + 2), lds(hs, 4 * i + 3), r);
                }
                // the scalar table is shared by all lanes: the first thread of the row slice in
                // lane group 0 writes it
                if (!LANE_HG && valid && q == 0 && blockIdx.y == 0) {
                    sts(hd, 2 * i, h0);
                    sts(hd, 2 * i + 1, h1);
                }
            } else {
                f0 = ldf(p.fsrc, 2 * i, g.N, t.q);
                f1 = ldf(p.fsrc, 2 * i + 1, g.N, t.q);
                h0 = lds(hs, 2 * i);
                h1 = lds(hs, 2 * i + 1);
            }
            if (valid) accum(acc, f0, f1, h0, h1);
        }
        settle(acc, total);
    }
    if constexpr (FOLD)
        reduce_bn<2>(total, g, t.active, red,
                     ClaimFinBn{evals_out, red.evals_dev, nullptr, red.evals_prev, LANE_HG ? nullptr : vx, r, g.N});
    else
        reduce_bn<3>(total, g, t.active, red, RoundFinBn{evals_out, LANE_HG ? nullptr : vx, g.N, red.evals_dev});
}

__global__ void __launch_bounds__(256) k_s_build(uint64_t I, const uint32_t* __restrict__ my_off,
                                                 const uint4* __restrict__ my_g, const Fr* __restrict__ my_c,
                                                 const __grid_constant__ EqArgsBn eqc, const __grid_constant__ EqArgsBn eqx,
                                                 Fr* __restrict__ s_out) {
    Fr* const tz = reinterpret_cast<Fr*>(eqsm_raw);
    Fr* const tx = tz + eq_elems(eqc);
    Fr* const u = tx + eq_elems(eqx);
    eq_build(tz, u, eqc);
    eq_build(tx, u + eq_scratch(eqc), eqx);
    __syncthreads();
    const uint32_t ndz = eq_tables(eqc), ndx = eq_tables(eqx);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < kRowLanes * I; i += stride) {
        const uint64_t y = i / kRowLanes;
        const uint32_t l = (uint32_t)i % kRowLanes, k0 = __ldg(my_off + y), k1 = __ldg(my_off + y + 1);
        Fr s = zero();
        for (uint32_t k = k0 + l; k < k1; k += kRowLanes) {
            const uint4 gt = __ldg(my_g + k);  // (x, z, c, 0)
            s = add(s, mul(mul(eq_at(tz, ndz, eqc.has_r2, gt.y), eq_at(tx, ndx, false, gt.x)), lds(my_c, k)));
        }
        s = row_sum(s, k1 - k0);
        if (l == 0) sts(s_out, y, s);
    }
}

// sum_z eq(r, z) vals[z] (eval_multilinear); the weights of a block of rows are computed from
// the digit tables into shared memory.
constexpr uint32_t kWsumRows = 128;  // rows a CTA takes at a time

__global__ void __launch_bounds__(256) k_wsum(const uint32_t* __restrict__ vals, uint64_t rows,
                                              const __grid_constant__ EqArgsBn eq, GeoBn g, RedBn red, uint32_t* out) {
    __shared__ Fr w[kWsumRows];
    Fr* const tab = reinterpret_cast<Fr*>(eqsm_raw);  // then the reduction's scratch
    const Tile t = tile(g);
    eq_build(tab, tab + eq_elems(eq), eq);
    const uint32_t nd = eq_tables(eq);
    Fr total[1] = {zero()};
    Wide acc[1] = {lift(zero())};
    for (uint64_t z0 = (uint64_t)blockIdx.x * kWsumRows; z0 < rows; z0 += (uint64_t)gridDim.x * kWsumRows) {
        __syncthreads();  // the digit tables are built, the last block's weights are done with
        const uint32_t n = rows - z0 < kWsumRows ? (uint32_t)(rows - z0) : kWsumRows;
        if (threadIdx.x < n) w[threadIdx.x] = eq_at(tab, nd, false, (uint32_t)(z0 + threadIdx.x));
        __syncthreads();
        for (uint32_t i = t.rs; t.active && i < n;) {
            for (uint32_t k = 0; k < kWideTerms && i < n; k++, i += g.rps) mac(acc[0], w[i], ldf(vals, z0 + i, g.N, t.q));
            settle(acc, total);
        }
    }
    __syncthreads();
    reduce_bn<1>(total, g, t.active, red, CopyFinBn{out, g.N});
}

// ---------------------------------------------------------------- persistent phases
// The rounds of a phase on small tables in one launch (the M31 k_phase of phase.cu, whose
// notes on the host traffic hold here): a round launched by itself takes 18-27 us on tables
// of a few hundred rows, mostly the launch, the reduction across CTAs and a chain of dependent
// 256-bit products in one finishing thread.  One CTA owns one copy and all its rows (a row's
// element is one 32-byte sector, so narrower is no loss).  Four lanes take a pair: each folds
// one of f0, f1, h0, h1, then three of them form the products of the three sums, so a round's
// chain is two products and the finisher's one (with a thread a pair it was seven in a row).
constexpr uint32_t kPhaseBlock = 256;
constexpr uint32_t kPhaseWarps = kPhaseBlock / 32;
constexpr uint32_t kSmemRowsBn = 128;  // rows of a per-copy table kept in shared memory
constexpr uint32_t kSpinsBn = 256;     // mailbox polls before sleeping between them

__device__ __forceinline__ void st_digits(uint32_t* out, const Fr& v, uint32_t parity) {
    uint32_t d[12];
    const uint32_t top = parity << 31;
    d[0] = (v.l[0] & 0x7fffffffu) | top;
#pragma unroll
    for (int k = 1; k < 8; k++) d[k] = (__funnelshift_l(v.l[k - 1], v.l[k], k) & 0x7fffffffu) | top;
    d[8] = (v.l[7] >> 24) | top;
    d[9] = d[10] = d[11] = top;
#pragma unroll
    for (int k = 0; k < 3; k++)
        asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(out + 4 * k), "r"(d[4 * k]),
                     "r"(d[4 * k + 1]), "r"(d[4 * k + 2]), "r"(d[4 * k + 3])
                     : "memory");
}
// Reads a mailbox slot: 0 not written yet, 1 the challenge is in *r, 2 abort.
__device__ __forceinline__ int ld_challenge(const uint32_t* box, Fr* r) {
    uint32_t d[12];
#pragma unroll
    for (int k = 0; k < 3; k++)
        asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(d[4 * k]), "=r"(d[4 * k + 1]), "=r"(d[4 * k + 2]), "=r"(d[4 * k + 3])
                     : "l"(box + 4 * k)
                     : "memory");
    uint32_t ok = d[0];
#pragma unroll
    for (int k = 1; k < 9; k++) ok &= d[k];
    if (!(ok >> 31)) return d[11] ? 2 : 0;
#pragma unroll
    for (int k = 0; k < 9; k++) d[k] &= 0x7fffffffu;
#pragma unroll
    for (int i = 0; i < 8; i++) r->l[i] = (d[i] >> i) | (d[i + 1] << (31 - i));
    return 1;
}
// Element of a table this kernel also writes (no read-only path); row r at p[r * stride].
struct RowsBn {
    Fr* p;
    size_t stride;
    __device__ __forceinline__ Fr get(uint32_t r) const {
        const uint4* q = reinterpret_cast<const uint4*>(p + (size_t)r * stride);
        const uint4 a = q[0], b = q[1];
        Fr f;
        f.l[0] = a.x; f.l[1] = a.y; f.l[2] = a.z; f.l[3] = a.w;
        f.l[4] = b.x; f.l[5] = b.y; f.l[6] = b.z; f.l[7] = b.w;
        return f;
    }
    __device__ __forceinline__ void set(uint32_t r, const Fr& f) const { sts(p, (size_t)r * stride, f); }
};

template <bool LANE_HG>
__global__ void __launch_bounds__(kPhaseBlock, 2) k_phase(PhaseArgsBn a) {
    extern __shared__ uint4 psm_raw[];
    __shared__ Fr rch, part[kPhaseWarps][3];
    __shared__ int stop;
    const uint32_t tid = threadIdx.x, lane = blockIdx.x, warp = tid >> 5;
    const size_t gs = a.N;
    constexpr uint32_t kTabs = LANE_HG ? 2 : 1;
    const uint32_t kf = a.k0 ? a.k0 : 1, S1 = 1u << (a.n - kf);  // the first round that folds leaves S1 rows
    Fr* const psm = reinterpret_cast<Fr*>(psm_raw);              // two buffers of f (and hg)
    Fr* const sbuf = psm + 2 * kTabs * kSmemRowsBn;              // phase two's scalar tables, S1 and S1 / 2
    auto mem = [&](uint32_t* b) { return RowsBn{reinterpret_cast<Fr*>(b) + lane, gs}; };
    // the table round k leaves: which = 0 f, 1 hg
    auto table = [&](uint32_t k, uint32_t which) -> RowsBn {
        if ((1u << (a.n - k)) <= kSmemRowsBn) return RowsBn{psm + ((k & 1) * kTabs + which) * kSmemRowsBn, 1};
        return mem(which == 0 ? ((k & 1) ? a.fA : a.fB) : ((k & 1) ? a.hA : a.hB));
    };
    // a published sum is a Montgomery form times a canonical value: v(rx) in phase two, else 1
    Fr xv = zero();
    xv.l[0] = 1u;
    if (!LANE_HG && tid < 3) xv = ldf_cv(a.vx, a.N, lane);
    const uint32_t e = tid & 3, quad = tid & 28;  // lane's part of its pair, the pair's first lane
    if (tid == 0) stop = 0;

    for (uint32_t k = a.k0; k < a.n; k++) {
        if (tid == 0) {
            if (k == a.k0) {
#pragma unroll
                for (int i = 0; i < 8; i++) rch.l[i] = a.r_first[i];
            } else {
                const uint32_t* box = a.mbox + kDigitWords * (k - 1);
                uint64_t t0 = 0;
                for (uint32_t it = 0;; it++) {
                    Fr r;
                    const int got = ld_challenge(box, &r);
                    if (got == 1) rch = r;
                    if (got == 2) stop = 1;
                    if (got) break;
                    if (it < kSpinsBn) continue;
                    uint64_t now;
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                    if (t0 == 0) t0 = now;
                    if (now - t0 > a.wait_ns) {
                        *reinterpret_cast<volatile unsigned int*>(a.err) = 1u;
                        stop = 1;
                        break;
                    }
                    __nanosleep(100);
                }
            }
        }
        __syncthreads();  // the challenge, and the previous round's tables, are visible
        if (stop) return;
        const uint32_t npairs = 1u << (a.n - k - 1);
        const Fr r = rch;
        // this lane's source and destination tables: f for e < 2, else hg or the scalars
        RowsBn src = mem(const_cast<uint32_t*>(a.v)), dst = {};
        if (k > 0) {
            if (e < 2) {
                if (k == a.k0) src = mem((k & 1) ? a.fB : a.fA);
                else if (k > 1) src = table(k - 1, 0);
                dst = table(k, 0);
            } else if (LANE_HG) {
                src = k == a.k0 ? mem((k & 1) ? a.hB : a.hA) : k == 1 ? mem(a.h0) : table(k - 1, 1);
                dst = table(k, 1);
            } else {
                const bool odd = (k - kf) & 1;
                src = RowsBn{k > kf ? (odd ? sbuf : sbuf + S1) : const_cast<Fr*>(a.s), 1};
                dst = RowsBn{odd ? sbuf + S1 : sbuf, 1};
            }
        }
        const uint32_t nw = npairs >= 8 * kPhaseWarps ? kPhaseWarps : (npairs + 7) / 8;  // warps with pairs
        Fr acc = zero(), mine = zero();
        if (warp < nw) {
#pragma unroll 1
            for (uint32_t i0 = 8 * warp; i0 < npairs; i0 += 8 * kPhaseWarps) {
                const uint32_t i = i0 + ((tid & 31) >> 2);
                mine = zero();
                if (i < npairs) {
                    if (k > 0) {
                        const uint32_t x = 4 * i + 2 * (e & 1);
                        mine = fold(src.get(x), src.get(x + 1), r);
                        dst.set(2 * i + (e & 1), mine);
                    } else if (e < 2) {
                        mine = ldf(a.v, 2 * i + e, a.N, lane);
                    } else if (LANE_HG) {
                        const uint32_t x = 2 * i + (e & 1);
                        mine = lds(a.a, x);
                        const uint32_t g0 = __ldg(a.mx_off + x), g1 = __ldg(a.mx_off + x + 1);
                        for (uint32_t g = g0; g < g1; g++)
                            mine = add(mine, mul(ldf(a.v, __ldg(&a.mx_g[g].x), a.N, lane), lds(a.w, g)));
                        mem(a.h0).set(x, mine);
                    } else {
                        mine = lds(a.s, 2 * i + (e & 1));
                    }
                }
                __syncwarp();
                // lanes 0, 1: f times h (of lanes 2, 3); lane 2: (f0 + f1)(h0 + h1)
                Fr p, q, u;
#pragma unroll
                for (int l = 0; l < 8; l++) {
                    p.l[l] = __shfl_sync(0xffffffffu, mine.l[l], quad | (e ^ 2));
                    q.l[l] = __shfl_sync(0xffffffffu, mine.l[l], quad | 1);
                    u.l[l] = __shfl_sync(0xffffffffu, mine.l[l], quad | 3);
                }
                const Fr x = e < 2 ? mine : add(p, q), y = e < 2 ? p : add(mine, u);
                acc = add(acc, mul(x, y));
            }
            // lane e of a warp's first pair collects component e
            for (uint32_t off = npairs < 8 ? 2 * npairs : 16; off >= 4; off >>= 1) {
                Fr o;
#pragma unroll
                for (int l = 0; l < 8; l++) o.l[l] = __shfl_xor_sync(0xffffffffu, acc.l[l], off);
                acc = add(acc, o);
            }
            if (nw > 1 && (tid & 31) < 3) part[warp][tid & 31] = acc;
        }
        if (nw > 1) __syncthreads();
        const uint32_t par = (a.parity ^ (k - a.k0)) & 1u;
        if (tid < 3) {
            Fr v = acc;
            for (uint32_t w = 1; w < nw; w++) v = add(v, part[w][tid]);
            // evaluation 2 from the three sums: 6 p1 + 3 p0 - 2 p2raw
            Fr p0, p1;
#pragma unroll
            for (int l = 0; l < 8; l++) {
                p0.l[l] = __shfl_sync(0x7u, v.l[l], 0);
                p1.l[l] = __shfl_sync(0x7u, v.l[l], 1);
            }
            if (tid == 2) {
                const Fr d = add(p1, p1);
                v = sub(add(add(add(d, d), d), add(add(p0, p0), p0)), add(v, v));
            }
            st_digits(a.evals_out + ((size_t)tid * a.N + lane) * kDigitWords, mul(v, xv), par);
            // rows 0 and 1 of the last f table are what lanes 0 and 1 hold
            if (k + 1 == a.n && tid < 2)
                st_digits(a.rows_out + ((size_t)tid * a.N + lane) * kDigitWords, mine, a.rows_parity);
        }
    }
}

uint32_t grid1(uint64_t n) {
    uint64_t b = (n + 255) / 256;
    if (b < 1) b = 1;
    if (b > 152ull * 16) b = 152ull * 16;
    return (uint32_t)b;
}

// CTAs of a kernel that builds eq tables: two an SM at most, since each CTA's build is up to six
// products a thread (1024 CTAs of a 2^16-row layer spent 22 us of 50 on it).
uint32_t grid_eq(uint64_t n) { return std::min(grid1(n), 2u * 152u); }

dim3 grid_rows(const GeoBn& g, uint64_t rows, uint32_t ctas) {
    const uint32_t groups = g.N / g.tpr;
    uint64_t need = (rows + g.rps - 1) / g.rps;
    uint64_t cap = ctas / groups;
    if (cap < 1) cap = 1;
    if (need < 1) need = 1;
    return dim3((uint32_t)(need < cap ? need : cap), groups, 1);
}

}  // namespace

// Dynamic shared memory of a kernel that builds eq tables; above 48 KiB the opt-in is set once
// per device and kernel (30 variables at four points: 140 KiB).
template <auto Kernel>
static cudaError_t eq_smem(size_t bytes) {
    static std::atomic<uint64_t> opted{0};  // one bit per device
    if (bytes <= 40 * 1024) return cudaSuccess;
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (opted.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    if (e == cudaSuccess) opted.fetch_or(bit);
    return e;
}

cudaError_t launch_load(const uint32_t* canon, uint32_t* mont, uint64_t n_elems, unsigned int* bad, cudaStream_t s) {
    k_load<<<grid1(n_elems), 256, 0, s>>>(canon, mont, n_elems, bad);
    return cudaGetLastError();
}

cudaError_t launch_gate_sums(bool mul_gates, uint64_t O, const uint32_t* off, const uint32_t* gates, const Fr* coef,
                             const GateEqBn& eq, unsigned long long* acc, unsigned int* ticket, uint32_t* out,
                             cudaStream_t s) {
    const uint32_t grid = grid_eq(O);
    const uint32_t u = std::max(eq_scratch(eq.z), eq_scratch(eq.x));
    const size_t smem = sizeof(Fr) * (eq_elems(eq.z) + eq_elems(eq.x) + (mul_gates ? eq_elems(eq.y) : 0) + u);
    const cudaError_t e = mul_gates ? eq_smem<k_gate_sums<true>>(smem) : eq_smem<k_gate_sums<false>>(smem);
    if (e != cudaSuccess) return e;
    if (mul_gates)
        k_gate_sums<true><<<grid, kBlock, smem, s>>>(O, off, gates, coef, eq, acc, ticket, out);
    else
        k_gate_sums<false><<<grid, kBlock, smem, s>>>(O, off, gates, coef, eq, acc, ticket, out);
    return cudaGetLastError();
}

cudaError_t launch_unload(uint32_t* v, uint64_t n_elems, cudaStream_t s) {
    k_unload<<<grid1(n_elems), 256, 0, s>>>(v, n_elems);
    return cudaGetLastError();
}

cudaError_t launch_evaluate(const uint32_t* in, uint32_t* out, uint64_t O, const uint32_t* mo_off, const uint4* mo_g,
                            const Fr* mo_c, const uint32_t* ao_off, const uint2* ao_g, const Fr* ao_c, const GeoBn& g,
                            uint32_t ctas, cudaStream_t s) {
    k_evaluate<<<grid_rows(g, O, ctas), 256, 0, s>>>(in, out, O, mo_off, mo_g, mo_c, ao_off, ao_g, ao_c, g);
    return cudaGetLastError();
}

cudaError_t launch_weights(uint64_t I, uint64_t Gm, const EqArgsBn& eqc, const uint4* mx_g, const Fr* mx_c,
                           const uint32_t* ax_off, const uint2* ax_g, const Fr* ax_c, Fr* a_out, Fr* w_out,
                           cudaStream_t s) {
    const size_t smem = sizeof(Fr) * (eq_elems(eqc) + eq_scratch(eqc));
    if (const cudaError_t e = eq_smem<k_weights>(smem)) return e;
    k_weights<<<grid_eq(kRowLanes * I > Gm ? kRowLanes * I : Gm), 256, smem, s>>>(I, Gm, eqc, mx_g, mx_c, ax_off, ax_g, ax_c, a_out, w_out);
    return cudaGetLastError();
}

cudaError_t launch_hg_round0(const uint32_t* v, uint64_t I, const uint32_t* mx_off, const uint4* mx_g, const Fr* a,
                             const Fr* w, uint32_t* hg, const GeoBn& g, uint32_t ctas, RedBn red, const uint32_t* claim,
                             uint32_t* evals_out, cudaStream_t s) {
    if (!claim) return cudaErrorInvalidValue;
    k_hg_round0<<<grid_rows(g, I / 2, ctas), 256, 3 * 8 * 256 * 4, s>>>(v, I, mx_off, mx_g, a, w, hg, g, red, claim,
                                                                       evals_out);
    return cudaGetLastError();
}

cudaError_t launch_round(bool lane_hg, bool fold_, const RoundPtrsBn& p, uint64_t npairs, const uint32_t* vx,
                         const GeoBn& g, uint32_t ctas, RedBn red, uint32_t* evals_out, cudaStream_t s) {
    const dim3 grid = grid_rows(g, npairs, ctas);
    const size_t smem = 3 * 8 * 256 * 4;
    if (fold_ && (!red.evals_prev || red.evals_prev == red.evals_dev)) return cudaErrorInvalidValue;
    if (lane_hg && fold_) k_round<true, true><<<grid, 256, smem, s>>>(p, npairs, vx, g, red, evals_out);
    else if (!lane_hg && fold_) k_round<false, true><<<grid, 256, smem, s>>>(p, npairs, vx, g, red, evals_out);
    else if (!lane_hg && !fold_) k_round<false, false><<<grid, 256, smem, s>>>(p, npairs, vx, g, red, evals_out);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// Shared memory of a launch whose first folding round leaves S1 rows.
static size_t phase_smem(bool lane_hg, uint32_t S1) {
    return sizeof(Fr) * (2 * (lane_hg ? 2 : 1) * (size_t)kSmemRowsBn + (lane_hg ? 0 : S1 + S1 / 2));
}

int phase_ctas_per_sm() {
    static std::atomic<int> known[64];  // of each device, plus one
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int>& k = known[dev & 63];
    if (const int v = k.load(std::memory_order_relaxed)) return v - 1;
    int least = 0;
    for (int lane_hg = 0; lane_hg < 2; lane_hg++) {
        auto* const kernel = lane_hg ? k_phase<true> : k_phase<false>;
        const size_t most = phase_smem(lane_hg != 0, kPhaseRows / 2);
        int n = 0;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kPhaseBlock, most);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (lane_hg == 0 || n < least) least = n;
    }
    k.store(least + 1, std::memory_order_relaxed);
    return least;
}

cudaError_t launch_phase(bool lane_hg, const PhaseArgsBn& a, bool dense, cudaStream_t s) {
    if (a.k0 >= a.n || a.n - a.k0 > kMboxRounds || a.N < 1) return cudaErrorInvalidValue;
    // rows of the first round's source tables; with k0 = 0 the layer input itself
    if ((1ull << (a.n - (a.k0 ? a.k0 - 1 : 0))) > kPhaseRows) return cudaErrorInvalidValue;
    if (a.k0 == 0 && (!a.v || (lane_hg && (!a.h0 || !a.mx_off || !a.a || !a.w)))) return cudaErrorInvalidValue;
    if (!lane_hg && (!a.vx || !a.s)) return cudaErrorInvalidValue;
    if (phase_ctas_per_sm() < 1) return cudaErrorInvalidConfiguration;
    const uint32_t kf = a.k0 ? a.k0 : 1, S1 = 1u << (a.n - kf);
    const size_t smem = phase_smem(lane_hg, S1);
    auto* const kernel = lane_hg ? k_phase<true> : k_phase<false>;
    if (!dense) {
        kernel<<<a.N, kPhaseBlock, smem, s>>>(a);
        return cudaGetLastError();
    }
    cudaLaunchAttribute split;
    split.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    split.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.N);
    cfg.blockDim = dim3(kPhaseBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &split;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

cudaError_t launch_s_build(uint64_t I, const uint32_t* my_off, const uint4* my_g, const Fr* my_c, const EqArgsBn& eqc,
                           const EqArgsBn& eqx, Fr* s_out, cudaStream_t s) {
    const size_t smem = sizeof(Fr) * (eq_elems(eqc) + eq_elems(eqx) + eq_scratch(eqc) + eq_scratch(eqx));
    if (const cudaError_t e = eq_smem<k_s_build>(smem)) return e;
    k_s_build<<<grid_eq(kRowLanes * I), 256, smem, s>>>(I, my_off, my_g, my_c, eqc, eqx, s_out);
    return cudaGetLastError();
}

cudaError_t launch_wsum(const uint32_t* vals, const EqArgsBn& eq, const GeoBn& g, uint32_t ctas, RedBn red,
                        uint32_t* out, cudaStream_t s) {
    const uint64_t rows = 1ull << eq.nvars, need = (rows + kWsumRows - 1) / kWsumRows;
    const uint32_t groups = g.N / g.tpr, cap = ctas / groups ? ctas / groups : 1;
    const dim3 grid((uint32_t)(need < cap ? need : cap), groups, 1);
    const size_t tabs = sizeof(Fr) * (eq_elems(eq) + eq_scratch(eq)), scratch = 8 * 256 * 4;
    const size_t smem = tabs > scratch ? tabs : scratch;
    if (const cudaError_t e = eq_smem<k_wsum>(smem)) return e;
    k_wsum<<<grid, 256, smem, s>>>(vals, rows, eq, g, red, out);
    return cudaGetLastError();
}

}  // namespace bn
}  // namespace gkrgpu
