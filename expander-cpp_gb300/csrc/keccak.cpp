// Keccak-f[1600] and the Keccak-256 / SHA3-256 sponges (keccak.hpp), written from the
// permutation's definition (theta, rho, pi, chi, iota on a 5 x 5 array of 64-bit lanes).
// The round constants and rotation offsets are derived at compile time from their definitions
// (the degree-8 LFSR x^8 + x^6 + x^5 + x^4 + 1 and the triangular offsets along the pi walk)
// rather than tabulated.
#include "keccak.hpp"

#include <string.h>

namespace gkrgpu {
namespace {

struct Tables {
    uint64_t rc[24];
    unsigned rot[25];  // rot[x + 5 y]
};
constexpr Tables make_tables() {
    Tables t{};
    // bit j + 7 i of the LFSR's output is bit 2^j - 1 of round i's constant
    unsigned r = 1;
    for (unsigned i = 0; i < 24; i++)
        for (unsigned j = 0; j < 7; j++) {
            t.rc[i] |= (uint64_t)(r & 1) << ((1u << j) - 1);
            r <<= 1;
            if (r & 0x100) r ^= 0x171;
        }
    unsigned x = 1, y = 0;
    for (unsigned k = 0; k < 24; k++) {
        t.rot[x + 5 * y] = ((k + 1) * (k + 2) / 2) % 64;
        const unsigned nx = y, ny = (2 * x + 3 * y) % 5;
        x = nx;
        y = ny;
    }
    return t;
}
constexpr Tables kT = make_tables();

inline uint64_t rotl(uint64_t v, unsigned n) { return n ? (v << n) | (v >> (64 - n)) : v; }

// a[x + 5 y].  Every loop over the lanes is unrolled, so that the rotations have constant
// amounts and the lanes stay in registers.
void keccak_f(uint64_t a[25]) {
    uint64_t s[25];
    memcpy(s, a, sizeof(s));
    for (int round = 0; round < 24; round++) {
        uint64_t c[5], b[25];
#pragma GCC unroll 5
        for (int x = 0; x < 5; x++) c[x] = s[x] ^ s[x + 5] ^ s[x + 10] ^ s[x + 15] ^ s[x + 20];
#pragma GCC unroll 5
        for (int x = 0; x < 5; x++) {
            const uint64_t d = c[(x + 4) % 5] ^ rotl(c[(x + 1) % 5], 1);
#pragma GCC unroll 5
            for (int y = 0; y < 5; y++) b[y + 5 * ((2 * x + 3 * y) % 5)] = rotl(s[x + 5 * y] ^ d, kT.rot[x + 5 * y]);
        }
#pragma GCC unroll 5
        for (int y = 0; y < 5; y++)
#pragma GCC unroll 5
            for (int x = 0; x < 5; x++) s[x + 5 * y] = b[x + 5 * y] ^ (~b[(x + 1) % 5 + 5 * y] & b[(x + 2) % 5 + 5 * y]);
        s[0] ^= kT.rc[round];
    }
    memcpy(a, s, sizeof(s));
}

void sponge256(const uint8_t* in, size_t len, uint8_t domain, uint8_t out[32]) {
    constexpr size_t rate = 136;
    uint64_t a[25];
    memset(a, 0, sizeof(a));
    auto absorb = [&](const uint8_t* blk) {
        for (size_t i = 0; i < rate / 8; i++) {
            uint64_t w;
            memcpy(&w, blk + 8 * i, 8);  // (both hosts are little-endian)
            a[i] ^= w;
        }
        keccak_f(a);
    };
    while (len >= rate) {
        absorb(in);
        in += rate;
        len -= rate;
    }
    uint8_t last[rate];
    memset(last, 0, rate);
    if (len) memcpy(last, in, len);
    last[len] ^= domain;
    last[rate - 1] ^= 0x80;
    absorb(last);
    memcpy(out, a, 32);
}

}  // namespace

void keccak256(const uint8_t* in, size_t len, uint8_t out[32]) { sponge256(in, len, 0x01, out); }
void sha3_256(const uint8_t* in, size_t len, uint8_t out[32]) { sponge256(in, len, 0x06, out); }

}  // namespace gkrgpu

extern "C" {
// Exported for the tests (checked against a SHA3-256 implementation and known digests).
void gkrgpu_keccak256(const uint8_t* in, uint64_t len, uint8_t* out) { gkrgpu::keccak256(in, (size_t)len, out); }
void gkrgpu_sha3_256(const uint8_t* in, uint64_t len, uint8_t* out) { gkrgpu::sha3_256(in, (size_t)len, out); }
}
