// 4-gram signatures and the count of what two of them share as a matrix
// product. Compiles as CUDA device code and as plain C++ (blg_hostcheck.cpp).
//
// A string's signature is the set of bins its 4-grams fall into, 248 bins, one
// bit each. One edit removes at most 4 grams of a string and adds at most 4,
// and a gram's coming or going changes at most one bin, so |X ^ Y| <= 8 d(x, y)
// (the q-gram lemma for sets; merging grams into bins only lowers the left
// side). With |X ^ Y| = |X| + |Y| - 2 |X & Y| the test for 128 x 256 pairs is a
// 128 x 256 x 256 product of 0/1 matrices: the tensor cores run it in 8-bit
// floats (e4m3), sums in FP32, exact here. The 8 bits left over in a row of 256
// carry the rest of the test, so that the sign of the sum is the answer:
//   sum = |X & Y| / 2 - |X| / 4 - |Y| / 4 + 2 k + 1/8  >= 0  iff  |X ^ Y| <= 8 k
#pragma once
#include "blg_device.cuh"

namespace blg {

constexpr int kSigWords = 8;                     // 32 bytes per string
constexpr int kSigBins = 248;                    // bits 6 and 7 of the last word's bytes stay 0
constexpr int kSigMaxK = 15;                     // largest k whose e4m3 is exact as it stands

// bin of a 4-gram g (its bytes in order, first highest), and its bit's position (word << 5 | bit)
BLG_HD uint32_t sig_bin(uint32_t g) { return (((g * 0x9E3779B1u) >> 16) * (uint32_t)kSigBins) >> 16; }
BLG_HD uint32_t sig_bit(uint32_t g) {
    const uint32_t bin = sig_bin(g);
    if (bin < 224u) return bin;
    const uint32_t r = bin - 224u;               // 24 bins: six low bits of each byte of the last word
    return 224u + 8u * (r / 6u) + r % 6u;
}

// Half the bins, for rows of 128 bytes: bins are merged in pairs, and the eight
// whose place the tail takes are left out (fewer bins only lower |X ^ Y|).
BLG_HD void sig_fold(uint32_t *w) {
    for (int i = 0; i < 4; i++) w[i] |= w[i + 4];
    w[3] &= 0x3f3f3f3fu;
}

// e4m3 of an integer 0..15 (four significant bits: exact)
BLG_HD uint32_t e4m3_int(uint32_t v) {
    if (v == 0) return 0;
    uint32_t e = v >= 8 ? 3 : v >= 4 ? 2 : v >= 2 ? 1 : 0;
    return ((e + 7u) << 3) | ((v << (3u - e)) & 7u);
}

// A row of 256 e4m3 bytes as 64 words: word 8 i + s holds bits s, s + 8, s + 16
// and s + 24 of signature word i. The choices' side keeps the masked bits
// as they lie (value of a byte with only bit s set: 2^-9, -8, -7, -6, -5, -3, 2
// for s = 0 .. 6), the queries' side holds 2^-1 over that value; s = 7 would be
// the sign, so it is shifted to 6.
BLG_HD uint32_t sig_choice_word(const uint32_t *w, int i, int s) {
    return s == 7 ? (w[i] >> 1) & 0x40404040u : w[i] & (0x01010101u << s);
}
BLG_HD uint32_t sig_query_word(const uint32_t *w, int i, int s) {
    // e4m3 of 2^-1 / value(s): 2^8, 2^7, 2^6, 2^5, 2^4, 2^2, 2^-2, 2^-2
    const uint32_t v = s == 0 ? 0x78u : s == 1 ? 0x70u : s == 2 ? 0x68u : s == 3 ? 0x60u : s == 4 ? 0x58u : s == 5 ? 0x48u : 0x28u;
    return ((w[i] >> s) & 0x01010101u) * v;
}

// The last two words of a row: the rest of the test, eight products
//   query  -4      -1/4     |X|>>4   |X|&15   2   1/8 (no query: 0)    0 (no query: -256)   0
//   choice |Y|>>4  |Y|&15   -4       -1/4     k   1 (no choice: -448)  1                    0
// A row without a query or a column without a choice comes out negative.
BLG_HD void sig_query_tail(int bits, bool valid, uint32_t &lo, uint32_t &hi) {
    const uint32_t m4 = 0xc8u, mq = 0xa8u, two = 0x40u, eighth = 0x20u, m256 = 0xf8u;
    lo = valid ? m4 | (mq << 8) | (e4m3_int((uint32_t)bits >> 4) << 16) | (e4m3_int((uint32_t)bits & 15u) << 24) : 0u;
    hi = valid ? two | (eighth << 8) : m256 << 16;
}
BLG_HD void sig_choice_tail(int bits, int k, bool valid, uint32_t &lo, uint32_t &hi) {
    const uint32_t m4 = 0xc8u, mq = 0xa8u, one = 0x38u, m448 = 0xfeu;
    lo = valid ? e4m3_int((uint32_t)bits >> 4) | (e4m3_int((uint32_t)bits & 15u) << 8) | (m4 << 16) | (mq << 24) : 0u;
    hi = valid ? e4m3_int((uint32_t)k) | (one << 8) | (one << 16) : (m448 << 8) | (one << 16);
}

}  // namespace blg
