// Bit-sliced edit distance: 32 patterns per machine word, one matrix cell per
// step. Compiles as CUDA device code and as plain C++ (blg_hostcheck.cpp
// checks it against the oracle on the CPU).
//
// The column methods (blg_device.cuh) give one pair's pattern positions the
// bits of a word, so the horizontal delta has to ripple through the word: an
// add with its carry chain and four shifts beside the logic, about 18 ALU
// operations per 64 cells. Here bit q of every word belongs to pattern q of a
// group of 32, and a step advances ONE cell (row i, column j) of all 32
// matrices. With the deltas of the cell's left edge (vertical: vp = +1, vm =
// -1) and top edge (horizontal: hp, hm), the diagonal delta is 0 exactly when
// the characters match or a -1 comes in (Hyyro's D0), and both outgoing
// deltas follow from it without any carry (the recurrence of csrc/myers.c:
// 22-36 for one row):
//   N   = ~(eq | vm | hm)         diagonal delta +1
//   hp' = vm | (N & ~vp)          hm' = vp & ~N
//   vp' = hm | (N & ~hp)          vm' = hp & ~N
// Five three-input operations per 32 cells.
#pragma once
#include "blg_device.cuh"

namespace blg {

// Run-time multipliers 1 and -1 of the cell step's multiply-adds (see Units
// in blg_device.cuh: constants would be folded back into ALU adds).
struct BitUnits {
    uint32_t one, neg;
};

// One three-input operation as written: left to itself the compiler absorbs
// vm into vm | ~(eq | vm | hm | vp) and loses the shared D0, 6.3 ALU
// operations a cell for five.
template <int LUT>
BLG_HD uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(r) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return r;
#else
    uint32_t r = 0;
    for (int x = 0; x < 8; x++)
        if (LUT >> x & 1) r |= (x & 4 ? a : ~a) & (x & 2 ? b : ~b) & (x & 1 ? c : ~c);
    return r;
#endif
}

// One cell of 32 matrices. eq: the patterns whose character at this row is the
// column's; vn = ~vp. FMA: hp' as (vm + vn) + (hm' - d0), three multiply-adds in
// place of one ALU operation (hp' = vm | (N & ~vp) with N = ~d0; the two are
// disjoint and N & vp = vp - hm', so it is vm + N - vp + hm' with no bit
// carrying, and -vp - 1 is vn, -1 - d0 is N). The ALU pipe does half the lanes
// of a warp per clock and is what this loop runs against, while the FMA pipe
// has little else to do.
template <bool FMA>
BLG_HD void bit_cell(uint32_t eq, uint32_t &vn, uint32_t &vm, uint32_t &hp, uint32_t &hm, BitUnits u) {
    const uint32_t d0 = lop3<0xfe>(eq, vm, hm);              // eq | vm | hm
    const uint32_t hm2 = d0 & ~vn;
    const uint32_t hp2 = FMA ? imad_lo(imad_lo(d0, u.neg, hm2), u.one, imad_lo(vm, u.one, vn))
                             : lop3<0xf2>(vm, d0, vn);       // vm | (~d0 & vn)
    const uint32_t vm2 = hp & d0;
    vn = lop3<0x0e>(hm, d0, hp);                             // ~hm & (d0 | hp)
    vm = vm2;
    hp = hp2;
    hm = hm2;
}

// Bit-sliced counters: plane p holds bit p of 32 counts.
constexpr int kBitPlanes = 11;                  // of a whole query: counts up to 2 x 512

BLG_HD void bit_full_add(uint32_t &sum, uint32_t &carry, uint32_t a, uint32_t b) {
    const uint32_t s = sum ^ a ^ b;
    carry = (sum & a) | (sum & b) | (a & b);
    sum = s;
}

// counts (eight planes) += the eight one-bit inputs x[0..7]
BLG_HD void bit_count8(uint32_t (&pl)[8], const uint32_t (&x)[8]) {
    uint32_t a, b, c, d, e;
    bit_full_add(pl[0], a, x[0], x[1]);
    bit_full_add(pl[0], b, x[2], x[3]);
    bit_full_add(pl[1], c, a, b);
    bit_full_add(pl[0], a, x[4], x[5]);
    bit_full_add(pl[0], b, x[6], x[7]);
    bit_full_add(pl[1], d, a, b);
    bit_full_add(pl[2], e, c, d);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int p = 3; p < 8; p++) {       // ripple the carry of weight 8
        const uint32_t t = pl[p] & e;
        pl[p] ^= e;
        e = t;
    }
}

// Eight planes of 32 bits -> 32 bytes: byte t of x[r] = the 8-bit count of bit
// 8t + r (an 8 x 8 bit transpose of every byte position, three rounds of
// masked swaps).
BLG_HD void bit_transpose8(uint32_t (&x)[8]) {
    auto swap = [](uint32_t &lo, uint32_t &hi, int s, uint32_t m) {
        const uint32_t t = ((lo >> s) ^ hi) & m;
        hi ^= t;
        lo ^= t << s;
    };
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 4; i++) swap(x[i], x[i + 4], 4, 0x0f0f0f0fu);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 8; i++)
        if (!(i & 2)) swap(x[i], x[i + 2], 2, 0x33333333u);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 8; i += 2) swap(x[i], x[i + 1], 1, 0x55555555u);
}

}  // namespace blg
