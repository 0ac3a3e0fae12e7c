// Host build of the device primitives (blg_device.cuh) for the CPU tests.
//
// The same step/score/saturation functions the kernels call are compiled
// here with g++ and driven two ways:
//  * blg_host_distance: pattern = shorter trimmed string, words processed
//    top to bottom in one column (the order k_search_seq uses);
//  * blg_host_wavefront: the anti-diagonal lane schedule of the
//    lane-spread kernels, emulated step by step: "lane" w handles column
//    s - w at step s and reads the carry lane w-1 produced one step earlier
//    (what __shfl_up_sync delivers on the GPU), with the max_dist exit
//    decided by the last word's lane.
// Both must equal the oracle for every input.
#include <cstdint>
#include <cstring>
#include <vector>

#include "blg_bits.cuh"
#include "blg_device.cuh"
#include "blg_sig.cuh"

using namespace blg;

namespace {

struct Pattern {
    int m = 0, words = 0;
    std::vector<uint64_t> peq;   // 256 x words
    Pattern(const uint8_t *p, int m_) : m(m_), words(m_ > 0 ? (m_ + 63) / 64 : 1), peq(256 * (size_t)words, 0) {
        for (int i = 0; i < m; i++) peq[(size_t)p[i] * words + i / 64] |= 1ull << (i % 64);
    }
    uint64_t eq(uint8_t c, int w) const { return peq[(size_t)c * words + w]; }
};

void normalise(const uint8_t *&a, int &la, const uint8_t *&b, int &lb, int trim) {
    if (trim) trim_affixes(a, la, b, lb);
    if (la > lb) {
        const uint8_t *t = a; a = b; b = t;
        int x = la; la = lb; lb = x;
    }
}

}  // namespace

extern "C" int blg_host_distance(const uint8_t *a, int la, const uint8_t *b, int lb, int trim, int k) {
    normalise(a, la, b, lb, trim);
    if (k >= 0 && lb - la > k) return k + 1;
    if (la == 0) return lb;
    Pattern P(a, la);
    const int W = P.words, lastbit = (la - 1) % 64;
    std::vector<uint64_t> pv(W, ~0ull), mv(W, 0);
    int score = la;
    for (int j = 0; j < lb; j++) {
        uint64_t ph, mh;
        step_top<uint64_t>(pv[0], mv[0], P.eq(b[j], 0), ph, mh);
        int h = hdelta<uint64_t>(ph, mh, W == 1 ? lastbit : 63);
        for (int w = 1; w < W; w++) {
            step_mid<uint64_t>(pv[w], mv[w], P.eq(b[j], w), h, ph, mh);
            h = hdelta<uint64_t>(ph, mh, w == W - 1 ? lastbit : 63);
        }
        score += h;
        if (hopeless(score, j, lb, k)) return k + 1;
    }
    return cap_k(score, k);
}

extern "C" int blg_host_wavefront(const uint8_t *a, int la, const uint8_t *b, int lb, int trim, int k) {
    normalise(a, la, b, lb, trim);
    if (k >= 0 && lb - la > k) return k + 1;
    if (la == 0) return lb;
    Pattern P(a, la);
    const int W = P.words, lastw = W - 1, lastbit = (la - 1) % 64;
    std::vector<uint64_t> pv(W, ~0ull), mv(W, 0);
    std::vector<int> carry(W, 0), next(W, 0);   // carry[w]: what lane w received last step
    int score = la;
    bool done = false;
    for (int s = 0; s < lb + W - 1 && !done; s++) {
        for (int w = 0; w < W; w++) {
            const int j = s - w;
            next[w] = 0;
            if (j < 0 || j >= lb) continue;
            uint64_t ph, mh;
            step_mid<uint64_t>(pv[w], mv[w], P.eq(b[j], w), w == 0 ? 1 : carry[w], ph, mh);
            const int hout = hdelta<uint64_t>(ph, mh, w == lastw ? lastbit : 63);
            next[w] = hout;
            if (w == lastw) {
                score += hout;
                if (hopeless(score, j, lb, k)) done = true;
            }
        }
        for (int w = W - 1; w >= 1; w--) carry[w] = next[w - 1];   // shfl_up by one lane
    }
    if (done) return k + 1;
    return cap_k(score, k);
}

// The pipe-balanced form the search kernels use: 32-bit halves, IMAD-style
// add/shift/score (plain arithmetic on the host), score kept as +1/-1 counts
// of the last word's output bit, words chained top to bottom in a column.
extern "C" int blg_host_distance_halves(const uint8_t *a, int la, const uint8_t *b, int lb, int trim, int k) {
    normalise(a, la, b, lb, trim);
    if (k >= 0 && lb - la > k) return k + 1;
    if (la == 0) return lb;
    Pattern P(a, la);
    const int W = P.words, lastbit = (la - 1) % 64;
    const Units u{1u, 2u};
    const uint32_t mult = u.one << (31 - (lastbit & 31));
    std::vector<Word2> st(W);
    for (auto &x : st) { x.pl = x.ph = ~0u; x.ml = x.mh = 0; }
    uint32_t accP = 0, accM = 0;
    for (int j = 0; j < lb; j++) {
        uint32_t Phl = 0, Phh = 0, Mhl = 0, Mhh = 0, cp = u.one, cm = 0;
        for (int w = 0; w < W; w++) {
            const uint64_t e = P.eq(b[j], w);
            step_h(st[w], (uint32_t)e, (uint32_t)(e >> 32), cp, cm, u, Phl, Phh, Mhl, Mhh);
            cp = top_bit(Phh, u);
            cm = top_bit(Mhh, u);
        }
        if (lastbit >= 32) {
            accP = imad_hi(imad_lo(Phh, mult, 0), u.two, accP);
            accM = imad_hi(imad_lo(Mhh, mult, 0), u.two, accM);
        } else {
            accP = imad_hi(imad_lo(Phl, mult, 0), u.two, accP);
            accM = imad_hi(imad_lo(Mhl, mult, 0), u.two, accM);
        }
        if (hopeless(la + (int)accP - (int)accM, j, lb, k)) return k + 1;
    }
    return cap_k(la + (int)accP - (int)accM, k);
}

// The banded loop (k <= 31) with the window bits read from a full Peq table.
extern "C" int blg_host_band(const uint8_t *a, int la, const uint8_t *b, int lb, int trim, int k) {
    normalise(a, la, b, lb, trim);
    if (k < 0 || k > 31) return -1;
    if (lb - la > k) return k + 1;
    if (la == 0) return lb;
    Pattern P(a, la);
    const Units u{1u, 2u};
    auto text = [&](int j) -> uint32_t { return b[j]; };
    auto eqw = [&](uint32_t c, int p0) -> uint32_t {
        uint32_t v = 0;
        for (int q = 0; q < 32; q++) {
            const int p = p0 + q;
            if (p >= 0 && p < la && ((P.eq((uint8_t)c, p / 64) >> (p % 64)) & 1u)) v |= 1u << q;
        }
        return v;
    };
    return band_core(la, lb, k, text, eqw, u, nullptr);
}

// The banded loop as the pairs path runs it (trimmed, shorter string as
// the pattern), also reporting the text columns it processed before its exit
// fired (0 for pairs settled by the length gap or an empty pattern).
extern "C" int blg_host_band_cols(const uint8_t *a, int la, const uint8_t *b, int lb, int k, int *cols) {
    normalise(a, la, b, lb, 1);
    *cols = 0;
    if (k < 0 || k > 31) return -1;
    if (lb - la > k) return k + 1;
    if (la == 0) return lb;
    Pattern P(a, la);
    const Units u{1u, 2u};
    auto text = [&](int j) -> uint32_t { return b[j]; };
    auto eqw = [&](uint32_t c, int p0) -> uint32_t {
        uint32_t v = 0;
        for (int q = 0; q < 32; q++) {
            const int p = p0 + q;
            if (p >= 0 && p < la && ((P.eq((uint8_t)c, p / 64) >> (p % 64)) & 1u)) v |= 1u << q;
        }
        return v;
    };
    return band_core(la, lb, k, text, eqw, u, cols);
}

// The banded loop with the pairs solver's block tables: nibble rows over a
// 64-position block of the pattern (bit i <-> position 32b - dhi + i), each
// column's window taken with one funnel shift, rows shifted by 32 positions
// and the next 32 bytes entered every 32 columns (k_solve_band's scheme).
extern "C" int blg_host_band_blocks(const uint8_t *a, int la, const uint8_t *b, int lb, int k) {
    normalise(a, la, b, lb, 1);
    if (k < 0 || k > 31) return -1;
    if (lb - la > k) return k + 1;
    if (la == 0) return lb;
    const int m = la, n = lb;
    const BandGeom bg = band_geom(m, n, k);
    const int dhi = bg.dhi;
    uint32_t lo[32] = {0}, hi[32] = {0};
    auto set = [&](uint32_t c, int bitpos) {
        uint32_t *h = bitpos >= 32 ? hi : lo;
        h[c >> 4] |= 1u << (bitpos & 31);
        h[16 + (c & 15)] |= 1u << (bitpos & 31);
    };
    const int first_end = m < 64 - dhi ? m : 64 - dhi;
    for (int p = 0; p < first_end; p++) set(a[p], p + dhi);
    int next_pos = first_end;
    const Units u{1u, 2u};
    auto text = [&](int j) -> uint32_t { return b[j]; };
    auto eqw = [&](uint32_t c, int p0) -> uint32_t {
        const int j = p0 + dhi;
        if ((j & 31) == 0 && j > 0) {
            for (int r = 0; r < 32; r++) { lo[r] = hi[r]; hi[r] = 0; }
            int cnt = m - next_pos;
            if (cnt > 32) cnt = 32;
            for (int i = 0; i < cnt; i++) set(a[next_pos + i], 32 + i);
            if (cnt > 0) next_pos += cnt;
        }
        const uint32_t xl = lo[c >> 4] & lo[16 + (c & 15)], xh = hi[c >> 4] & hi[16 + (c & 15)];
        const int s = j & 31;
        return s == 0 ? xl : (xl >> s) | (xh << (32 - s));
    };
    return band_core(m, n, k, text, eqw, u, nullptr);
}

// Same, with the pattern as the LONGER string (the search kernels' case:
// the query is the pattern whatever the choice's length), no trimming.
extern "C" int blg_host_band_query(const uint8_t *q, int m, const uint8_t *t, int n, int k) {
    if (k < 0 || k > 31) return -1;
    if (m == 0) return cap_k(n, k);
    if ((n > m ? n - m : m - n) > k) return k + 1;
    Pattern P(q, m);
    const Units u{1u, 2u};
    auto text = [&](int j) -> uint32_t { return t[j]; };
    auto eqw = [&](uint32_t c, int p0) -> uint32_t {
        uint32_t v = 0;
        for (int qq = 0; qq < 32; qq++) {
            const int p = p0 + qq;
            if (p >= 0 && p < m && ((P.eq((uint8_t)c, p / 64) >> (p % 64)) & 1u)) v |= 1u << qq;
        }
        return v;
    };
    return band_core(m, n, k, text, eqw, u, nullptr);
}

// The search's banded run stopped after `stop` columns (a multiple of 4) and
// resumed from its saved state with fresh text and window readers, the
// window bits taken from the unpadded Peq words as the resume pass reads
// them (32-bit halves p0 >> 5 and the next, zero outside the pattern).
extern "C" int blg_host_band_resume(const uint8_t *q, int m, const uint8_t *t, int n, int k, int stop) {
    if (k < 0 || k > 31 || stop < 0 || (stop & 3)) return -1;
    if (m == 0) return cap_k(n, k);
    if ((n > m ? n - m : m - n) > k) return k + 1;
    Pattern P(q, m);
    const int nw = (m + 63) / 64;
    auto half = [&](uint32_t c, int r) -> uint32_t {
        if (r < 0 || r >= 2 * nw) return 0u;
        const uint64_t w = P.eq((uint8_t)c, r >> 1);
        return (r & 1) ? (uint32_t)(w >> 32) : (uint32_t)w;
    };
    auto eqw = [&](uint32_t c, int p0) -> uint32_t {
        const int r = p0 >> 5, s = p0 & 31;
        const uint32_t lo = half(c, r), hi = half(c, r + 1);
        return s == 0 ? lo : (lo >> s) | (hi << (32 - s));
    };
    const BandGeom bg = band_geom(m, n, k);
    BandState s = band_start(bg);
    auto text1 = [&](int j) -> uint32_t { return t[j]; };
    if (band_steps(k, bg, s, stop < n ? stop : n, text1, eqw)) return k + 1;
    const BandState saved = s;                          // what the queue item carries
    BandState r = saved;
    const uint8_t *rest = t + saved.j;
    auto text2 = [&](int j) -> uint32_t { return rest[j - saved.j]; };
    if (band_steps(k, bg, r, n, text2, eqw)) return k + 1;
    return band_finish(k, bg, r);
}

extern "C" int blg_host_store(int d, int dtype) {
    if (dtype == DT_UINT8) return (int)saturate_u8(d);
    if (dtype == DT_UINT16) return (int)saturate_u16(d);
    return d;
}

// The bit-sliced search of up to 32 queries (packed: bytes and offsets) against
// one text, as k_search_bits runs it: stripes of 64 rows with the deltas
// between them kept per column, counts of the last column's vertical deltas
// in planes, transposed to bytes. out: one distance per query.
extern "C" void blg_host_bits(const uint8_t *buf, const int64_t *off, int nq, const uint8_t *t, int n, int32_t *out) {
    int longest = 0;
    for (int q = 0; q < nq; q++) longest = longest < off[q + 1] - off[q] ? (int)(off[q + 1] - off[q]) : longest;
    const int stripes = longest > 0 ? (longest + 63) / 64 : 1;
    std::vector<uint32_t> hp((size_t)n, ~0u), hm((size_t)n, 0);
    const BitUnits u{1u, ~0u};
    uint32_t acc[kBitPlanes] = {0};
    for (int s = 0; s < stripes; s++) {
        const int rows = s == stripes - 1 ? ((longest - 64 * s + 7) / 8 * 8 > 8 ? (longest - 64 * s + 7) / 8 * 8 : 8) : 64;
        uint32_t vn[64], vm[64], valid[64] = {0};
        for (int i = 0; i < 64; i++) {
            vn[i] = 0;
            vm[i] = 0;
            for (int q = 0; q < nq; q++)
                if (64 * s + i < off[q + 1] - off[q]) valid[i] |= 1u << q;
        }
        for (int j = 0; j < n; j++) {
            for (int i = 0; i < rows; i++) {
                uint32_t eq = 0;
                for (int q = 0; q < nq; q++)
                    if ((valid[i] >> q & 1u) && buf[off[q] + 64 * s + i] == t[j]) eq |= 1u << q;
                if (i & 1) bit_cell<true>(eq, vn[i], vm[i], hp[j], hm[j], u);
                else bit_cell<false>(eq, vn[i], vm[i], hp[j], hm[j], u);
            }
        }
        uint32_t pl[8] = {0};
        for (int i = 0; i < rows; i += 4) {
            uint32_t x[8];
            for (int b = 0; b < 4; b++) {
                x[b] = ~vn[i + b] & valid[i + b];
                x[4 + b] = ~vm[i + b] & valid[i + b];
            }
            bit_count8(pl, x);
        }
        uint32_t carry = 0, c2;
        for (int p = 0; p < kBitPlanes; p++) {
            bit_full_add(acc[p], c2, p < 8 ? pl[p] : 0u, carry);
            carry = c2;
        }
    }
    uint32_t lo[8], hi[8];
    for (int p = 0; p < 8; p++) {
        lo[p] = acc[p];
        hi[p] = p + 8 < kBitPlanes ? acc[p + 8] : 0u;
    }
    bit_transpose8(lo);
    bit_transpose8(hi);
    for (int q = 0; q < nq; q++) {
        const int cnt = (int)((lo[q & 7] >> (q & 24) & 0xffu) | (hi[q & 7] >> (q & 24) & 0xffu) << 8);
        out[q] = n - (int)(off[q + 1] - off[q]) + cnt;
    }
}

// Signatures of two strings and the product of their e4m3 rows: the sum whose
// sign k_filter_pairs reads (valid: bit 0 the query's row, bit 1 the choice's;
// bit 2: half the bins); *diff receives |X ^ Y|.
extern "C" float blg_host_sig_sum(const uint8_t *x, int m, const uint8_t *y, int n, int k, int valid, int *diff) {
    auto value = [](uint32_t b) {
        const int e = (int)(b >> 3 & 15u), f = (int)(b & 7u);
        float v = e ? 1.0f + (float)f / 8.0f : (float)f / 8.0f;
        for (int i = e ? e : 1; i > 7; i--) v *= 2.0f;
        for (int i = e ? e : 1; i < 7; i++) v *= 0.5f;
        return b & 0x80u ? -v : v;
    };
    uint32_t s[2][kSigWords] = {{0}, {0}};
    const uint8_t *p[2] = {x, y};
    const int len[2] = {m, n};
    int bits[2] = {0, 0};
    const int words = valid & 4 ? 32 : 64;
    for (int t = 0; t < 2; t++) {
        for (int i = 0; i + 3 < len[t]; i++) {
            const uint32_t b = sig_bit((uint32_t)p[t][i] << 24 | (uint32_t)p[t][i + 1] << 16 | (uint32_t)p[t][i + 2] << 8 | p[t][i + 3]);
            if (valid >> t & 1) s[t][b >> 5] |= 1u << (b & 31);
        }
        if (valid & 4) sig_fold(s[t]);
        for (int w = 0; w < words / 8; w++) bits[t] += popc32(s[t][w]);
    }
    *diff = 0;
    for (int w = 0; w < words / 8; w++) *diff += popc32(s[0][w] ^ s[1][w]);
    uint32_t ql, qh, cl, ch;
    sig_query_tail(bits[0], valid & 1, ql, qh);
    sig_choice_tail(bits[1], k, valid & 2, cl, ch);
    float sum = 0.0f;
    for (int w = 0; w < words; w++) {
        const uint32_t a = w == words - 2 ? ql : w == words - 1 ? qh : sig_query_word(s[0], w >> 3, w & 7);
        const uint32_t b = w == words - 2 ? cl : w == words - 1 ? ch : sig_choice_word(s[1], w >> 3, w & 7);
        for (int i = 0; i < 32; i += 8) sum += value(a >> i & 0xffu) * value(b >> i & 0xffu);
    }
    return sum;
}

// band64_core with its match bits from the pattern itself.
extern "C" int blg_host_band64(const uint8_t *a, int m, const uint8_t *b, int n, int k) {
    return band64_core(m, n, k, [&](int j, int p0, uint64_t (&e)[4]) {
        for (int x = 0; x < 4; x++) {
            e[x] = 0;
            for (int i = 0; i < 64; i++) {
                const int p = p0 + x + i;
                if (j + x < n && p >= 0 && p < m && a[p] == b[j + x]) e[x] |= 1ull << i;
            }
        }
    });
}
