// Exact cdist, bit-sliced over queries (blg_bits.cuh).
//
// The reference gives one thread a (query, choice) pair and one 64-bit word
// per 64 query characters (csrc/gpu_kernels.cu:34-69). Here a machine word
// holds one cell of 32 queries' matrices and a lane holds one choice, so a
// warp advances 32 x 32 pairs together.
//
//  * A group of 32 queries of similar length (the search's queries sorted by
//    length) has a table in shared memory: for every symbol the queries use and
//    every row, the queries with that symbol at that row. A lane's text
//    character picks the symbol's rows and the column walks down them with
//    16-byte loads at constant offsets. Symbols lie `stride` words apart, 4 mod
//    32, so eight different symbols at one row hit different banks.
//  * The vertical deltas of 64 rows stay in registers (128 of them; 231 per
//    thread, 8 warps per SM). Longer queries run stripe by stripe: the
//    horizontal deltas leaving a stripe's bottom row, two words per column,
//    pass through a per-warp scratch row in global memory that L2 holds.
//  * The last stripe has as many rows as the group's longest query needs (a
//    multiple of 8), the loop over columns ends at each lane's own choice
//    length, and a tile's choices are taken in order of length, so lanes of a
//    warp end together.
//  * The distances are n + the sum of the last column's vertical deltas over a
//    query's rows, counted bit-sliced and transposed to bytes at the end.
//
// Bound: the ALU pipe (half a warp per clock and scheduler), 76% busy with the
// FMA pipe at 56%; two warps per scheduler leave the rest to dependent
// latency, and three (168 registers) spill. A cell takes four LOP3, three
// multiply-adds and a quarter of an LDS.128. Measured, 4096 x 65536 reads of
// 64 bases, int32: 9.2 ms; five LOP3 and no multiply-adds 9.7; the expressions
// left to the compiler 11.6; 12 warps of 168 registers 10.2; the prefix-reuse
// word kernel (k_search_pfx) 14.8. 401 x 50021 reads of 16 to 256 bases,
// uint16: 4.1 ms against 13.4 of the word kernels.
#include <algorithm>

#include "blg_bits.cuh"
#include "blg_kernels.cuh"
#include "blg_search_bits.h"

namespace blg {

constexpr int kBitsThreads = 256;                // 8 warps x 255 registers fill the register file
constexpr int kBitsRows = 64;                    // rows of a stripe

struct BitGroup {                                // a query of the group
    int64_t row;                                 // first output element of its row; -1: no such query
    int32_t m, pad;
};

// R rows of one stripe over a lane's whole text. tab: the stripe's first row of
// symbol 0; voff: byte offset of the rows of valid queries. h_in / h_out: the
// stripe above / below exists, its deltas in scr (this lane's column 0, two
// rows of 32 words per column). Adds the stripe's part of the counts of
// (vertical delta + 1) to pl.
template <int R>
__device__ __forceinline__ void bit_stripe(const char *tab, uint32_t voff, const uint32_t *s_map, const uint32_t *tw,
                                           int n, uint32_t *scr, bool h_in, bool h_out, BitUnits u,
                                           uint32_t (&pl)[8]) {
    uint32_t vn[R], vm[R];                        // ~(+1), -1 of each row's vertical delta
#pragma unroll
    for (int i = 0; i < R; i++) { vn[i] = 0; vm[i] = 0; }
    uint32_t w4 = __ldg(tw), next = __ldg(tw + kTileCands);
    const uint32_t *tp = tw + 2 * kTileCands;
    uint32_t off = s_map[w4 & 0xffu];
    uint32_t hpn = ~0u, hmn = 0;
    if (h_in && n > 0) {
        hpn = scr[0];
        hmn = scr[32];
    }
#pragma unroll 1
    for (int j = 0; j < n; j++) {
        const uint4 *row = reinterpret_cast<const uint4 *>(tab + off);
        // the next column's symbol and incoming deltas, while this one runs
        w4 >>= 8;
        if ((j & 3) == 3) {
            w4 = next;
            next = __ldg(tp);                    // up to two words past the text: spare rows follow the tiles
            tp += kTileCands;
        }
        off = s_map[w4 & 0xffu];
        uint32_t hp = hpn, hm = hmn;
        uint32_t *h = scr + (size_t)j * 64;
        if (h_in && j + 1 < n) {
            hpn = h[64];
            hmn = h[96];
        }
#pragma unroll
        for (int i = 0; i < R; i += 4) {
            const uint4 e = row[i / 4];
            bit_cell<true>(e.x, vn[i], vm[i], hp, hm, u);
            bit_cell<true>(e.y, vn[i + 1], vm[i + 1], hp, hm, u);
            bit_cell<true>(e.z, vn[i + 2], vm[i + 2], hp, hm, u);
            bit_cell<true>(e.w, vn[i + 3], vm[i + 3], hp, hm, u);
        }
        if (h_out) {
            h[0] = hp;
            h[32] = hm;
        }
    }
#pragma unroll
    for (int p = 0; p < 8; p++) pl[p] = 0;
    const uint4 *val = reinterpret_cast<const uint4 *>(tab + voff);
#pragma unroll
    for (int i = 0; i < R; i += 4) {
        const uint4 e = val[i / 4];
        const uint32_t x[8] = {~vn[i] & e.x, ~vn[i + 1] & e.y, ~vn[i + 2] & e.z, ~vn[i + 3] & e.w,
                               ~vm[i] & e.x, ~vm[i + 1] & e.y, ~vm[i + 2] & e.z, ~vm[i + 3] & e.w};
        bit_count8(pl, x);                       // at most 2 x 64: eight planes
    }
}

// The stripe with the fewest rows that holds `rows` (1..64).
__device__ __forceinline__ void bit_stripe_rows(int rows, const char *tab, uint32_t voff, const uint32_t *s_map,
                                                const uint32_t *tw, int n, uint32_t *scr, bool h_in, bool h_out,
                                                BitUnits u, uint32_t (&pl)[8]) {
    switch ((rows + 7) >> 3) {
    case 0:
    case 1: bit_stripe<8>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    case 2: bit_stripe<16>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    case 3: bit_stripe<24>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    case 4: bit_stripe<32>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    case 5: bit_stripe<40>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    case 6: bit_stripe<48>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    case 7: bit_stripe<56>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    default: bit_stripe<64>(tab, voff, s_map, tw, n, scr, h_in, h_out, u, pl); break;
    }
}

// The work is the line of (group, 32 choices) units, group after group, the
// longest queries first and a tile's longest choices first; a unit weighs
// what its group's rows do. CTA b takes the b-th part of equal weight, so it
// builds one table or two and its warps pull units of one group from a
// shared counter with nothing to wait for until the group changes. A launch
// with no more units than warps gives every CTA units of one group only: a
// second group would be a second round (96 x 3500 reads of 64: 62 us, 36).
__global__ void __launch_bounds__(kBitsThreads, 1) k_search_bits(BitSearch B, int dtype, void *out, uint32_t one,
                                                                 uint32_t *status) {
    extern __shared__ __align__(16) uint32_t s_tab[];          // [nsym + 2][stride]
    __shared__ uint32_t s_map[256];
    __shared__ BitGroup s_grp[32];
    __shared__ int s_next;
    const BitUnits u{one, 0u - one};
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int stride = B.stride;
    if (tid < 256) s_map[tid] = (uint32_t)B.map[tid] * (uint32_t)stride * 4u;
    const uint32_t voff = (uint32_t)(B.nsym + 1) * (uint32_t)stride * 4u;
    const int64_t nc = B.T.n;
    const int units = (int)((nc + 31) / 32);                   // of a group
    uint32_t *scr = B.scratch
                        ? B.scratch + ((int64_t)blockIdx.x * (kBitsThreads / 32) + warp) * B.scratch_words + lane
                        : nullptr;
    // this CTA's part: units [u0, u1) counted from the first unit of group g0
    auto place = [&](int64_t w, int &g, int &unit) {           // the first unit at or past weight w
        g = upper_index(B.weight, B.groups, w);
        const int64_t per = (B.weight[g + 1] - B.weight[g]) / units;
        unit = (int)((w - B.weight[g] + per - 1) / per);
    };
    int g0, t0, g1, t1;
    if (B.per > 0) {
        const int parts = (units + B.per - 1) / B.per;         // of a group
        g0 = g1 = blockIdx.x / parts;
        t0 = (blockIdx.x - g0 * parts) * B.per;
        t1 = min(units, t0 + B.per);
    } else {
        const int64_t total = B.weight[B.groups];
        place(total * blockIdx.x / gridDim.x, g0, t0);
        place(total * (blockIdx.x + 1) / gridDim.x, g1, t1);
        if (blockIdx.x + 1 == gridDim.x) {
            g1 = B.groups - 1;
            t1 = units;
        }
    }
    for (int gi = g0; gi <= g1; gi++) {
        const int first = gi == g0 ? t0 : 0, end = gi == g1 ? t1 : units;
        if (first >= end) continue;                            // uniform
        const int g = B.groups - 1 - gi;                       // longest first
        __syncthreads();                                       // every warp is done with the previous group
        const int q1 = min(B.nq, g * 32 + 32);
        const int longest = B.qlen[q1 - 1];                    // sorted by length
        const int stripes = max(1, (longest + kBitsRows - 1) / kBitsRows);
        const int last_rows = longest - (stripes - 1) * kBitsRows;
        const int words = (B.nsym + 2) * stride;
        for (int x = tid; x < words; x += kBitsThreads) s_tab[x] = 0;
        if (tid < 32) {
            const int q = g * 32 + tid;
            s_grp[tid] = q < B.nq ? BitGroup{(int64_t)B.qidx[q] * nc, B.qlen[q], 0} : BitGroup{-1, 0, 0};
        }
        if (tid == 0) s_next = first;
        __syncthreads();
        for (int q = warp; q < q1 - g * 32; q += kBitsThreads / 32) {
            int m;
            const uint8_t *p = string_at(B.Q, B.qidx[g * 32 + q], m, status);
            m = min(m, longest);
            for (int i = lane; i < m; i += 32) {
                atomicOr(&s_tab[B.map[p[i]] * stride + i], 1u << q);
                atomicOr(&s_tab[(B.nsym + 1) * stride + i], 1u << q);
            }
        }
        __syncthreads();
        while (true) {
            int t = 0;
            if (lane == 0) t = atomicAdd(&s_next, 1);
            t = __shfl_sync(kFull, t, 0);
            if (t >= end) break;
            const int64_t tile = t / (kTileCands / 32);
            const bool valid = (int64_t)t * 32 + lane < nc;
            const int pos = valid ? B.order[(int64_t)t * 32 + lane] : 0;
            const int64_t c = tile * kTileCands + pos;
            const int n = valid ? __ldg(B.T.len + c) : 0;
            const uint32_t *tw = B.T.words + B.T.base[tile] + pos;
            uint32_t pl[8], hi[8];
#pragma unroll
            for (int p = 0; p < 8; p++) hi[p] = 0;
#pragma unroll 1
            for (int s = 0; s < stripes; s++) {
                const bool last = s == stripes - 1;
                bit_stripe_rows(last ? last_rows : kBitsRows,
                                reinterpret_cast<const char *>(s_tab) + (size_t)s * kBitsRows * 4, voff, s_map, tw, n,
                                scr, s > 0, !last, u, pl);
                if (stripes > 1) {                             // counts so far: bit-sliced, after the columns' deltas
                    uint32_t *acc = scr + B.scratch_words - kBitPlanes * 32;
                    uint32_t carry = 0;
#pragma unroll
                    for (int p = 0; p < kBitPlanes; p++) {
                        uint32_t v = s > 0 ? acc[p * 32] : 0u, c2;
                        bit_full_add(v, c2, p < 8 ? pl[p < 8 ? p : 0] : 0u, carry);
                        carry = c2;
                        if (!last) acc[p * 32] = v;
                        else if (p < 8) pl[p < 8 ? p : 0] = v;
                        else hi[p < 8 ? 0 : p - 8] = v;
                    }
                }
            }
            bit_transpose8(pl);
            if (stripes > 1) bit_transpose8(hi);
            if (valid) {
#pragma unroll
                for (int r = 0; r < 8; r++)
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        const BitGroup q = s_grp[8 * b + r];
                        if (q.row < 0) continue;               // uniform
                        const int cntv = (int)(((pl[r] >> (8 * b)) & 0xffu) | (((hi[r] >> (8 * b)) & 0xffu) << 8));
                        store1(out, dtype, q.row + c, n - q.m + cntv);
                    }
            }
        }
    }
}

// ------------------------------------------------------------- launcher --
int bits_stride(int64_t longest) {                 // words between symbols: at least the rows, 4 mod 32
    const int64_t rows = std::max<int64_t>(8, (longest + 7) & ~int64_t(7));
    return (int)((rows + 27) / 32 * 32 + 4);
}

size_t bits_table_bytes(int nsym, int64_t longest) { return (size_t)(nsym + 2) * bits_stride(longest) * 4; }

int bits_warps(int sms) { return sms * (kBitsThreads / 32); }

int64_t bits_scratch_words(int64_t longest_choice) { return (2 * longest_choice + kBitPlanes) * 32; }

// What a unit of a group of queries up to `longest` weighs: its rows, and the
// columns' own overhead as a few more.
int64_t bits_unit_weight(int64_t longest) {
    const int64_t stripes = std::max<int64_t>(1, (longest + kBitsRows - 1) / kBitsRows);
    return std::max<int64_t>(8, (longest + 7) & ~int64_t(7)) + 4 * stripes;
}

cudaError_t launch_search_bits(cudaStream_t st, int sms, BitSearch B, int64_t longest, int dtype, void *out,
                               uint32_t *status) {
    if (B.nq <= 0 || B.T.n <= 0) return cudaSuccess;
    B.stride = bits_stride(longest);
    const int64_t units = (B.T.n + 31) / 32;                   // of a group
    int64_t grid = std::min<int64_t>(units * B.groups, sms);
    B.per = 0;
    if (units * B.groups <= (int64_t)sms * (kBitsThreads / 32)) {
        int64_t per = (units * B.groups + sms - 1) / sms;
        while (per < units && B.groups * ((units + per - 1) / per) > sms) per++;
        if (B.groups * ((units + per - 1) / per) <= sms) {
            B.per = (int)per;
            grid = B.groups * ((units + per - 1) / per);
        }
    }
    const size_t smem = bits_table_bytes(B.nsym, longest);
    cudaError_t e = cudaFuncSetAttribute(k_search_bits, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_search_bits<<<(unsigned)grid, kBitsThreads, smem, st>>>(B, dtype, out, 1u, status);
    return cudaGetLastError();
}

}  // namespace blg
