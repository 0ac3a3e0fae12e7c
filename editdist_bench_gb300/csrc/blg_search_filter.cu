// Thresholded search, dense in length: the 4-gram filter on the tensor cores.
//
// A thresholded search first has to find, among all (query, choice) pairs of
// compatible length, the few whose 4-grams allow a distance within max_dist (the
// reference runs its column loop on every pair, csrc/gpu_kernels.cu:34-69).
// k_search_band tests pair by pair, 16 byte counters against 16: about
// 0.6 SM clocks a pair. Here the test is a matrix product of signatures
// (blg_sig.cuh): a tile of 128 queries x 256 choices is four or eight
// tcgen05.mma of 128 x 256 x 32 (128 clocks each) and takes about 1750 clocks,
// 0.05 a pair; the warps that read and write its operands bind (1470 and
// 1300 clocks of work a tile), not the products. Measured: k = 2 on 4096 x 65536
// reads of 64, uint8: 72 us a search against 498 of the per-pair filter; k =
// 4 on 1024 x 2^20 reads of 100 to 256 (1 GiB of output, 140 us of writing):
// 207 against 345.
//
// One CTA per SM walks its share of the tiles; its warps have roles and meet
// on mbarriers:
//   warp 0        issues the products (one lane); the accumulators, 2 x 256
//                 columns, fill TMEM, so a tile is computed while the one
//                 before is read
//   warp 1        writes the output's k + 1: bulk copies of a constant from
//                 shared memory, which cost the other warps nothing, so the
//                 HBM-bound fill of the matrix runs under the filter
//   warps 4..11   read the accumulators (32 rows x 128 columns each) and AND the
//                 signs of 32 columns at a time; pairs with a sum >= 0 go to
//                 the list
//   warps 12..19  spread signatures (32 bytes a string) into e4m3 rows in shared
//                 memory, a choice per thread, 80 operations a row; the
//                 queries' rows when the query tile changes
// The operands never exist in HBM: 32 bytes per string are read, not 256.
// Rows are in core matrices (8 rows x 16 bytes contiguous, no swizzle), chunk
// by chunk of 16 bytes, so a warp's stores are 512 contiguous bytes.
//
// k_solve_passers then runs the listed pairs, a lane each: the 16-bin count
// bound (stronger on long strings, where most bins are taken), then their
// distance by furthest-reaching points. A list that ran full leaves the whole
// search to the repair launch of k_search_band.
#include <algorithm>

#include "blg_kernels.cuh"
#include "blg_reach.cuh"
#include "blg_search_filter.h"
#include "blg_sig.cuh"
#include "blg_tma.cuh"

namespace blg {

constexpr int kFltThreads = 640;
constexpr int kFltReaders = 8;                           // reading warps: 4 .. 11; producing: 12 .. 19
constexpr int kFltM = 128, kFltN = 256;                  // tile: queries x choices
constexpr int kFltHits = 16;                             // chunks with a passer that a reading warp keeps back
constexpr int kFillPiece = 4096;                         // bytes of one bulk copy of the fill constant
constexpr int64_t kFillItem = 65536;                     // bytes claimed at a time

// K: bytes of a row, 256, or 128 with the signature folded in two (sig_fold).
template <int K>
struct __align__(128) FilterShared {
    uint8_t a[kFltM * K];
    uint8_t b[2][kFltN * K];
    uint8_t pattern[kFillPiece];
    uint32_t hit[kFltReaders][kFltHits][32];             // per row: the chunk's columns that pass
    uint2 hit_at[kFltReaders][kFltHits];                 // first row's query, first column's choice
    int64_t start[kFltMaxTiles + 1];                     // first tile of each query tile
    int32_t lo[kFltMaxTiles], hi[kFltMaxTiles];          // its choice range
    uint64_t full[2], empty[2], tfull[2], tempty[2];
    uint32_t tmem;
    int abort;
    int done;                                            // reading warps that have read their last tile
};

// ---- tcgen05 in inline PTX
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t k_stride, uint32_t mn_stride) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)(k_stride >> 4) << 16) | ((uint64_t)(mn_stride >> 4) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ void umma_e4m3(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// 32 columns of the warp's 32 rows: the load, and the wait for it (which names
// the registers, so that nothing reads them before).
__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                   "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]),
                   "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]),
                   "+r"(v[30]), "+r"(v[31])::"memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// A role's wait: bounded; one that gives up raises the status bit and the
// CTA's abort flag, on which every role leaves its loop. A lane's own verdict:
// for the lane that issues the products alone.
__device__ __forceinline__ bool role_wait(int *abort, uint64_t *bar, uint32_t parity, uint32_t polls, uint32_t *status) {
    for (uint32_t i = 0; i < polls; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*(volatile int *)abort) return false;
    }
    atomicOr(status, ST_QUEUE_TIMEOUT);
    *(volatile int *)abort = 1;
    return false;
}

// The wait of a whole warp, one verdict for all lanes: near the bound, or with
// the flag just raised, lanes see different things, and what follows in the
// reading and producing warps (TMEM loads, votes, shuffles) needs all of them.
// Every poll is voted on, so the lanes never part (1024 x 2^20 reads at max_dist 4
// 205.5 us; 206.9 with a vote after lanes that poll by themselves).
__device__ __forceinline__ bool warp_wait(int *abort, uint64_t *bar, uint32_t parity, uint32_t polls, uint32_t *status) {
    for (uint32_t i = 0; i < polls; i++) {
        if (__all_sync(kFull, mbar_try_wait(bar, parity))) return true;
        if (__any_sync(kFull, *(volatile int *)abort)) return false;
    }
    *(volatile int *)abort = 1;
    atomicOr(status, ST_QUEUE_TIMEOUT);
    return false;
}

// The output's k + 1, in items of kFillItem bytes from its first 16-byte
// boundary, claimed one by one (F.ctr) by the fill warps of the filter and of the
// solver. Claimed and not divided up beforehand: the SMs do not write at one
// speed, and 1 GiB takes 164 us in equal shares, 140 claimed (as a grid of one
// block per piece, or cudaMemset). Called by a whole warp; lane 0 copies the
// constant in `pattern` (kFillPiece bytes of shared memory) with bulk copies.
// stop(): leave the rest to others.
template <typename StopFn>
__device__ __forceinline__ void fill_items(const BatchFill &fill, unsigned long long *ctr, const uint8_t *pattern,
                                           bool ends, StopFn stop) {
    const int es = elem_bytes(fill.dtype), lane = threadIdx.x & 31;
    const int64_t bytes = fill.n * es;
    if (bytes <= 0) return;
    uint8_t *o = reinterpret_cast<uint8_t *>(fill.out);
    const int64_t head = min(bytes, (int64_t)((16 - (reinterpret_cast<uintptr_t>(o) & 15)) & 15));
    const int64_t body = (bytes - head) & ~int64_t(15), items = (body + kFillItem - 1) / kFillItem;
    if (ends) {                                          // element by element, at most 15 bytes each
        for (int64_t e = lane; e < head / es; e += 32) store1(fill.out, fill.dtype, e, (int)fill.value);
        for (int64_t e = (head + body) / es + lane; e < fill.n; e += 32) store1(fill.out, fill.dtype, e, (int)fill.value);
    }
    if (lane == 0) {
        uint64_t policy;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
        const uint32_t src = smem_addr(pattern);
        while (!stop()) {
            const int64_t it = (int64_t)atomicAdd(ctr, 1ull);
            if (it >= items) break;
            const int64_t b1 = min(body, (it + 1) * kFillItem);
            for (int64_t b = it * kFillItem; b < b1; b += kFillPiece) {
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(
                                 o + head + b),
                             "r"(src), "r"((uint32_t)min((int64_t)kFillPiece, b1 - b)), "l"(policy)
                             : "memory");
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory");
        }
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
}

__device__ __forceinline__ void fill_pattern(uint8_t *pattern, const BatchFill &fill) {
    const uint32_t v = fill.dtype == DT_UINT8 ? fill.value * 0x01010101u
                       : fill.dtype == DT_UINT16 ? fill.value * 0x00010001u : fill.value;
    for (int x = threadIdx.x; x < kFillPiece / 4; x += blockDim.x) reinterpret_cast<uint32_t *>(pattern)[x] = v;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// The class and place in it of the i-th sequential query by length.
__device__ __forceinline__ int seq_query(const SurvClasses &C, int i, int &at) {
    int c = 0;
    while (c + 1 < C.n && i >= C.cls[c].nq) i -= C.cls[c++].nq;
    at = i;
    return c;
}

// One row of 64 words (row r of `rows`), chunk j of 4 words at j * rows * 16.
template <int ROWS, int K, typename WordFn>
__device__ __forceinline__ void write_row(uint8_t *dst, int r, int j0, int j1, WordFn word) {
#pragma unroll
    for (int j = 0; j < K / 16; j++)
        if (j >= j0 && j < j1)
            *reinterpret_cast<uint4 *>(dst + (size_t)j * (ROWS * 16) + r * 16) =
                make_uint4(word(4 * j), word(4 * j + 1), word(4 * j + 2), word(4 * j + 3));
}

// whole_fill: the fill ends here; else it stops with the CTA's last tile and
// the solver goes on with it.
template <int K>
__global__ void __launch_bounds__(kFltThreads, 1)
    k_filter_pairs(SurvClasses C, int nq, const uint32_t *qsig, const uint32_t *csig, const int64_t *lstart,
                   int64_t min_len, int64_t n_len, int k, PasserList L, BatchFill fill, bool whole_fill, uint32_t polls,
                   uint32_t *status) {
    extern __shared__ __align__(128) uint8_t s_raw[];
    FilterShared<K> &S = *reinterpret_cast<FilterShared<K> *>(s_raw);
    constexpr int W = K / 4;                             // words of a row, the last two for the tail
    __shared__ __align__(16) unsigned char s_cls_raw[sizeof(SurvClasses)];
    SurvClasses &SC = *reinterpret_cast<SurvClasses *>(s_cls_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int qtiles = (nq + kFltM - 1) / kFltM;
    if (tid == 0) {
        SC = C;
        for (int i = 0; i < 2; i++) {
            mbar_init(&S.full[i], 8);                    // the producing warps
            mbar_init(&S.empty[i], 1);                   // a commit
            mbar_init(&S.tfull[i], 1);                   // a commit
            mbar_init(&S.tempty[i], kFltReaders);                  // the reading warps
        }
        S.abort = 0;
        S.done = 0;
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&S.tmem)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fill_pattern(S.pattern, fill);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // the fill starts at once; the others plan first and meet without it
    if (warp == 1)
        fill_items(fill, L.count + 1, S.pattern, blockIdx.x == 0,
                   [&] { return !whole_fill && *(volatile int *)&S.done >= kFltReaders; });
    auto sync_rest = [] { asm volatile("bar.sync 1, %0;" ::"n"(kFltThreads - 32) : "memory"); };
    int issued = 0;
    if (warp != 1) {
    // every query tile's choice range: lengths within k of its shortest and longest query
    for (int t = tid; t < qtiles; t += kFltThreads) {
        int at;
        const int c0 = seq_query(SC, t * kFltM, at);
        const int64_t m0 = SC.cls[c0].qlen[at];
        const int c1 = seq_query(SC, min(nq, t * kFltM + kFltM) - 1, at);
        const int64_t m1 = SC.cls[c1].qlen[at];
        int64_t x = m0 - k - min_len, y = m1 + k - min_len + 1;
        x = x < 0 ? 0 : (x > n_len ? n_len : x);
        y = y < x ? x : (y > n_len ? n_len : y);
        S.lo[t] = (int32_t)lstart[x];
        S.hi[t] = (int32_t)lstart[y];
    }
    sync_rest();
    if (warp == 2) {                                     // prefix of the tile counts
        int64_t run = 0;
        for (int t0 = 0; t0 < qtiles; t0 += 32) {
            const int t = t0 + lane;
            const int64_t n = t < qtiles ? (S.hi[t] - S.lo[t] + kFltN - 1) / kFltN : 0;
            int64_t incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t v = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += v;
            }
            if (t < qtiles) S.start[t] = run + incl - n;
            run += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0) S.start[qtiles] = run;
    }
    sync_rest();
    const int64_t total = S.start[qtiles];
    const int64_t i0 = total * blockIdx.x / gridDim.x, i1 = total * (blockIdx.x + 1) / gridDim.x;
    const int ntiles = (int)(i1 - i0);
    int qt = ntiles > 0 ? upper_index(S.start, qtiles, i0) : 0;   // (an empty query tile shares its start: the last one wins)
    auto advance = [&](int i) {                          // the query tile of this CTA's i-th tile
        while (i0 + i >= S.start[qt + 1]) qt++;
    };

    if (warp == 0) {
        if (lane == 0) {
            // D f32 | A, B e4m3, both K-major | N | M
            const uint32_t idesc = (1u << 4) | ((kFltN / 8) << 17) | ((kFltM / 16) << 24);
            for (int i = 0; i < ntiles; i++) {
                const int buf = i & 1;
                const uint32_t par = (uint32_t)(i >> 1) & 1u;
                if (!role_wait(&S.abort, &S.full[buf], par, polls, status)) break;
                if (!role_wait(&S.abort, &S.tempty[buf], par ^ 1u, polls, status)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = smem_addr(S.a), b = smem_addr(S.b[buf]);
#pragma unroll
                for (int kk = 0; kk < K / 32; kk++)
                    umma_e4m3(S.tmem + buf * kFltN, umma_desc(a + kk * 2 * kFltM * 16, kFltM * 16, 128),
                              umma_desc(b + kk * 2 * kFltN * 16, kFltN * 16, 128), idesc, kk > 0);
                umma_commit(&S.empty[buf]);
                umma_commit(&S.tfull[buf]);
                issued = i + 1;
            }
        }
        __syncwarp();
    } else if (warp >= 4 && warp < 4 + kFltReaders) {
        const int w = warp - 4, rows = (w & 3) * 32, half = (w >> 2) * (kFltN / 2);   // (TMEM rows go by warp mod 4)
        int held = 0;                                    // hit chunks kept back (uniform)
        auto flush = [&]() {                             // every lane; the kept chunks' passers to the list
            __syncwarp();
            int n = 0;
            for (int x = 0; x < held; x++) n += __popc(S.hit[w][x][lane]);
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            unsigned long long at = 0;
            if (lane == 31) at = atomicAdd(L.count, (unsigned long long)incl);
            at = __shfl_sync(kFull, at, 31) + (unsigned long long)(incl - n);
            for (int x = 0; x < held; x++) {
                const uint2 h = S.hit_at[w][x];
                for (uint32_t m = S.hit[w][x][lane]; m; m &= m - 1, at++)
                    if (at < L.cap) L.item[at] = (unsigned long long)(h.x + lane) << 32 | (h.y + (uint32_t)(__ffs(m) - 1));
            }
            held = 0;
            __syncwarp();
        };
        // the signs of 32 columns of the rows from query q on, columns from choice c
        // on. A chunk with a pair that passes (a sum >= 0) leaves its columns as a
        // mask per row, 32 shifts for the warp; the masks become list entries
        // sixteen chunks at a time, one scan and one atomic for all. The slowest
        // reading warp holds up the tile: entries made on the spot took 0.9 us a tile
        // with nine passers, 0.45 with none, a walk of the passing lanes alone 2.2.
        auto take = [&](const uint32_t (&v)[32], uint32_t q, uint32_t c) {
            uint32_t a[11];
#pragma unroll
            for (int x = 0; x < 10; x++) a[x] = v[3 * x] & v[3 * x + 1] & v[3 * x + 2];
            a[10] = v[30] & v[31];
            const uint32_t neg = (a[0] & a[1] & a[2]) & (a[3] & a[4] & a[5]) & (a[6] & a[7] & a[8]) & (a[9] & a[10]);
            if (!__any_sync(kFull, (int32_t)neg >= 0)) return;
            uint32_t b[4] = {0, 0, 0, 0};                // sign bits, column x at bit x: four chains of eight shifts
#pragma unroll
            for (int x = 7; x >= 0; x--)
#pragma unroll
                for (int y = 0; y < 4; y++) b[y] = __funnelshift_l(v[8 * y + x], b[y], 1);
            S.hit[w][held][lane] = ~(b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24));
            if (lane == 0) S.hit_at[w][held] = make_uint2(q, c);
            if (++held == kFltHits) flush();
        };
        for (int i = 0; i < ntiles; i++) {
            const int buf = i & 1;
            advance(i);
            if (!warp_wait(&S.abort, &S.tfull[buf], (uint32_t)(i >> 1) & 1u, polls, status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t q = (uint32_t)(qt * kFltM + rows);
            const uint32_t base = (uint32_t)(S.lo[qt] + (i0 + i - S.start[qt]) * kFltN) + half;
            const uint32_t t0 = S.tmem + ((uint32_t)rows << 16) + buf * kFltN + half;
            uint32_t v0[32], v1[32];
            tmem_load32(t0, v0);
#pragma unroll 1
            for (int c0 = 0; c0 < kFltN / 2; c0 += 64) {
                tmem_wait(v0);
                tmem_load32(t0 + c0 + 32, v1);
                take(v0, q, base + c0);
                tmem_wait(v1);
                if (c0 + 64 < kFltN / 2) tmem_load32(t0 + c0 + 64, v0);
                take(v1, q, base + c0 + 32);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.tempty[buf]);
        }
        if (held > 0) flush();
        if (lane == 0) atomicAdd(&S.done, 1);
    } else if (warp >= 4 + kFltReaders) {
        const int r = tid - (4 + kFltReaders) * 32;                         // a choice of the tile each
        int built = -1;
        uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;      // the next tile's signature, in flight
        bool nvalid = false;
        auto fetch = [&](int i) {
            advance(i);
            const int64_t x = S.lo[qt] + (i0 + i - S.start[qt]) * kFltN + r;
            nvalid = x < S.hi[qt];
            if (nvalid) {
                const uint4 *p = reinterpret_cast<const uint4 *>(csig) + x * 2;
                n0 = __ldg(p);
                n1 = __ldg(p + 1);
            } else {
                n0 = n1 = make_uint4(0, 0, 0, 0);
            }
        };
        if (ntiles > 0) fetch(0);
        for (int i = 0; i < ntiles; i++) {
            const int buf = i & 1, qcur = qt;
            const uint32_t par = (uint32_t)(i >> 1) & 1u;
            uint32_t wd[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
            if (K == 128) sig_fold(wd);
            const bool valid = nvalid;
            if (i + 1 < ntiles) fetch(i + 1);
            if (!warp_wait(&S.abort, &S.empty[buf], par ^ 1u, polls, status)) break;
            if (qcur != built) {
                // the queries' rows: every product on the old ones has to be done
                if (i > 0 && !warp_wait(&S.abort, &S.empty[buf ^ 1], (uint32_t)((i - 1) >> 1) & 1u, polls, status)) break;
                built = qcur;
                const int row = r & (kFltM - 1), half = r / kFltM;       // two threads a row
                const int q = qcur * kFltM + row;
                uint32_t qw[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (q < nq) {
                    int at;
                    const int c = seq_query(SC, q, at);
                    const uint32_t *p = qsig + (size_t)SC.cls[c].qidx[at] * kSigWords;
#pragma unroll
                    for (int x = 0; x < 8; x++) qw[x] = __ldg(p + x);
                }
                if (K == 128) sig_fold(qw);
                int bits = 0;
#pragma unroll
                for (int x = 0; x < K / 32; x++) bits += __popc(qw[x]);
                uint32_t tlo, thi;
                sig_query_tail(bits, q < nq, tlo, thi);
                write_row<kFltM, K>(S.a, row, half * (K / 32), (half + 1) * (K / 32), [&](int x) {
                    return x == W - 2 ? tlo : x == W - 1 ? thi : sig_query_word(qw, x >> 3, x & 7);
                });
            }
            int bits = 0;
#pragma unroll
            for (int x = 0; x < K / 32; x++) bits += __popc(wd[x]);
            uint32_t tlo, thi;
            sig_choice_tail(bits, k, valid, tlo, thi);
            write_row<kFltN, K>(S.b[buf], r, 0, K / 16, [&](int x) {
                return x == W - 2 ? tlo : x == W - 1 ? thi : sig_choice_word(wd, x >> 3, x & 7);
            });
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.full[buf]);
        }
    }
    }
    // products in flight end before TMEM goes back: the last commits of both
    // buffers (under the normal bound, whatever `polls` is)
    for (int i = max(0, issued - 2); i < issued; i++)
        if (!mbar_wait(&S.tfull[i & 1], (uint32_t)(i >> 1) & 1u)) atomicOr(status, ST_QUEUE_TIMEOUT);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(512) : "memory");
}

// The listed pairs, a lane each, by furthest-reaching points (blg_reach.cuh),
// where the banded loop (survivor_warp) walks every column of a near-copy with
// two scattered loads of the query's Peq rows, 32 lanes in 64 cache lines:
// 52,000 passers of 100 to 256 bytes at k = 4 took 84 us that way and take 50.
// The strings are first copied into shared memory, whose slots hold the launch's
// longest (sequential queries end at 512 bytes).
// The filter leaves off filling the output when its tiles are done, long
// before 1 GiB is written; here a third warp goes on with it, and as the fill
// may pass an element after its result, results go to a list (list_emit) that
// k_solve_finish stores. L.item null: the output is filled, results in place.
constexpr int kLvThreads = 64;
constexpr int kLvMaxK = kSigMaxK;
constexpr int kLvMaxLength = 512;                        // of a query: 64 bytes of each of eight words

// The repair launch's plan and its gate, by the blocks of a launch.
__device__ __forceinline__ void repair_plan(const SurvClasses &C, const RepairPlan &R, int k) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *R.gate.count = R.gate.cap + 1;
    if (blockIdx.x < C.n) surv_plan_class(C, blockIdx.x, R.lstart, R.min_len, R.n_len, k, R.jobsz);
}

__global__ void __launch_bounds__(kLvThreads + 32)
    k_solve_passers(SurvClasses C, DevStrings Q, DevStrings CS, const int32_t *perm, const uint4 *ccnt,
                    const uint4 *qcnt, int k, int dtype, void *out, int64_t nc, int slot, PasserList P, ResultList L,
                    BatchFill fill, RepairPlan plan, uint32_t *status) {
    extern __shared__ __align__(16) uint8_t s_dyn[];     // per warp [2][32][slot], then F
    __shared__ __align__(16) uint8_t s_pattern[kFillPiece];
    __shared__ __align__(16) unsigned char s_raw[sizeof(SurvClasses)];
    SurvClasses &SC = *reinterpret_cast<SurvClasses *>(s_raw);
    for (int x = threadIdx.x; x < (int)(sizeof(SurvClasses) / 4); x += blockDim.x)
        reinterpret_cast<uint32_t *>(s_raw)[x] = reinterpret_cast<const uint32_t *>(&C)[x];
    fill_pattern(s_pattern, fill);
    __syncthreads();
    const unsigned long long total = *P.count;
    if (total > P.cap) {                                 // the whole search runs in place, over a filled output
        if (!L.item) repair_plan(SC, plan, k);           // (else k_solve_finish plans it)
        return;
    }
    if (threadIdx.x >= kLvThreads) {
        fill_items(fill, P.count + 1, s_pattern, false, [] { return false; });
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t *slots = s_dyn + warp * 64 * slot;
    int16_t *f = reinterpret_cast<int16_t *>(s_dyn + (kLvThreads / 32) * 64 * slot) + (k + 1) * kLvThreads + threadIdx.x;
    const unsigned long long warps = (unsigned long long)gridDim.x * (kLvThreads / 32);
    for (unsigned long long at = ((unsigned long long)blockIdx.x * (kLvThreads / 32) + warp) * 32; at < total;
         at += warps * 32) {
        bool live = at + lane < total;
        const uint8_t *a = Q.buf, *b = CS.buf;
        int m = 0, n = 0;
        int64_t oidx = 0;
        if (live) {
            const unsigned long long e = P.item[at + lane];
            const int64_t sidx = (int64_t)(e & 0xffffffffu);
            int qi;
            const int cls = seq_query(SC, (int)(e >> 32), qi);
            const int64_t row = __ldg(SC.cls[cls].qidx + qi);
            const uint4 cc = __ldg(ccnt + sidx);
            b = string_at(CS, sidx, n, status);
            a = string_at(Q, row, m, status);
            oidx = row * nc + perm[sidx];
            // outside the length window, or beyond k by the 16-bin counts: the output keeps its k + 1
            live = (n > m ? n - m : m - n) <= k && gram_dist(__ldg(qcnt + row), cc) <= 8u * (uint32_t)k;
        }
        const int sa = (int)(reinterpret_cast<uintptr_t>(a) & 15), sb = (int)(reinterpret_cast<uintptr_t>(b) & 15);
        // the lane's strings into its slots, 16 bytes at a time, all in flight at once (a lane's own copies: 24
        // instructions a warp for what shuffled addresses and whole lines took 1100)
        __syncwarp();
        if (live) {
            const uint32_t dst = smem_addr(slots + lane * slot);
            const uint8_t *pa = a - sa, *pb = b - sb;
            for (int x = 0; x < sa + m; x += 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + x), "l"(pa + x) : "memory");
            for (int x = 0; x < sb + n; x += 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 32 * slot + x), "l"(pb + x) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!live) continue;
        const uint32_t base = (uint32_t)(warp * 64 + lane) * (uint32_t)slot;
        const uint32_t *w = reinterpret_cast<const uint32_t *>(s_dyn);
        const int d = furthest_distance<kLvThreads>(w, base + sa, m, w, base + 32 * slot + sb, n, k, f);
        if (d <= k) {
            if (L.item) list_emit(L, out, dtype, oidx, d);
            else store1(out, dtype, oidx, d);
        }
    }
}

// After a run with listed results: they go to the output. Where a list ran
// full, the output's k + 1 and the plan of the repair launch instead, which
// does the whole search in place (gate: its count past its cap).
__global__ void __launch_bounds__(256)
    k_solve_finish(SurvClasses C, int k, PasserList P, ResultList L, BatchFill fill, RepairPlan plan) {
    __shared__ __align__(16) unsigned char s_raw[sizeof(SurvClasses)];
    SurvClasses &SC = *reinterpret_cast<SurvClasses *>(s_raw);
    const unsigned long long passers = *P.count, results = *L.count;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (passers <= P.cap && results <= L.cap) {
        for (int64_t i = tid; i < (int64_t)results; i += stride) {
            const unsigned long long e = L.item[i];
            store1(reinterpret_cast<void *>((uintptr_t)(e >> 8)), (int)((e >> 6) & 3u), 0, (int)(e & 63u));
        }
        return;
    }
    if (passers > P.cap) fill_share(fill.out, fill.n, fill.dtype, fill.value, tid, stride);   // (nobody went on with it)
    if (threadIdx.x == 0) SC = C;
    __syncthreads();
    repair_plan(SC, plan, k);
}

// ------------------------------------------------------------- launchers --
template <int K>
static cudaError_t launch_filter_k(cudaStream_t st, int sms, const SurvClasses &C, int nq, const uint32_t *qsig,
                                   const uint32_t *csig, const int64_t *lstart, int64_t min_len, int64_t n_len, int k,
                                   const PasserList &L, const BatchFill &fill, bool whole_fill, uint32_t polls,
                                   uint32_t *status) {
    const int smem = (int)sizeof(FilterShared<K>);
    const cudaError_t e = cudaFuncSetAttribute(k_filter_pairs<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_filter_pairs<K><<<sms, kFltThreads, smem, st>>>(C, nq, qsig, csig, lstart, min_len, n_len, k, L, fill, whole_fill,
                                                      polls, status);
    return cudaGetLastError();
}

cudaError_t launch_filter_pairs(cudaStream_t st, int sms, const SurvClasses &C, int nq, const uint32_t *qsig,
                                const uint32_t *csig, bool folded, const int64_t *lstart, int64_t min_len,
                                int64_t n_len, int k, const PasserList &L, const BatchFill &fill, bool whole_fill,
                                int32_t wait_polls, uint32_t *status) {
    if (nq <= 0 || C.n <= 0) return cudaSuccess;
    if (k < 0 || k > kSigMaxK || (nq + kFltM - 1) / kFltM > kFltMaxTiles) return cudaErrorInvalidValue;
    const uint32_t polls = wait_polls < 0 ? kMbarPolls : (uint32_t)wait_polls;
    return folded ? launch_filter_k<128>(st, sms, C, nq, qsig, csig, lstart, min_len, n_len, k, L, fill, whole_fill, polls, status)
                  : launch_filter_k<256>(st, sms, C, nq, qsig, csig, lstart, min_len, n_len, k, L, fill, whole_fill, polls, status);
}

cudaError_t launch_solve_passers(cudaStream_t st, int sms, const SurvClasses &C, const DevStrings &Q,
                                 const DevStrings &CS, const int32_t *perm, const uint4 *ccnt, const uint4 *qcnt,
                                 int64_t longest, int k, int dtype, void *out, int64_t nc, const PasserList &P,
                                 const ResultList &L, const BatchFill &fill, const RepairPlan &plan, uint32_t *status) {
    if (C.n <= 0) return cudaSuccess;
    if (k < 0 || k > kLvMaxK || longest > kLvMaxLength) return cudaErrorInvalidValue;
    // a slot holds the launch's longest strings from any 16-byte boundary and octet's
    // slack (a string up to k longer than its query), an odd number of 16-byte banks
    int slot = (int)(longest + k + 15 + 16 + 15) & ~15;
    if (!(slot & 16)) slot += 16;
    const int smem = (kLvThreads / 32) * 64 * slot + (2 * k + 3) * kLvThreads * 2;
    cudaError_t e = cudaFuncSetAttribute(k_solve_passers, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve_passers, kLvThreads + 32, smem);
    if (e != cudaSuccess) return e;
    k_solve_passers<<<sms * std::max(1, per_sm), kLvThreads + 32, smem, st>>>(C, Q, CS, perm, ccnt, qcnt, k, dtype, out, nc,
                                                                             slot, P, L, fill, plan, status);
    return cudaGetLastError();
}

cudaError_t launch_solve_finish(cudaStream_t st, int sms, const SurvClasses &C, int k, const PasserList &P,
                                const ResultList &L, const BatchFill &fill, const RepairPlan &plan) {
    k_solve_finish<<<sms * 2, 256, 0, st>>>(C, k, P, L, fill, plan);
    return cudaGetLastError();
}

}  // namespace blg
