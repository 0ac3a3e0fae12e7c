// Exact distances of pairs that are mostly near each other: bands first.
//
// The full-width solvers spread a pattern's 64-bit words over lanes and walk
// the whole matrix (blg_pairs_sched.cu; the reference one thread per pair,
// csrc/gpu_kernels.cu:6-32). A pair within 31 edits needs a 32-bit window per
// column (band_core in blg_device.cuh), one within 63 a 64-bit window, whatever
// its length, and the pairs that are compared at all are mostly copies of each
// other:
//  1. k_pairs_near runs every pair in a band of 31, batches of consecutive pairs
//     sorted by length inside a CTA. Pairs beyond it go to a list.
//  2. k_pairs_mid runs the list in a band of 63. What is left goes to the
//     full-width solvers' records.
// Unrelated pairs leave either band after some 2 k columns.
//
// Bound: instruction issue of the column loops (45 instructions a column and
// lane in the 32-bit band, 70 in the 64-bit one), and for few pairs the chain
// of one warp's columns. 250007 pairs of 8 to 256 bytes with up to 30% edits: 105
// us near, 70 mid, 59 for the 600 pairs left, 243 in all against 355 of the
// full-width path.
#include <algorithm>

#include "blg_kernels.cuh"
#include "blg_sched.h"
#include "blg_tma.cuh"

namespace blg {

constexpr int kNearThreads = 256, kNearMaxBatch = 1024, kNearK = 31;
constexpr int kMidThreads = 64, kMidK = 63;

// The warp's lanes with `push` set append their record to a list (capacity:
// every pair).
__device__ __forceinline__ void push_record(bool push, const LongItem &it, LongItem *list, int32_t *count) {
    const unsigned mask = __ballot_sync(kFull, push);
    if (!mask) return;
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (lane == __ffs(mask) - 1) at = atomicAdd(count, __popc(mask));
    at = __shfl_sync(kFull, at, __ffs(mask) - 1) + __popc(mask & ((1u << lane) - 1u));
    if (push) list[at] = it;
}

__device__ __forceinline__ TextScan scan_at(const uint8_t *p) {
    TextScan s;
    s.init(p);
    return s;
}

// batch: consecutive pairs a CTA takes at a time, sorts by columns (longer
// string, buckets of four) and hands to its warps 32 at a time, longest first:
// lanes of a warp walk alike and still read one neighbourhood of memory. In
// natural order half of the lanes idled (15.4k warp instructions for 32 pairs
// of 8 to 256 bytes, 215 us for 250007 pairs with the spans staged).
template <bool SYM>
__global__ void __launch_bounds__(kNearThreads)
    k_pairs_near(DevStrings A, DevStrings B, int batch, int dtype, void *out, LongItem *far, int32_t *nfar,
                 const uint32_t *alpha, uint32_t *status) {
    extern __shared__ __align__(16) uint8_t s_dyn[];           // rows [R][threads] uint2
    __shared__ uint8_t s_map[256];
    __shared__ uint16_t s_order[kNearMaxBatch];
    __shared__ int s_hist[256], s_next;
    if (alpha && (alpha_size(alpha) <= kBandSymbols) != SYM) return;   // uniform: the other variant runs the set
    if (SYM) alpha_map(alpha, s_map);
    const int tid = threadIdx.x, lane = tid & 31;
    uint2 *tc = reinterpret_cast<uint2 *>(s_dyn) + tid;
    for (int64_t first = (int64_t)blockIdx.x * batch; first < A.n; first += (int64_t)gridDim.x * batch) {
        const int cnt = (int)min((int64_t)batch, A.n - first);
        __syncthreads();                                       // the previous batch is done with the order
        s_hist[tid] = 0;
        if (tid == 0) s_next = 0;
        __syncthreads();
        int key[kNearMaxBatch / kNearThreads], rank[kNearMaxBatch / kNearThreads];
#pragma unroll
        for (int x = 0; x < kNearMaxBatch / kNearThreads; x++) {
            const int j = x * kNearThreads + tid;
            key[x] = -1;
            if (j < cnt) {
                const int64_t la = A.off[first + j + 1] - A.off[first + j], lb = B.off[first + j + 1] - B.off[first + j];
                key[x] = 255 - (int)min((int64_t)255, (la > lb ? la : lb) >> 2);
                rank[x] = atomicAdd(&s_hist[key[x]], 1);
            }
        }
        __syncthreads();
        if (tid < 32) {                                        // exclusive scan, eight buckets a lane
            int v[8], sum = 0;
#pragma unroll
            for (int x = 0; x < 8; x++) { v[x] = s_hist[tid * 8 + x]; sum += v[x]; }
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, incl, o);
                if (tid >= o) incl += y;
            }
            int run = incl - sum;
#pragma unroll
            for (int x = 0; x < 8; x++) { s_hist[tid * 8 + x] = run; run += v[x]; }
        }
        __syncthreads();
#pragma unroll
        for (int x = 0; x < kNearMaxBatch / kNearThreads; x++)
            if (key[x] >= 0) s_order[s_hist[key[x]] + rank[x]] = (uint16_t)(x * kNearThreads + tid);
        __syncthreads();
        while (true) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s_next, 32);
            at = __shfl_sync(kFull, at, 0) + lane;
            if (at - lane >= cnt) break;
            LongItem it;
            it.pat = it.txt = nullptr;
            it.m = it.n = 0;
            it.idx = 0;
            bool push = false;
            if (at < cnt) {
                it.idx = first + s_order[at];
                int la, lb;
                const uint8_t *a = string_at(A, it.idx, la, status), *b = string_at(B, it.idx, lb, status);
                const bool swap = la > lb;                     // the shorter string is the pattern
                it.pat = swap ? b : a;
                it.txt = swap ? a : b;
                it.m = swap ? lb : la;
                it.n = swap ? la : lb;
                int d = kNearK + 1;
                if (it.m == 0) d = it.n;
                else if (it.n - it.m <= kNearK)
                    d = band_rows_distance<SYM, kNearThreads>(tc, s_map, [&](int pos) { return scan_at(it.pat + pos); },
                                                              [&](int pos) { return scan_at(it.txt + pos); }, it.m, it.n,
                                                              kNearK, nullptr);
                push = it.m > 0 && d > kNearK;
                if (!push) store1(out, dtype, it.idx, d);
            }
            __syncwarp();
            push_record(push, it, far, nfar);
        }
    }
}

// The listed pairs in a band of 63. Per-thread rows of three 32-bit words over a
// 96-position block of the pattern (band_rows_distance with one word more):
// columns 32 b .. 32 b + 31 read their 64-bit windows with two funnel shifts;
// every 32 columns the rows move down a word and 32 pattern bytes enter.
template <bool SYM>
__global__ void __launch_bounds__(kMidThreads)
    k_pairs_mid(PairsPlan plan, const LongItem *far, const int32_t *nfar, int dtype, void *out, int32_t *left,
                const uint32_t *alpha) {
    constexpr int R = SYM ? kBandSymbols + 1 : 32, T = kMidThreads;
    extern __shared__ __align__(16) uint8_t s_dyn[];           // rows [R][3][threads]
    __shared__ uint8_t s_map[256];
    if (alpha && (alpha_size(alpha) <= kBandSymbols) != SYM) return;
    if (SYM) alpha_map(alpha, s_map);
    const int lane = threadIdx.x & 31;
    uint32_t *rows = reinterpret_cast<uint32_t *>(s_dyn) + threadIdx.x;        // word w of row r at [(r * 3 + w) * T]
    const int total = *nfar;
    for (int base = (blockIdx.x * T + threadIdx.x) & ~31; base < total; base += gridDim.x * T) {
        const bool valid = base + lane < total;
        LongItem it;
        it.m = it.n = 0;
        if (valid) it = far[base + lane];
        const uint8_t *p = it.pat, *t = it.txt;
        __syncwarp();
        int cls = -1;
        if (valid) {
            const int m = it.m, n = it.n;
            int d = kMidK + 1;
            if (n - m <= kMidK) {
                const int dhi = (n - m) + ((kMidK - (n - m)) >> 1);
                auto enter = [&](uint32_t c, int bit) {        // pattern byte c at block bit `bit` (0..95)
                    const uint32_t v = 1u << (bit & 31);
                    if (SYM) {
                        rows[(s_map[c] * 3 + (bit >> 5)) * T] |= v;
                    } else {
                        rows[((c >> 4) * 3 + (bit >> 5)) * T] |= v;
                        rows[((16 + (c & 15)) * 3 + (bit >> 5)) * T] |= v;
                    }
                };
#pragma unroll
                for (int r = 0; r < R * 3; r++) rows[r * T] = 0;
                int next = min(m, 96 - dhi);                   // block 0: positions 0 .. next - 1 at bits pos + dhi
                auto ps = scan_at(p);
                {
                    auto fs = scan_at(p);
                    for (int x = 0; x < next; x += 4) {
                        const uint32_t w4 = fs.next4();
#pragma unroll
                        for (int b = 0; b < 4; b++)
                            if (x + b < next) enter((w4 >> (8 * b)) & 0xffu, x + b + dhi);
                    }
                    ps = scan_at(p + next);
                }
                auto ts = scan_at(t);
                d = band64_core(m, n, kMidK, [&](int j, int, uint64_t (&e)[4]) {
                    if ((j & 31) == 0 && j > 0) {
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            rows[(r * 3) * T] = rows[(r * 3 + 1) * T];
                            rows[(r * 3 + 1) * T] = rows[(r * 3 + 2) * T];
                            rows[(r * 3 + 2) * T] = 0;
                        }
                        const int cnt = min(32, m - next);
                        for (int x = 0; x < cnt; x += 4) {
                            const uint32_t q4 = ps.next4();
#pragma unroll
                            for (int b = 0; b < 4; b++)
                                if (x + b < cnt) enter((q4 >> (8 * b)) & 0xffu, 64 + x + b);
                        }
                        next += max(cnt, 0);
                    }
                    const uint32_t w4 = ts.next4();
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        const uint32_t c = (w4 >> (8 * x)) & 0xffu;
                        uint32_t w0, w1, w2;
                        if (SYM) {
                            const uint32_t *r = rows + s_map[c] * 3 * T;
                            w0 = r[0], w1 = r[T], w2 = r[2 * T];
                        } else {
                            const uint32_t *h = rows + (c >> 4) * 3 * T, *l = rows + (16 + (c & 15)) * 3 * T;
                            w0 = h[0] & l[0], w1 = h[T] & l[T], w2 = h[2 * T] & l[2 * T];
                        }
                        const uint32_t sh = (uint32_t)((j + x) & 31);
                        e[x] = (uint64_t)__funnelshift_r(w1, w2, sh) << 32 | __funnelshift_r(w0, w1, sh);
                    }
                });
            }
            if (d <= kMidK) store1(out, dtype, it.idx, d);
            else {
                const int W = (m + 63) >> 6;
                cls = W <= 1 ? 0 : W <= 2 ? 1 : W <= 4 ? 2 : W <= 8 ? 3 : W <= 16 ? 4 : 5;
            }
        }
#pragma unroll
        for (int c = 0; c < kPairClasses; c++) push_record(cls == c, it, plan.sorted[c], left + c);
    }
}

// ------------------------------------------------------------- launchers --
// Both launches: variant and alpha as for launch_solve_band. far, nfar: the
// first kernel's list (room for every pair; zero count), left: the counts of
// the records left in plan.sorted (zero).
template <bool SYM>
static cudaError_t launch_near_mid(cudaStream_t st, int sms, const DevStrings &A, const DevStrings &B, int dtype, void *out, const PairsPlan &plan, LongItem *far, int32_t *nfar,
                                   int32_t *left, const uint32_t *alpha, uint32_t *status) {
    constexpr int R = SYM ? kBandSymbols + 1 : 32;
    // six batches an SM where there are pairs enough: blocks come and go, so the
    // longest ones do not decide
    int batch = kNearMaxBatch;
    while (batch > kNearThreads && (A.n + batch - 1) / batch < 6 * (int64_t)sms) batch >>= 1;
    int smem = R * kNearThreads * 8, per_sm = 1;
    cudaError_t e = cudaFuncSetAttribute(k_pairs_near<SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int64_t want = (A.n + batch - 1) / batch;
    k_pairs_near<SYM><<<(unsigned)std::min<int64_t>(want, 1 << 20), kNearThreads, smem, st>>>(A, B, batch, dtype, out, far,
                                                                                            nfar, alpha, status);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    smem = R * 3 * kMidThreads * 4;
    e = cudaFuncSetAttribute(k_pairs_mid<SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pairs_mid<SYM>, kMidThreads, smem);
    if (e != cudaSuccess) return e;
    k_pairs_mid<SYM><<<sms * std::max(1, per_sm), kMidThreads, smem, st>>>(plan, far, nfar, dtype, out, left, alpha);
    return cudaGetLastError();
}

cudaError_t launch_pairs_bands(cudaStream_t st, int sms, const DevStrings &A, const DevStrings &B, int dtype,
                               void *out, const PairsPlan &plan, LongItem *far, int32_t *nfar, int32_t *left,
                               int variant, const uint32_t *alpha, uint32_t *status) {
    if (A.n <= 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (variant != 0) e = launch_near_mid<true>(st, sms, A, B, dtype, out, plan, far, nfar, left, alpha, status);
    if (e == cudaSuccess && variant != 1)
        e = launch_near_mid<false>(st, sms, A, B, dtype, out, plan, far, nfar, left, variant < 0 ? alpha : nullptr, status);
    return e;
}

}  // namespace blg
