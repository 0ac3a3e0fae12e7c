// Pairs under a small max_dist: one kernel over furthest-reaching points.
//
// The scheduled path (blg_pairs_sched.cu) trims every pair, writes a 32-byte
// record, sorts the records by cost and walks each pair's columns in the banded
// loop, 25 instructions each, reading scattered strings a second time. With a
// small k a pair takes some k^2 / 2 diagonals and an eighth of a column step
// per character instead (blg_reach.cuh; the common prefix is its first run, so
// nothing is trimmed), and the pairs can be taken in natural order: a warp's 32
// pairs are one contiguous span of either side, copied into shared memory whole
// lines at a time, and its results are stored together. No records, no sort,
// no second read. (The reference runs its column loop per pair over global
// memory, csrc/gpu_kernels.cu:6-32.)
//
// Bound: instruction issue of the lanes' own loops, some 90 a step, and their
// divergence (a warp lasts as long as its longest pair); at k <= 1 the strings'
// way from HBM. 2^20 pairs of 8 to 256 bytes, uint8: 302 us at k = 8 (scheduled
// path 385), 81 at k = 1 (198); 300007 lines of 4 to 60 at k = 3 19 (63).
#include <algorithm>

#include "blg_kernels.cuh"
#include "blg_reach.cuh"
#include "blg_tma.cuh"

namespace blg {

constexpr int kReachThreads = 128;

__global__ void __launch_bounds__(kReachThreads)
    k_pairs_reach(DevStrings A, DevStrings B, int span, int k, int dtype, void *out, uint32_t *status) {
    extern __shared__ __align__(16) uint8_t s_dyn[];   // per warp [2][side], then F
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int side = span + 32;                        // (octet's slack)
    uint8_t *sa = s_dyn + warp * 2 * side, *sb = sa + side;
    int16_t *f = reinterpret_cast<int16_t *>(s_dyn + (kReachThreads / 32) * 2 * side) + (k + 1) * kReachThreads +
                 threadIdx.x;
    const int64_t n = A.n, warps = (int64_t)gridDim.x * (kReachThreads / 32);
    for (int64_t g = (int64_t)blockIdx.x * (kReachThreads / 32) + warp; g * 32 < n; g += warps) {
        const int64_t i = g * 32 + lane;
        const bool valid = i < n;
        int la = 0, lb = 0;
        const uint8_t *ga = valid ? string_at(A, i, la, status) : A.buf;
        const uint8_t *gb = valid ? string_at(B, i, lb, status) : B.buf;
        // the group's spans: offsets are in order (the launcher's condition)
        const int last = (int)min((int64_t)32, n - g * 32) - 1;
        auto first16 = [&](const uint8_t *p) {
            return (unsigned long long)__shfl_sync(kFull, (unsigned long long)reinterpret_cast<uintptr_t>(p), 0) & ~15ull;
        };
        const unsigned long long a0 = first16(ga), b0 = first16(gb),
                                 a1 = __shfl_sync(kFull, (unsigned long long)reinterpret_cast<uintptr_t>(ga + la), last),
                                 b1 = __shfl_sync(kFull, (unsigned long long)reinterpret_cast<uintptr_t>(gb + lb), last);
        const bool staged = a1 - a0 <= (unsigned)span && b1 - b0 <= (unsigned)span;
        __syncwarp();                                  // the previous group is done with the stage
        if (staged) {
            for (uint32_t x = lane * 16; x < (uint32_t)(a1 - a0); x += 512)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(sa + x)), "l"(a0 + x) : "memory");
            for (uint32_t x = lane * 16; x < (uint32_t)(b1 - b0); x += 512)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(sb + x)), "l"(b0 + x) : "memory");
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncwarp();
        if (valid) {
            int d = k + 1;
            if ((la > lb ? la - lb : lb - la) <= k) {
                const uintptr_t ua = reinterpret_cast<uintptr_t>(ga), ub = reinterpret_cast<uintptr_t>(gb);
                if (staged)
                    d = furthest_distance<kReachThreads>(reinterpret_cast<const uint32_t *>(sa), (uint32_t)(ua - a0), la,
                                                         reinterpret_cast<const uint32_t *>(sb), (uint32_t)(ub - b0), lb, k, f);
                else
                    d = furthest_distance<kReachThreads>(reinterpret_cast<const uint32_t *>(ua & ~uintptr_t(3)),
                                                         (uint32_t)(ua & 3), la,
                                                         reinterpret_cast<const uint32_t *>(ub & ~uintptr_t(3)),
                                                         (uint32_t)(ub & 3), lb, k, f);
            }
            store1(out, dtype, i, d);
        }
    }
}

// The offsets of A and B are in order, and no pair's shorter string is longer
// than the other kernels' limit of 2048 (which they refuse by pair).
// avg: mean bytes of the longer side's strings, which sizes the stage (a quarter
// more than 32 of them: groups differ).
cudaError_t launch_pairs_reach(cudaStream_t st, int sms, const DevStrings &A, const DevStrings &B, double avg, int k,
                               int dtype, void *out, uint32_t *status) {
    if (A.n <= 0) return cudaSuccess;
    if (k < 0 || k > 31) return cudaErrorInvalidValue;
    const int span = std::min(kReachMaxSpan, ((int)std::min(avg * 40.0, 1e6) + 256) & ~15);
    const int smem = (kReachThreads / 32) * 2 * (span + 32) + (2 * k + 3) * kReachThreads * 2;
    cudaError_t e = cudaFuncSetAttribute(k_pairs_reach, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pairs_reach, kReachThreads, smem);
    if (e != cudaSuccess) return e;
    const int64_t want = (A.n + kReachThreads - 1) / kReachThreads;
    k_pairs_reach<<<(unsigned)std::min<int64_t>(want, (int64_t)sms * std::max(1, per_sm)), kReachThreads, smem, st>>>(
        A, B, span, k, dtype, out, status);
    return cudaGetLastError();
}

}  // namespace blg
