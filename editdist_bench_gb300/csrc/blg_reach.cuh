// Thresholded edit distance by furthest-reaching points (Ukkonen 1985; Landau
// and Vishkin 1989): F(e, d) is the last position of the first string that e
// edits can reach on diagonal d = j - i, F(e, d) = max(F(e-1, d) + 1, F(e-1, d-1),
// F(e-1, d+1) + 1) extended over equal characters, eight at a time; the
// distance is the first e with F(e, n - m) = m. A pair takes at most about k^2
// / 2 steps and n / 8 more, whatever its strings' bytes.
#pragma once
#include "blg_device.cuh"

namespace blg {

// Eight characters at byte offset p of the words s: three words and two funnel
// shifts (reads up to 11 bytes past the last character asked for).
__device__ __forceinline__ uint2 octet(const uint32_t *s, uint32_t p) {
    const uint32_t *w = s + (p >> 2);
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2], sh = (p & 3u) * 8u;
    return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}

// min(d, k + 1) of m characters at byte offset a of A and n at b of B; |n - m| <=
// k, m and n below 32767. f: this thread's column of F(e - 1, .), diagonal 0,
// stride T, room from -k - 1 to k + 1. One flat loop: an iteration compares
// eight characters on the lane's diagonal and, where they end the run, moves
// to its next one. Lanes of a warp are in different runs, so loops within the
// loop would last as long as the warp's longest run at every step (7400 warp
// instructions for 32 pairs of 100 to 256 bytes at k = 4, measured).
template <int T>
__device__ __forceinline__ int furthest_distance(const uint32_t *A, uint32_t a, int m, const uint32_t *B, uint32_t b, int n,
                                                 int k, int16_t *f) {
    const int goal = n - m;
    const int glo = goal - k, ghi = goal + k;
    int e = 0, d = 0, hi = 0, i = 0, end = min(m, n), mid = -2, right = -2;
    int16_t *p = f;
    f[-T] = f[T] = -2;                                       // diagonals not reached yet
    while (true) {
        const uint2 x = octet(A, a + i), y = octet(B, b + i + d);
        const uint32_t u = x.x ^ y.x, v = x.y ^ y.y;
        const uint32_t w = u ? u : v;
        const int q = (u ? 0 : 4) + (w ? (__ffs(w) - 1) >> 3 : 4);
        i = min(i + q, end);
        if (q == 8 && i < end) continue;
        if (d == goal && i >= m) return e;
        *p = (int16_t)i;
        // the next diagonal, or the next number of edits from its lowest one, by
        // selects: some lane of the warp changes level at nearly every step
        const bool up = d == hi;
        e += up ? 1 : 0;
        if (e > k) return k + 1;
        if (up) {
            f[(e + 1) * T] = -2;
            f[(-e - 1) * T] = -2;
        }
        // the diagonals that a path of k edits to the goal can still be on
        const int lo = max(max(-e, glo + e), -m);
        hi = min(min(e, ghi - e), n);
        d = up ? lo : d + 1;
        p = f + d * T;
        const int left = up ? (int)p[-T] : mid;
        mid = up ? (int)p[0] : right;
        right = p[T];
        end = min(m, n - d);                                 // the diagonal's last position
        i = min(max(max(mid + 1, left), right + 1), end);
    }
}

}  // namespace blg
