"""Exact pairs in bands first (k_pairs_near, k_pairs_mid): distances on both
sides of 31 and 63, batch and block edges, both row layouts, and what the bands
leave to the full-width solvers. Integer distances, compared for equality."""
import ctypes

import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _build, _lib, workloads as W
from test_search_filter import TEXT


@pytest.mark.parametrize("k", [0, 1, 31, 32, 33, 62, 63])
def test_band64_host(k):
    lib = ctypes.CDLL(_build.build_hostcheck())
    rng = np.random.default_rng(k)
    a = W.random_strings(rng, rng.integers(1, 257, 300))
    b = W.mutate(rng, a, rng.uniform(0, 0.4, 300))
    want = oracle.pairs(a, b, k)
    for i in range(300):
        x, y = a[0][a[1][i]:a[1][i + 1]].tobytes(), b[0][b[1][i]:b[1][i + 1]].tobytes()
        if len(x) > len(y):
            x, y = y, x
        if x and len(y) - len(x) <= k:
            assert lib.blg_host_band64(x, len(x), y, len(y), k) == want[i]


def _run(s, out):
    ctx = _lib.context()
    ctx.check(ctx.lib.blg_profile_enable(ctx.h, 1))
    s.run(out)
    buf = ctypes.create_string_buffer(8192)
    ctx.check(ctx.lib.blg_profile_report(ctx.h, buf, 8192))
    ctx.check(ctx.lib.blg_profile_enable(ctx.h, 0))
    return out.get(), buf.value.decode()


@pytest.mark.gpu
@pytest.mark.parametrize("n,lo,hi,alphabet,rate", [(66001, 8, 256, W.DNA_N, 0.3), (70000, 30, 300, TEXT, 0.4),
                                                   (257, 33, 128, W.DNA, 0.3), (4099, 0, 128, TEXT, 0.2),
                                                   (66000, 60, 600, W.DNA, 0.1), (65536, 33, 40, W.DNA, 0.2)])
def test_bands_pairs(gpu, n, lo, hi, alphabet, rate):
    rng = np.random.default_rng(n + hi)
    a = W.random_strings(rng, rng.integers(lo, hi + 1, n), alphabet)
    b = W.mutate(rng, a, rng.uniform(0, rate, n), alphabet)
    far = rng.choice(n, n // 50, replace=False)               # unrelated and empty partners among the near ones
    order = np.arange(n)
    order[far] = n + np.arange(len(far))
    b = W.take(W.concat(b, W.random_strings(rng, rng.integers(0, hi + 1, len(far)), alphabet)), order)
    want = oracle.pairs(a, b, None, threads=8)
    for x, y in ((a, b), (b, a)):
        s = gpu.PairsBatch(x, y)
        for dt in ("int32", "uint16", "uint8"):
            got, labels = _run(s, s.alloc(dt))
            np.testing.assert_array_equal(got, oracle.saturate(want, dt))
            assert "pairs_bands" in labels, labels
    out = s.alloc("int32")
    for _ in range(3):                                        # direct, captured, replayed
        s.run(out)
    np.testing.assert_array_equal(out.get(), want)


@pytest.mark.gpu
def test_unrelated_pairs_keep_the_full_width_path(gpu):
    rng = np.random.default_rng(4)
    a, b = (W.random_strings(rng, rng.integers(60, 200, 70000)) for _ in range(2))
    s = gpu.PairsBatch(a, b)
    got, labels = _run(s, s.alloc("int32"))
    assert "pairs_bands" not in labels, labels
    np.testing.assert_array_equal(got, oracle.pairs(a, b, None, threads=8))
