"""Thresholded pairs by furthest-reaching points (k_pairs_reach): equal to the
oracle at the edges of its groups of 32 pairs, its stage, its length windows
and its max_dist range. Integer distances, compared for equality."""
import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_search_filter import TEXT

pytestmark = pytest.mark.gpu


def _check(gpu, a, b, ks, label=True):
    ctx = _lib.context()
    s = gpu.PairsBatch(a, b)
    for k in ks:
        want = oracle.pairs(a, b, k, threads=4)
        for dt in ("uint8", "uint16", "int32"):
            out = s.alloc(dt)
            for _ in range(3):                          # direct, captured, replayed
                s.run(out, max_dist=k)
            np.testing.assert_array_equal(out.get(), oracle.saturate(want, dt))
        np.testing.assert_array_equal(gpu.pairwise_packed(a, b, max_dist=k), want)


@pytest.mark.parametrize("n,lo,hi,alphabet", [(1, 40, 40, W.DNA), (31, 0, 8, W.DNA), (33, 30, 90, TEXT), (4097, 0, 40, TEXT),
                                              (5000, 33, 64, W.DNA), (3000, 8, 256, W.DNA_N), (300, 500, 2048, W.DNA),
                                              (40000, 33, 60, TEXT)])
def test_reach_pairs(gpu, n, lo, hi, alphabet):
    rng = np.random.default_rng(n + hi)
    a = W.random_strings(rng, rng.integers(lo, hi + 1, n), alphabet)
    b = W.mutate(rng, a, rng.uniform(0, 0.2, n), alphabet)
    _check(gpu, a, b, (0, 1, 2, 3, 5, 8, 9, 16))


def test_reach_pairs_shapes(gpu):
    """Equal, unrelated and empty strings, one side a prefix or suffix of the
    other, gaps of exactly k and k + 1, long pairs among short ones (a group
    whose span passes the stage)."""
    rng = np.random.default_rng(9)
    base = W.unpack(W.random_strings(rng, rng.integers(0, 120, 400)))
    long = W.unpack(W.random_strings(rng, [1900, 2000, 2048, 1500] * 8))
    a, b = [], []
    for i, x in enumerate(base):
        cut = int(rng.integers(0, 10))
        a.append(x)
        b.append([x, x[cut:], x[:len(x) - cut], x + b"A" * cut, b"", b"T" * cut + x, x[::-1], x[:cut] + x[cut + 3:]][i % 8])
        if i % 12 == 0:
            y = long[i // 12 % len(long)]
            a.append(y)
            b.append(y[:700] + y[703:1100] + b"G" + y[1100:])
    pack = lambda v: (np.frombuffer(b"".join(v), dtype=np.uint8).copy(), np.concatenate([[0], np.cumsum([len(x) for x in v])]).astype(np.int64))
    _check(gpu, pack(a), pack(b), (0, 1, 2, 3, 4, 7, 8, 9, 12))
    _check(gpu, pack(b), pack(a), (3, 8))


def test_reach_leaves_refused_lengths_to_the_other_path(gpu):
    """A pair of more than 2048 bytes after trimming stays refused; one that
    trims to less stays accepted."""
    rng = np.random.default_rng(2)
    x = W.unpack(W.random_strings(rng, [5000]))[0]
    near = x[:2500] + b"NN" + x[2500:]
    far = x[::-1]
    pack = lambda v: (np.frombuffer(v, dtype=np.uint8).copy(), np.array([0, len(v)], dtype=np.int64))
    assert gpu.pairwise_packed(pack(x), pack(near), max_dist=3)[0] == 2
    with pytest.raises(ValueError):
        gpu.pairwise_packed(pack(x), pack(far), max_dist=3)
