"""Which kernel a pairs run takes by its size, lengths and max_dist (blg_api.cu:
pairs_use_reach), on both sides of each limit, by the profile's labels. Results
are compared for equality on every route."""
import ctypes

import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_gpu_prefix import _labels
from test_search_filter import TEXT

pytestmark = pytest.mark.gpu


def _run(gpu, a, b, k, dtype="uint8"):
    s = gpu.PairsBatch(a, b)
    out = s.alloc(dtype)
    labels = _labels(_lib.context(), lambda: s.run(out, max_dist=k))
    np.testing.assert_array_equal(out.get(), oracle.saturate(oracle.pairs(a, b, k, threads=8), dtype))
    return labels


def _near(rng, n, lo, hi, alphabet, rate=0.05):
    a = W.random_strings(rng, rng.integers(lo, hi + 1, n), alphabet)
    return a, W.mutate(rng, a, rate, alphabet)


# words (the tile kernel from k = 3), near-copies of longer strings, many and few
@pytest.mark.parametrize("n,lo,hi,ks", [(5000, 4, 20, {2: True, 3: False}), (40000, 40, 60, {9: True, 10: False}),
                                        (1 << 15, 40, 60, {12: True, 17: False})])
def test_reach_limits(gpu, n, lo, hi, ks):
    a, b = _near(np.random.default_rng(n), n, lo, hi, W.DNA)
    for k, reach in ks.items():
        labels = _run(gpu, a, b, k)
        assert ("pairs_reach" in labels) == reach, (k, labels)
        assert not reach or "pairs_solve" in labels, labels       # the stage it is, beside the kernel


# what a sample finds unrelated among strings 64 bytes apart, strings too long for the
# stage, both sides of each limit
@pytest.mark.parametrize("n,lo,hi,related,ks", [(40000, 64, 64, False, {4: True, 5: False, 9: False}),
                                                (40000, 64, 64, True, {9: True, 10: False}),
                                                (40000, 128, 128, False, {3: True, 4: False}),
                                                (2000, 128, 128, False, {8: True, 9: False}),
                                                (2000, 64, 64, False, {12: True, 13: False}),
                                                (40000, 64, 72, False, {9: True, 10: False}),
                                                (2000, 63, 63, False, {16: True, 17: False}),
                                                (40000, 400, 420, True, {3: False}),
                                                (1000, 400, 420, True, {9: True, 10: False})])
def test_reach_leaves_what_it_would_slow_down(gpu, n, lo, hi, related, ks):
    rng = np.random.default_rng(n + lo)
    a, b = _near(rng, n, lo, hi, TEXT, 0.01)
    if not related:
        b = W.random_strings(rng, np.diff(a[1]), TEXT)
    for k, reach in ks.items():
        labels = _run(gpu, a, b, k)
        assert ("pairs_reach" in labels) == reach, (k, labels)
        np.testing.assert_array_equal(gpu.pairwise_packed(a, b, max_dist=k), oracle.pairs(a, b, k, threads=8))


# many pairs of another origin, or at most one in 50
@pytest.mark.parametrize("n,share,alphabet,bands", [(20000, 0.25, W.DNA, False), (20000, 0.0, W.DNA, True), (70000, 0.5, W.DNA, False),
                                                    (70000, 0.02, W.DNA, True), (70000, 0.1, TEXT, False), (70000, 0.0, TEXT, True),
                                                    (120000, 0.0, TEXT, False), (120000, 0.0, W.DNA, True)])
def test_bands_leave_mixed_sets(gpu, n, share, alphabet, bands):
    rng = np.random.default_rng(7)
    a, b = _near(rng, n, 60, 90, alphabet)
    other = np.flatnonzero(rng.random(n) < share)
    order = np.arange(n)
    order[other] += n
    b = W.take(W.concat(b, W.random_strings(rng, np.diff(a[1]), alphabet)), order)
    labels = _run(gpu, a, b, None, "int32")
    assert ("pairs_bands" in labels) == bands, labels


def test_reach_leaves_copies_that_share_all_banks(gpu):
    a = W.random_strings(np.random.default_rng(3), np.full(40000, 128))
    assert "pairs_reach" not in _run(gpu, a, a, 2)
