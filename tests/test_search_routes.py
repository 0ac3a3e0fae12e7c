"""Which kernel a thresholded search takes by its size, lengths and data
(blg_api.cu: search_small, filter_plan), by the profile's labels, and the dense
output and result list of each. Results are compared for equality."""
import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_gpu_prefix import _labels
from test_search_filter import TEXT, _run, _sets

pytestmark = pytest.mark.gpu


def _families(rng, nq, nc, length, families, rate=0.08, alphabet=W.DNA):
    """Every string a mutant of one of some stems, cut or filled to one length."""
    stems = W.random_strings(rng, np.full(families, length), alphabet)
    fix = lambda p: (np.concatenate([np.resize(np.append(p[0][p[1][i]:p[1][i + 1]], alphabet[0]), length)
                                     for i in range(len(p[1]) - 1)]), np.arange(len(p[1])) * length)
    return tuple(fix(W.mutate(rng, W.take(stems, rng.integers(0, families, n)), rate, alphabet)) for n in (nq, nc))


# one launch or the survivor kernel: pairs in all, columns within the window, k
@pytest.mark.parametrize("nq,nc,length,ks", [(64, 20000, 64, {1: True, 2: False, 3: False}), (16, 30000, 64, {2: True, 3: True}),
                                             (64, 40000, 8, {1: True}), (64, 28000, 80, {0: False})])
def test_small_search_limits(gpu, nq, nc, length, ks):
    q, c = _families(np.random.default_rng(nq + nc), nq, nc, length, 16)
    s = gpu.SearchBatch(q, c)
    for k, small in ks.items():
        got, labels = _run(gpu, s, s.alloc("uint8"), k)
        assert ("search_small" in labels) == small, (k, labels)
        np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, k, threads=8), "uint8"))


# strings of a few families pass the 4-gram test by the million
@pytest.mark.parametrize("length,families,k,filtered", [(64, 2, 6, False), (64, 8, 5, True), (100, 8, 6, False),
                                                        (100, 400, 2, True), (64, 5000, 4, True)])
def test_filter_leaves_related_strings(gpu, length, families, k, filtered):
    q, c = _families(np.random.default_rng(families), 600, 20000, length, families, 0.02)
    s = gpu.SearchBatch(q, c)
    want = oracle.saturate(oracle.cross(q, c, k, threads=8), "uint8")
    got, labels = _run(gpu, s, s.alloc("uint8"), k)
    assert ("filter_pairs" in labels) == filtered, labels
    np.testing.assert_array_equal(got, want)
    qi, ci, d = s.matches(k)
    wi, wj = np.nonzero(want <= k)
    np.testing.assert_array_equal(qi, wi)
    np.testing.assert_array_equal(ci, wj)
    np.testing.assert_array_equal(d, want[wi, wj])


def test_filter_longest_queries(gpu):
    """Queries of 512 bytes, the most that a slot of the filter's solver holds, and
    choices up to max_dist longer, starting at every byte of a 16-byte line."""
    rng = np.random.default_rng(9)
    q = W.random_strings(rng, rng.integers(509, 513, 130), TEXT)
    c = W.concat(W.mutate(rng, W.take(q, rng.integers(0, 130, 2000)), rng.uniform(0, 0.012, 2000), TEXT),
                 W.random_strings(rng, rng.integers(506, 516, 28000), TEXT))
    c = W.take(c, rng.permutation(30000))
    s = gpu.SearchBatch(q, c)
    got, labels = _run(gpu, s, s.alloc("uint8"), 3)
    assert "filter_pairs" in labels, labels
    np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, 3, threads=16), "uint8"))
    assert set(np.unique(got)) == {0, 1, 2, 3, 4}


# work units of 1024, 512, 256 and 128 survivors, a last one partly full, beside an uneven problem
@pytest.mark.parametrize("nq,nc", [(400, 13007), (300, 10001), (100, 15003), (10, 2005)])
def test_batch_unit_sizes(gpu, nq, nc):
    rng = np.random.default_rng(nq)
    probs = [_sets(rng, nq, nc, 64, 64, W.DNA) + (2, "uint8"), _sets(rng, 3, 701, 10, 90, TEXT) + (7, "uint16")]
    b = gpu.ProblemBatch(probs)
    for rep in range(2):
        for got, (q, c, k, dt) in zip([o.get() for o in b.run()], probs):
            np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, k, threads=16), dt))


# unrelated strings: none passes the 4-gram test, or so many that nothing is left to pack
@pytest.mark.parametrize("nq,nc,lo,hi,k,small", [(40, 25001, 64, 64, 3, True), (132, 17251, 42, 42, 6, True),
                                                 (154, 10409, 106, 201, 8, True), (40, 25001, 64, 64, 6, False)])
def test_small_search_of_unrelated_strings(gpu, nq, nc, lo, hi, k, small):
    rng = np.random.default_rng(nq)
    q, c = (W.random_strings(rng, rng.integers(lo, hi + 1, n)) for n in (nq, nc))
    s = gpu.SearchBatch(q, c)
    got, labels = _run(gpu, s, s.alloc("uint8"), k)
    assert ("search_small" in labels) == small, labels
    np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, k, threads=8), "uint8"))


def test_filter_counts_passers_within_the_window(gpu):
    """Short strings pass the 4-gram test whatever their lengths' difference; only those
    within it are solved."""
    rng = np.random.default_rng(5)
    q, c = (W.random_strings(rng, rng.integers(38, 174, n)) for n in (379, 123334))
    got = []
    labels = _labels(_lib.context(), lambda: got.append(gpu.cdist_matches_packed(q, c, 6)))
    assert "filter_pairs" in labels, labels
    wi, wj = np.nonzero(oracle.cross(q, c, 6, threads=8) <= 6)
    np.testing.assert_array_equal(got[0][0], wi)
    np.testing.assert_array_equal(got[0][1], wj)


# a few of the pairs pass, or most of a window that holds all of them: texts
@pytest.mark.parametrize("nq,nc,length,k", [(231, 15976, 34, 5), (179, 17754, 85, 12)])
def test_small_search_of_unrelated_texts(gpu, nq, nc, length, k):
    rng = np.random.default_rng(k)
    q, c = (W.random_strings(rng, np.full(n, length), TEXT) for n in (nq, nc))
    s = gpu.SearchBatch(q, c)
    got, labels = _run(gpu, s, s.alloc("uint8"), k)
    assert "search_small" in labels, labels
    np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, k, threads=8), "uint8"))
