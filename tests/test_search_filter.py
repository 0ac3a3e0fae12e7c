"""The tensor-core filter of thresholded searches (k_filter_pairs,
k_solve_passers): signatures, the sign of their product, whole searches.
Distances are integers: every comparison is for equality."""
import ctypes

import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _build, _lib, workloads as W

TEXT = np.arange(32, 96, dtype=np.uint8)


def test_signature_sum():
    """The sum is (|X & Y| / 2 - ...) + 1/8 exactly, so its sign is |X ^ Y| <=
    8 k; no pair within k is ruled out; rows without a string never pass."""
    lib = ctypes.CDLL(_build.build_hostcheck())
    lib.blg_host_sig_sum.restype = ctypes.c_float
    rng = np.random.default_rng(5)
    d = ctypes.c_int()
    for alphabet in (W.DNA, TEXT, np.arange(256, dtype=np.uint8)):
        for n in (0, 1, 3, 4, 5, 9, 33, 64, 200, 600):
            x = W.random_strings(rng, np.full(6, n), alphabet)
            y = W.concat(W.mutate(rng, x, rng.uniform(0, 0.2, 6), alphabet), W.random_strings(rng, np.full(3, n), alphabet))
            want = oracle.cross(x, y, threads=1)
            for i in range(6):
                a = x[0][x[1][i]:x[1][i + 1]].tobytes()
                for j in range(9):
                    b = y[0][y[1][j]:y[1][j + 1]].tobytes()
                    for k in (0, 1, 2, 7, 15):
                        for half in (0, 4):
                            s = lib.blg_host_sig_sum(a, len(a), b, len(b), k, 3 + half, ctypes.byref(d))
                            assert s == (8 * k - d.value) / 4 + 0.125
                            assert s >= 0 or want[i, j] > k
                        for v in (0, 1, 2, 4, 5, 6):
                            assert lib.blg_host_sig_sum(a, len(a), b, len(b), k, v, ctypes.byref(d)) < 0


def _run(gpu, s, out, k):
    ctx = _lib.context()
    ctx.check(ctx.lib.blg_profile_enable(ctx.h, 1))
    s.run(out, max_dist=k)
    buf = ctypes.create_string_buffer(8192)
    ctx.check(ctx.lib.blg_profile_report(ctx.h, buf, 8192))
    ctx.check(ctx.lib.blg_profile_enable(ctx.h, 0))
    return out.get(), buf.value.decode()


def _sets(rng, nq, nc, lo, hi, alphabet, rate=0.06):
    q = W.random_strings(rng, rng.integers(lo, hi + 1, nq), alphabet)
    near = W.mutate(rng, W.take(q, rng.integers(0, nq, nc // 20)), rng.uniform(0, rate, nc // 20), alphabet)
    c = W.concat(near, W.random_strings(rng, rng.integers(lo, hi + 1, nc - nc // 20), alphabet))
    return q, W.take(c, rng.permutation(nc))


# partial query and choice tiles, one word class and several, one length and
# many, the smallest and largest k, odd row sizes
@pytest.mark.gpu
@pytest.mark.parametrize("nq,nc,lo,hi,alphabet,k", [(128, 32768, 64, 64, "dna", 2), (900, 5001, 64, 64, "dna", 0),
                                                    (257, 20003, 50, 80, "dna", 4), (1000, 20001, 100, 140, "dna", 3),
                                                    (260, 16001, 172, 172, "text", 13), (129, 32001, 18, 18, "text", 1),
                                                    (600, 30011, 20, 60, "text", 2)])
def test_filter_search(gpu, nq, nc, lo, hi, alphabet, k):
    rng = np.random.default_rng(nq + nc + k)
    al = W.DNA if alphabet == "dna" else TEXT
    q, c = _sets(rng, nq, nc, lo, hi, al)
    want = oracle.cross(q, c, k, threads=8)
    s = gpu.SearchBatch(q, c)
    for dt in ("uint8", "uint16", "int32"):
        got, labels = _run(gpu, s, s.alloc(dt), k)
        np.testing.assert_array_equal(got, oracle.saturate(want, dt))
        assert "filter_pairs" in labels, labels
    qi, ci, d = s.matches(k)
    wi, wj = np.nonzero(want <= k)
    np.testing.assert_array_equal(qi, wi)
    np.testing.assert_array_equal(ci, wj)
    np.testing.assert_array_equal(d, want[wi, wj])


@pytest.mark.gpu
def test_filter_short_and_empty_strings(gpu):
    """Queries and choices without a single 4-gram beside long ones."""
    rng = np.random.default_rng(8)
    q, c = _sets(rng, 500, 12000, 64, 70, W.DNA)
    q = W.concat(q, W.random_strings(rng, [0, 0, 1, 2, 3, 4, 5]))
    c = W.concat(c, W.random_strings(rng, [0, 1, 1, 2, 3, 3, 4, 6] * 3))
    s = gpu.SearchBatch(q, c)
    got, labels = _run(gpu, s, s.alloc("uint8"), 2)
    assert "filter_pairs" in labels, labels
    np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, 2, threads=8), "uint8"))


@pytest.mark.gpu
def test_filter_list_overflow(gpu):
    """2200 x 2200 equal strings: every pair passes, more than the list holds."""
    one = W.random_strings(np.random.default_rng(3), [64])
    x = W.take(one, np.zeros(2200, dtype=np.int64))
    y = W.concat(x, W.random_strings(np.random.default_rng(4), [64] * 5))
    s = gpu.SearchBatch(x, y)
    got, labels = _run(gpu, s, s.alloc("uint8"), 2)
    assert "filter_pairs" in labels, labels
    assert (got[:, :2200] == 0).all() and (got[:, 2200:] == 3).all()
    qi, ci, d = s.matches(2)
    assert len(qi) == 2200 * 2200 and (d == 0).all()


@pytest.mark.gpu
def test_filter_one_call_chunks(gpu):
    """Row chunks of a one-call search start anywhere: the fill's ends are
    written element by element."""
    rng = np.random.default_rng(21)
    q, c = _sets(rng, 701, 100003, 64, 64, W.DNA)
    got = gpu.cdist_packed(q, c, max_dist=2, dtype="uint8")
    np.testing.assert_array_equal(got, oracle.saturate(oracle.cross(q, c, 2, threads=16), "uint8"))


# one launch for small searches (k_search_small): a lone query, several word
# classes, empty strings on both sides, every length window from none to all
@pytest.mark.gpu
@pytest.mark.parametrize("nq,nc,lo,hi,k", [(1, 1, 5, 5, 1), (1, 20011, 3, 16, 2), (3, 129, 0, 3, 0), (40, 3000, 0, 40, 3),
                                           (70, 5000, 1, 300, 31), (9, 1000, 500, 530, 9)])
def test_small_search(gpu, nq, nc, lo, hi, k):
    rng = np.random.default_rng(nq + nc)
    q, c = _sets(rng, nq, max(nc, 20), lo, hi, TEXT, 0.2)
    c = W.take(c, np.arange(nc))
    want = oracle.cross(q, c, k, threads=4)
    s = gpu.SearchBatch(q, c)
    for dt in ("uint8", "uint16", "int32"):
        got, labels = _run(gpu, s, s.alloc(dt), k)
        np.testing.assert_array_equal(got, oracle.saturate(want, dt))
        assert "search_small" in labels, labels
    np.testing.assert_array_equal(gpu.cdist_packed(q, c, max_dist=k), want)
