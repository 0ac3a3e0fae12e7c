"""The paths that a run takes when a device list runs full, and the kernels that
larger or rarer calls than the other tests' still reach, each held by the
profile's labels: the filter whose solver goes on with the fill (its results
listed, its repair), the survivor kernel's own list and repair, row chunks of a
one-call filtered search, the banded pairs solver over chunks of different
alphabets. Every run twice on one context, so counters that are not cleared show."""
import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_gpu_prefix import _labels
from test_search_filter import _run, _sets

pytestmark = pytest.mark.gpu


def _copies(nq, nc, copies, length=64):
    """nq equal queries; choices: `copies` more of them, none where the sample of the
    choices looks (every nc / 64th), the rest unrelated. (queries, choices, is a copy)"""
    rng = np.random.default_rng(copies)
    one = W.random_strings(rng, [length])
    assert nc % 64 == 0
    free = np.flatnonzero(np.arange(nc) % (nc // 64) != 0)
    at = rng.choice(free, copies, replace=False)
    c = W.random_strings(rng, np.full(nc, length))
    c[0].reshape(nc, length)[at] = one[0]
    same = np.zeros(nc, bool)
    same[at] = True
    return W.take(one, np.zeros(nq, dtype=np.int64)), c, same


# results: listed and scattered; more results than their list holds; more passers than theirs
@pytest.mark.parametrize("copies", [300, 768, 2304])
def test_deferred_filter_lists(gpu, copies):
    nq, nc = 2048, 49152                                      # 400 MB of output: longer to write than to filter
    q, c, same = _copies(nq, nc, copies)
    s = gpu.SearchBatch(q, c)
    out = s.alloc("int32")
    want = np.where(same, 0, 3)
    for rep in range(2):
        got, labels = _run(gpu, s, out, 2)
        assert "filter_pairs" in labels and "solve_finish" in labels, labels
        assert (got == want).all(), rep
        _lib.context().check(_lib.context().lib.blg_memset(_lib.context().h, out.ptr, 0x55, nq * nc * 4))
    qi, ci, d = s.matches(2)                                  # the same lists without an output
    assert len(qi) == nq * copies and (d == 0).all()
    np.testing.assert_array_equal(ci[:copies], np.flatnonzero(same))
    np.testing.assert_array_equal(qi, np.repeat(np.arange(nq), copies))


# the survivor kernel's list (max_dist past the filter's), over 4 M pairs
@pytest.mark.parametrize("dtype", ["uint8", "uint16", "int32"])
def test_survivor_list_and_repair(gpu, dtype):
    q, c, same = _copies(2200, 2240, 1500)
    s = gpu.SearchBatch(q, c)
    out = s.alloc(dtype)
    row = oracle.saturate(oracle.cross(W.take(q, [0]), c, 20), dtype)[0]
    assert (row[same] == 0).all() and (row[~same] == 21).all()
    for rep in range(2):
        got, labels = _run(gpu, s, out, 20)
        assert "search_band " in labels and "search_small" not in labels and "filter_pairs" not in labels, labels
        np.testing.assert_array_equal(got, np.broadcast_to(row, got.shape))


def test_survivor_list_against_oracle(gpu):
    rng = np.random.default_rng(17)
    q, c = _sets(rng, 80, 60007, 40, 60, W.DNA)
    s = gpu.SearchBatch(q, c)
    got, labels = _run(gpu, s, s.alloc("uint16"), 16)
    assert "search_band " in labels and "search_small" not in labels and "filter_pairs" not in labels, labels
    np.testing.assert_array_equal(got, oracle.cross(q, c, 16, threads=16))


def test_filter_runs_in_one_call_chunks(gpu):
    rng = np.random.default_rng(22)
    q, c = _sets(rng, 701, 100003, 64, 64, W.DNA)
    got = []
    labels = _labels(_lib.context(), lambda: got.append(gpu.cdist_packed(q, c, max_dist=2, dtype="uint8")))
    assert "filter_pairs" in labels, labels
    rows = np.arange(0, 701, 23)
    np.testing.assert_array_equal(got[0][rows], oracle.saturate(oracle.cross(W.take(q, rows), c, 2, threads=16), "uint8"))


def test_banded_pairs_over_chunks_of_two_alphabets(gpu):
    rng = np.random.default_rng(23)
    sets = [W.random_strings(rng, rng.integers(1, 120, n), al) for n, al in
            ((1 << 17, W.DNA), ((1 << 17) + 5, np.arange(20, 220, dtype=np.uint8)))]
    near = [W.mutate(rng, x, 0.08, al) for x, al in zip(sets, (W.DNA, np.arange(20, 220, dtype=np.uint8)))]
    a, b = W.concat(*sets), W.concat(*near)
    got = []
    labels = _labels(_lib.context(), lambda: got.append(gpu.pairwise_packed(a, b, max_dist=12, dtype="uint8")))
    assert "pairs_band" in labels, labels
    np.testing.assert_array_equal(got[0], oracle.saturate(oracle.pairs(a, b, 12, threads=16), "uint8"))
