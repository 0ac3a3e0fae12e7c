"""Which kernel an exact search takes (blg_api.cu: bits_applies, class_prefix):
where the bit-sliced one cannot run, the prefix layout that was built for the
search is used, and a chunk of a one-call search is not taken for a search of 33
to 64 queries. Results are compared for equality on every route."""
import ctypes

import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_gpu_prefix import _labels, _stemmed_choices

pytestmark = pytest.mark.gpu


def _run(gpu, q, c):
    s = gpu.SearchBatch(q, c)
    out = s.alloc("int32")
    labels = _labels(_lib.context(), lambda: s.run(out))
    np.testing.assert_array_equal(out.get(), oracle.cross(q, c, threads=8))
    return labels


def test_prefix_layout_where_the_symbol_table_is_too_large(gpu):
    """250 different bytes in queries of up to 512: no room for the bit-sliced table."""
    rng = np.random.default_rng(1)
    al = np.arange(250, dtype=np.uint8)
    q = W.concat(W.random_strings(rng, rng.integers(1, 128, 300), al), W.random_strings(rng, [512, 500], al))
    c = _stemmed_choices(rng, 5000, 40, 30)
    labels = _run(gpu, q, c)
    assert "search_pfx" in labels and "search_bits" not in labels, labels


# a wave of units on every SM partition and a few more, equal and mixed lengths,
# one query among a group's 32
@pytest.mark.parametrize("nq,nc,lo,hi", [(100, 5000, 64, 64), (32, 20000, 100, 128), (65, 5000, 100, 128),
                                         (4, 40000, 16, 256), (33, 20000, 250, 256), (1, 65536, 16, 256)])
def test_exact_routes_agree(gpu, nq, nc, lo, hi):
    rng = np.random.default_rng(nq)
    q, c = (W.random_strings(rng, rng.integers(lo, hi + 1, n)) for n in (nq, nc))
    labels = _run(gpu, q, c)
    if (lo, hi) in ((64, 64), (100, 128)):     # 52 us bit-sliced, 104 with prefixes, 165 word by word; 175 / 371 / 443
        assert "search_bits" in labels, labels
    if nq == 4:                                # 850 us bit-sliced, 1215 with prefixes, 510 word by word
        assert "search_tt" in labels and "search_bits" not in labels, labels


def test_chunks_of_a_larger_search(gpu):
    """400 queries in one call run in chunks of 50 and fewer."""
    rng = np.random.default_rng(2)
    q, c = W.random_strings(rng, np.full(400, 40)), W.random_strings(rng, np.full(1 << 17, 40))
    got = []
    labels = _labels(_lib.context(), lambda: got.append(gpu.cdist_packed(q, c, dtype="uint16")))
    assert "search_bits" in labels and "search_pfx" not in labels, labels
    rows = np.arange(0, 400, 37)
    np.testing.assert_array_equal(got[0][rows], oracle.saturate(oracle.cross(W.take(q, rows), c, threads=8), "uint16"))


# choices that share most of their columns, queries past the prefix kernel's two words
# alone and beside short ones
@pytest.mark.parametrize("nq,lo,hi", [(300, 150, 256), (300, 129, 129), (300, 60, 256), (300, 64, 128)])
def test_long_queries_beside_shared_prefixes(gpu, nq, lo, hi):
    rng = np.random.default_rng(lo)
    q = W.random_strings(rng, rng.integers(lo, hi + 1, nq))
    c, off = W.random_strings(rng, np.full(9001, 64))
    c.reshape(-1, 64)[:, :48] = rng.choice(W.DNA, (40, 48))[rng.integers(0, 40, 9001)]
    labels = _run(gpu, q, (c, off))
    if lo > 128:
        assert "search_bits" in labels and "search_pfx" not in labels, labels
    if hi <= 128:
        assert "search_pfx" in labels and "search_bits" not in labels, labels


# one call: the choices are sorted only where that takes less than it saves
@pytest.mark.parametrize("nq,nc,stem,symbols,pfx", [(100, 8001, 0, 4, False), (100, 8001, 48, 4, False), (64, 8001, 0, 4, False),
                                                    (4000, 8001, 60, 4, True), (4000, 8001, 0, 4, False),
                                                    (300, 8001, 48, 250, True), (2000, 8001, 48, 250, True)])
def test_one_call_sorts_where_it_pays(gpu, nq, nc, stem, symbols, pfx):
    rng = np.random.default_rng(nq + stem)
    q = W.random_strings(rng, rng.integers(100, 129, nq), np.arange(symbols, dtype=np.uint8) if symbols > 4 else W.DNA)
    if symbols > 4:                                # a table too large for the bit-sliced kernel
        q = W.concat(q, W.random_strings(rng, [512], np.arange(symbols, dtype=np.uint8)))
    c, off = W.random_strings(rng, np.full(nc, 64))
    c.reshape(-1, 64)[:, :stem] = rng.choice(W.DNA, (40, stem))[rng.integers(0, 40, nc)]
    got = []
    labels = _labels(_lib.context(), lambda: got.append(gpu.cdist_packed(q, (c, off), dtype="uint8")))
    assert ("search_pfx" in labels) == ("prefix_text" in labels) == pfx, labels
    rows = np.unique(np.append(np.arange(0, nq, 1 + nq // 40), len(q[1]) - 2))
    np.testing.assert_array_equal(got[0][rows], oracle.saturate(oracle.cross(W.take(q, rows), (c, off), threads=8), "uint8"))
