"""Layouts that a search runs without: where the device has no room for them, or needs
theirs, the search is uploaded and runs all the same, on the kernels that need
none. The failures are made on the host (blg_set_fault_injection)."""
import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_search_filter import TEXT, _run

pytestmark = pytest.mark.gpu


def _inject(what):
    ctx = _lib.context()
    ctx.check(ctx.lib.blg_set_fault_injection(ctx.h, what, -1))


def _exact(gpu, s, want):
    out = s.alloc("int32")
    got, labels = _run(gpu, s, out, None)
    np.testing.assert_array_equal(got, want)
    return "search_bits" in labels


def _near(gpu, s, k, rows, want):
    got, labels = _run(gpu, s, s.alloc("uint8"), k)
    np.testing.assert_array_equal(got[rows], want)
    return "filter_pairs" in labels


@pytest.mark.parametrize("fault", [-2, -3])
def test_searches_run_without_their_spares(gpu, fault):
    rng = np.random.default_rng(31)
    q, c = W.random_strings(rng, np.full(80, 100)), W.random_strings(rng, np.full(9000, 100))    # two stripes
    want = oracle.cross(q, c, threads=16)
    big_q = W.random_strings(rng, np.full(16, 24), TEXT)
    big_c = W.random_strings(rng, np.full(2200000, 24), TEXT)                                    # 70 MB of signatures
    rows = [0, 15]
    big_want = oracle.saturate(oracle.cross(W.take(big_q, rows), big_c, 1, threads=16), "uint8")
    try:
        if fault == -2:
            _inject(-2)
        s, t = gpu.SearchBatch(q, c), gpu.SearchBatch(big_q, big_c)
        if fault == -3:                                   # there to begin with, given back for another's sake
            assert _exact(gpu, s, want) and _near(gpu, t, 1, rows, big_want)
            _inject(-3)
        assert not _exact(gpu, s, want)
        assert not _near(gpu, t, 1, rows, big_want)
        np.testing.assert_array_equal(gpu.cdist_packed(q, c), want)
    finally:
        _inject(-1)
    if fault == -2:                                       # the stripes' room alone came too late
        u = gpu.SearchBatch(q, c)
        _inject(-2)
        try:
            assert not _exact(gpu, u, want)
        finally:
            _inject(-1)
        assert _exact(gpu, u, want)
