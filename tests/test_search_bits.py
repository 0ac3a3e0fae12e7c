"""The exact search bit-sliced over queries (k_search_bits): 32 queries per
word, stripes of 64 rows, tiles of 1024 choices. Integer distances: every
comparison is for equality. On the CPU the cell, the stripes and the counts
(blg_bits.cuh) run against the oracle; on the GPU whole searches do."""
import ctypes

import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _build, _lib, workloads as W

BYTES = np.arange(256, dtype=np.uint8)
ALPHABETS = {"dna": W.DNA, "text": BYTES[32:96], "bytes": BYTES, "bytes255": BYTES[:255]}


@pytest.mark.parametrize("lengths", [[0], [1, 1], [7, 8, 9], [63, 64, 65], [0, 64, 128, 130], [255, 256, 257, 300],
                                     [512] * 3, list(range(1, 33))])
def test_bits_host(lengths):
    lib = ctypes.CDLL(_build.build_hostcheck())
    rng = np.random.default_rng(len(lengths) + lengths[-1])
    q = W.random_strings(rng, np.array(lengths))
    t = W.concat(W.random_strings(rng, [0, 1, 31, 64, 200, 511]), W.mutate(rng, W.take(q, [len(lengths) - 1] * 3), 0.1))
    want = oracle.cross(q, t, threads=1)
    for j in range(len(t[1]) - 1):
        out = np.zeros(len(lengths), np.int32)
        text = np.ascontiguousarray(t[0][t[1][j]:t[1][j + 1]])
        lib.blg_host_bits(q[0].ctypes.data_as(ctypes.c_void_p), q[1].ctypes.data_as(ctypes.c_void_p), len(lengths),
                          text.ctypes.data_as(ctypes.c_void_p), len(text), out.ctypes.data_as(ctypes.c_void_p))
        np.testing.assert_array_equal(out, want[:, j])


def _search(gpu, q, c, dtype="int32"):
    ctx = _lib.context()
    s = gpu.SearchBatch(q, c)
    out = s.alloc(dtype)
    ctx.check(ctx.lib.blg_profile_enable(ctx.h, 1))
    s.run(out)
    buf = ctypes.create_string_buffer(8192)
    ctx.check(ctx.lib.blg_profile_report(ctx.h, buf, 8192))
    ctx.check(ctx.lib.blg_profile_enable(ctx.h, 0))
    return out.get(), buf.value.decode()


# nq, nc, query lengths, choice lengths: partial groups and tiles, stripe and
# row-count edges, empty strings, one length and many, the longest queries
@pytest.mark.gpu
@pytest.mark.parametrize("alphabet", ["dna", "text"])
@pytest.mark.parametrize("nq,nc,ql,cl", [(33, 1025, (0, 9), (0, 12)), (97, 3000, (1, 64), (1, 64)),
                                         (70, 1500, (64, 64), (64, 64)), (65, 1024, (60, 70), (0, 300)),
                                         (130, 6000, (250, 258), (200, 256)), (300, 5000, (500, 512), (400, 600)),
                                         (200, 40000, (8, 30), (8, 30))])
def test_bits_search(gpu, alphabet, nq, nc, ql, cl):
    rng = np.random.default_rng(nq * 7 + nc)
    q = W.random_strings(rng, rng.integers(ql[0], ql[1] + 1, nq), ALPHABETS[alphabet])
    c = W.concat(W.random_strings(rng, rng.integers(cl[0], cl[1] + 1, nc - 20), ALPHABETS[alphabet]),
                 W.mutate(rng, W.take(q, rng.integers(0, nq, 20)), 0.1, ALPHABETS[alphabet]))
    want = oracle.cross(q, c, threads=8)
    for dt in ("int32", "uint16", "uint8"):
        got, labels = _search(gpu, q, c, dt)
        np.testing.assert_array_equal(got, oracle.saturate(want, dt))
        assert "search_bits" in labels, labels
    np.testing.assert_array_equal(gpu.cdist_packed(q, c), want)


# every byte value in the choices, 255 and 256 of them in the queries (256 have
# no room in the symbol map), queries past the sequential classes beside short ones
@pytest.mark.gpu
@pytest.mark.parametrize("alphabet,lo,hi", [("bytes255", 30, 90), ("bytes", 30, 90), ("dna", 1, 700)])
def test_bits_search_other_routes(gpu, alphabet, lo, hi):
    rng = np.random.default_rng(hi)
    q = W.random_strings(rng, rng.integers(lo, hi + 1, 70), ALPHABETS[alphabet])
    if alphabet == "bytes255":
        q = W.concat(q, (BYTES[:255].copy(), np.array([0, 85, 170, 255])))
    c = W.random_strings(rng, rng.integers(0, 200, 1100), BYTES)
    got, _ = _search(gpu, q, c)
    np.testing.assert_array_equal(got, oracle.cross(q, c, threads=8))
