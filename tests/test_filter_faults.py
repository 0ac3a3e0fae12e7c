"""The tensor-core filter's bounded waits cut short: whatever role gives up first,
the kernel ends, the call reports the timeout, and the context stays usable.
Every lane of a warp has to leave the loop together, since TMEM loads, votes and
shuffles follow its waits. No test here faults, traps or hangs a GPU."""
import numpy as np
import pytest

import oracle
from editdist_bench_gb300 import _lib, workloads as W
from test_search_filter import _run, _sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [0, 1, 2, 5, 20])
@pytest.mark.parametrize("nq,nc,length,k", [(900, 20003, 64, 2), (1000, 5001, 64, 0)])      # whole and folded rows
def test_filter_wait_timeout_is_reported_and_recoverable(gpu, nq, nc, length, k, polls):
    ctx = _lib.context()
    rng = np.random.default_rng(nq + k)
    q, c = _sets(rng, nq, nc, length, length, W.DNA)
    want = oracle.saturate(oracle.cross(q, c, k, threads=8), "uint8")
    s = gpu.SearchBatch(q, c)
    out = s.alloc("uint8")
    try:
        ctx.check(ctx.lib.blg_set_fault_injection(ctx.h, -1, polls))
        for call in (lambda: (s.run(out, max_dist=k), gpu.synchronize(), out.get())[2],
                     lambda: gpu.cdist_packed(q, c, max_dist=k, dtype="uint8")):
            if polls == 0:
                with pytest.raises(RuntimeError, match="timed out"):
                    call()
                continue
            try:                                   # a few polls may be enough: then the result is right
                np.testing.assert_array_equal(call(), want)
            except RuntimeError as e:
                assert "timed out" in str(e)
    finally:
        ctx.check(ctx.lib.blg_set_fault_injection(ctx.h, -1, -1))
    got, labels = _run(gpu, s, out, k)
    assert "filter_pairs" in labels, labels
    np.testing.assert_array_equal(got, want)
