"""GPU: a context's device memory is reused between calls, given back with the
context, and handles may outlive it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pool_is_given_back_with_the_context(sv, ctx, O):
    X = O.synth_counts(400, 300, -1.0, 1.5, depth=0.5, seed=3)
    free0, total = ctx.memory()
    c = sv.Context(0)
    big = sv.CountMatrix.generate(20000, 4000, np.ones(4000), np.ones(20000), seed=1, ctx=c)
    nbytes = 16 * big.nnz
    assert nbytes > 256 << 20
    del big
    kept = free0 - ctx.memory()[0]
    assert kept <= total // 16 + nbytes // 4        # bounded while the context lives
    held = sv.CountMatrix.from_csc(X, ctx=c)
    c.close()
    assert free0 - ctx.memory()[0] < nbytes // 4    # and given back with it
    held.h, h = None, held.h                        # a handle freed after its context
    assert c.lib.sv_counts_free(h) == 0


def test_handles_freed_on_another_thread(sv, O):
    X = O.synth_counts(300, 200, -1.0, 1.5, depth=0.5, seed=5)
    c = sv.Context(0)
    ref = sv.normalize_cells(sv.CountMatrix.from_csc(X, ctx=c), scale_factor=1e4).values_csc()
    for _ in range(20):
        d = sv.normalize_cells(sv.CountMatrix.from_csc(X, ctx=c), scale_factor=1e4)
        got = d.values_csc()
        box = [d]
        del d
        t = threading.Thread(target=box.clear)
        t.start()
        t.join()
        assert np.array_equal(got, ref)
    c.close()
