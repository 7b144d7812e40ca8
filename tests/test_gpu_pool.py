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


@pytest.mark.parametrize("genes,mu", [(200, 1.0), (8000, 20.0)])      # blocks of the pool, and larger ones
def test_handles_freed_while_the_stream_is_captured(sv, genes, mu):
    """Blocks that another thread frees during a capture wait for its end: the graph holds
    what was captured and nothing else, and the memory is given back afterwards."""
    import ctypes as C
    c = sv.Context(0)
    cells = 200000
    free0, total = c.memory()
    pair = [sv.CountMatrix.generate(cells, genes, np.full(genes, mu), np.ones(cells), seed=s, ctx=c) for s in (1, 2)]
    assert (4 * pair[0].nnz > total // 64) == (genes == 8000)
    h = [p.h for p in pair]
    for p in pair:
        p.h = None
    nodes = C.c_int64()
    sv._lib.check(c.lib.sv_selftest_free_in_capture(c.h, h[0], h[1], C.byref(nodes)))
    assert nodes.value == 1
    assert free0 - c.memory()[0] <= total // 16 + (256 << 20)
    X = sv.CountMatrix.generate(3000, 2000, np.ones(2000), np.ones(3000), seed=3, ctx=c)   # the context goes on
    D = sv.normalize_cells(X, scale_factor=1e4, dtype="float32")
    em = sv.pca(sv.scale_features(D, scale_max=10.0), 5)
    assert np.all(np.isfinite(em.coordinates))
    c.close()
    d = sv.Context(0)
    assert free0 - d.memory()[0] <= 256 << 20
    d.close()


def _fill(nbytes):
    import torch
    return torch.empty(nbytes, dtype=torch.uint8, device="cuda")


def test_kept_memory_is_there_for_others(sv):
    """What a context keeps between calls goes back to the device when it is trimmed, and
    when another context has no memory left."""
    import torch
    torch.cuda.empty_cache()
    a, b = sv.Context(0), sv.Context(0)
    n, genes = 400000, 2000

    def make(c):
        return sv.CountMatrix.generate(n, genes, np.full(genes, 3.0), np.ones(n), seed=1, ctx=c)

    free0 = a.memory()[0]
    nbytes = 16 * make(a).nnz                       # 10 GB in blocks of the pool, dropped at once
    kept = free0 - a.memory()[0]
    assert kept > nbytes // 2
    a.trim()
    assert free0 - a.memory()[0] < 256 << 20
    make(a)
    fill = _fill(a.memory()[0] - nbytes // 2)       # half of it besides what a keeps
    try:
        assert make(b).nnz * 16 == nbytes
    finally:
        del fill
        torch.cuda.empty_cache()
        a.close()
        b.close()
