"""GPU: calls whose extra device memory only makes them faster -- the table of the small
counts' values, the arena of the kept SNN entries, the neighbour search's tile lists --
do without it where the device has no room for it."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def c(sv, ctx):
    """A context of its own, and nothing kept by others that an allocation could have."""
    gc.collect()
    c = sv.Context(0)
    c.others = [ctx, sv.default_context()]
    yield c
    c.close()


class _Room:
    """All of the device's memory but `nbytes` taken."""
    def __init__(self, c, nbytes):
        self.c, self.nbytes = c, nbytes

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        for c in [self.c] + self.c.others:
            c.trim()
        self.fill = torch.empty(self.c.memory()[0] - self.nbytes, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        import torch
        self.fill = None
        torch.cuda.empty_cache()


def _kernels(c, call):
    c.profile_reset()
    c.profile(True)
    out = call()
    c.profile(False)
    return out, c.profile_report()


def test_normalize_without_a_table(sv, c):
    n, genes = 2000000, 300
    X = sv.CountMatrix.generate(n, genes, np.full(genes, 1.0), np.ones(n), seed=1, ctx=c)
    assert X.nnz >= 64 * n
    ref = sv.normalize_cells(X, scale_factor=1e4, dtype="float32").values_csc()
    need, table = 2 * 4 * X.nnz + 8 * n, 32 * 4 * n
    with _Room(c, need + table // 2 + (64 << 20)):
        got = sv.normalize_cells(X, scale_factor=1e4, dtype="float32")
        assert c.memory()[0] < table                # no room for it
    assert np.array_equal(got.values_csc(), ref)


def _sweep(sv, c, call, same, rooms, extra, first):
    """call() in less and less room, until there is too little for the call itself: whether
    one of the runs did without the kernel `extra`, or began again without it (then others
    ran more often than the `first` time)."""
    without = False
    for mb in rooms:
        with _Room(c, mb << 20):
            try:
                out, kernels = _kernels(c, call)
            except sv._lib.SeveroGPUError as e:
                assert e.code == sv._lib.SV_ERR_OOM
                return without
        assert same(out)
        without |= extra not in kernels or any(kernels[k][0] > first[k][0] for k in first)
    return without


@pytest.mark.parametrize("precision,rooms", [("fp32", range(4096, 512, -384)), ("bf16", range(1536, 256, -96))])
def test_neighbours_without_lists(sv, c, precision, rooms):
    n = 1000000
    rng = np.random.default_rng(1)
    X = (8 * rng.standard_normal((50, 8)))[rng.integers(0, 50, n)] + rng.standard_normal((n, 8))
    X = np.asfortranarray(X.astype(np.float32))

    def call():
        return sv.ann(X, 10, precision=precision, ctx=c)

    (idx, dist), kernels = _kernels(c, call)
    assert "knn_tile_lists" in kernels
    assert _sweep(sv, c, call, lambda out: np.array_equal(out[1], dist), rooms, "knn_tile_lists", kernels)


def test_snn_without_an_arena(sv, c):
    n, k = 150000, 30
    rng = np.random.default_rng(2)
    nn = (np.arange(n)[:, None] // 200 * 200 + rng.integers(0, 200, (n, k))) % n + 1
    nn = np.asfortranarray(nn.astype(np.int32))

    def call():
        return sv.jaccard_index(nn, k, ctx=c)

    def same(G):
        return (np.array_equal(G.indptr, ref.indptr) and np.array_equal(G.indices, ref.indices) and
                np.array_equal(G.data, ref.data))

    ref, kernels = _kernels(c, call)
    assert "snn_emit" in kernels
    assert _sweep(sv, c, call, same, range(1024, 64, -32), "snn_emit", kernels)
