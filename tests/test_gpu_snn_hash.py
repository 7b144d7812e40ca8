"""GPU: hashed SNN columns at the edges of their work split: lists of 1, 32, 33 and
70 neighbours (groups of 32 reverse lists), repeated neighbours (column sizes of
their own), columns of one warp, of one block and hubs in one graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,hub,dtype", [(900, 1, 0, np.float64), (1500, 32, 0, np.float32),
                                           (1500, 33, 40, np.float64), (2500, 70, 3, np.float32),
                                           (17000, 5, 2, np.float64)])
@pytest.mark.parametrize("kparam", ["k", "diag", "2k"])
def test_snn_hash_edges(sv, ctx, O, n, k, hub, dtype, kparam):
    rng = np.random.default_rng(n + k)
    idx = rng.integers(0, n, (n, k)).astype(np.int32)      # repeats within a list
    near = (np.arange(n)[:, None] + rng.integers(-k, k + 1, (n, k))) % n
    idx = np.where(rng.random((n, k)) < 0.8, near, idx).astype(np.int32)
    if hub:
        idx[:, 0] = rng.integers(0, hub, n)                # hubs: up to n / hub reverse neighbours
    kp = {"k": k, "diag": None, "2k": 2 * k}[kparam]
    W = sv.jaccard_index(idx + 1, kp, prune=1 / 15, dtype=dtype, ctx=ctx)
    R = O.jaccard_index(O.knn_graph(idx + 1, n), kp, 1 / 15, dtype)
    assert np.array_equal(W.indptr, R.indptr) and np.array_equal(W.indices, R.indices)
    assert np.array_equal(W.data, R.data) and W.data.dtype == R.data.dtype
