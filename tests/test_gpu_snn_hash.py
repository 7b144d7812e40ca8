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


def test_threads_with_other_list_lengths(sv):
    """Two contexts in two threads, long lists in one and short ones in the other: what a
    launch asks for in shared memory does not depend on what the other thread set."""
    import threading
    lists = {k: np.asfortranarray(np.random.default_rng(k).integers(1, 65, (64, k)).astype(np.int32))
             for k in (2, 1024)}
    errors = []

    def work(k):
        try:
            c = sv.Context(0)
            first = sv.jaccard_index(lists[k], k, ctx=c)
            for _ in range(400):
                G = sv.jaccard_index(lists[k], k, ctx=c)
                assert np.array_equal(G.indptr, first.indptr) and np.array_equal(G.data, first.data)
            c.close()
        except Exception as e:
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in (2, 1024, 2, 1024)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:2]
