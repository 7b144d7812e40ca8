"""GPU: the tensor-core neighbour search over cells of pivots returns what a scan of
all tiles returns -- the halves of the tiles, which its shortlists are made of, stay
those of the order along the widest dimension -- at the smallest sizes, with last
tiles of one half, of one point and of all but one, with equal points and with
points that no bound holds for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, d, kind):
    rng = np.random.default_rng(n + d)
    if kind == "clusters":
        X = rng.normal(0, 5, (30, d))[rng.integers(0, 30, n)] + rng.normal(0, 1, (n, d))
    elif kind == "equal":
        X = rng.integers(0, 2, (n, d)) * 3.0
        X[: n // 2] = X[0]
    else:
        X = rng.normal(0, 1, (n, d))
        X[n // 3, 0] = np.inf
        X[n // 2] = np.nan
    return X.astype(np.float32)


@pytest.mark.parametrize("kind", ["clusters", "equal", "unbounded"])
@pytest.mark.parametrize("n,d,k", [(1024, 50, 20), (1025, 8, 5), (1151, 61, 32), (1152, 30, 21), (1153, 16, 20),
                                   (1279, 50, 32), (5000, 50, 30), (30001, 20, 15)])
def test_listed_search_is_the_full_scan(sv, ctx, monkeypatch, n, d, k, kind):
    X = _points(n, d, kind)
    idx, dist = sv.ann(X, k, precision="bf16", ctx=ctx)
    monkeypatch.setenv("SV_KNN_NOPRUNE", "1")
    idx1, dist1 = sv.ann(X, k, precision="bf16", ctx=ctx)
    ok = np.isfinite(X).all(axis=1)                  # other queries have no order to agree on
    if kind == "equal":                              # equal keys: which of them is not decided
        assert np.array_equal(dist[ok], dist1[ok])
    else:
        assert np.array_equal(idx[ok], idx1[ok]) and np.array_equal(dist[ok], dist1[ok])
