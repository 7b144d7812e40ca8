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


def _listed(sv, ctx, monkeypatch, X, k):
    """Whether the search took the lists, its result and that of a scan of all tiles."""
    ctx.profile_reset()
    ctx.profile(True)
    idx, dist = sv.ann(X, k, precision="bf16", ctx=ctx)
    ctx.profile(False)
    lists = "knn_tile_lists" in ctx.profile_report()
    monkeypatch.setenv("SV_KNN_NOPRUNE", "1")
    return (lists, idx, dist) + tuple(sv.ann(X, k, precision="bf16", ctx=ctx))


@pytest.mark.parametrize("n,d,k", [(150000, 50, 20), (150016, 20, 32), (150017, 8, 5), (150143, 30, 21),
                                   (150144, 50, 30), (150271, 61, 15)])
def test_lists_over_clusters_are_the_full_scan(sv, ctx, monkeypatch, n, d, k):
    """From 150,000 points in clusters on: last tiles of one half, one point, all but one."""
    lists, idx, dist, idx1, dist1 = _listed(sv, ctx, monkeypatch, _points(n, d, "clusters"), k)
    assert lists
    assert np.array_equal(idx, idx1) and np.array_equal(dist, dist1)


@pytest.mark.parametrize("n,kind", [(149999, "clusters"), (150001, "normal"), (150001, "unbounded"),
                                    (150001, "equal")])
def test_other_points_keep_the_widest_dimension(sv, ctx, monkeypatch, n, kind):
    X = _points(n, 50, kind) if kind != "equal" else np.full((n, 50), 2.0, np.float32)
    lists, idx, dist, idx1, dist1 = _listed(sv, ctx, monkeypatch, X, 20)
    assert not lists
    ok = np.isfinite(X).all(axis=1)
    if kind == "equal":
        assert np.all(dist == 0) and np.all(dist1 == 0)
    else:
        assert np.array_equal(idx[ok], idx1[ok]) and np.array_equal(dist[ok], dist1[ok])
