"""GPU: the FP32 neighbour search, without and over tile lists, against FP64 brute
force, where the lists begin (8,192 points), at ragged last tiles and blocks, for
clustered, unclustered, sorted, repeated and non-finite points, every padded
dimension's edges, and both metrics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, d, shape, rng):
    if shape == "clusters":
        c = 8.0 * rng.standard_normal((40, d))
        X = c[np.sort(rng.integers(0, 40, n))] + rng.standard_normal((n, d))
    elif shape == "one":
        X = rng.standard_normal((n, d)) / np.sqrt(1 + np.arange(d))
    else:
        X = rng.integers(-1, 2, (n, d)).astype(float)      # many equal points and distances
    return X.astype(np.float32)


def _brute(X, k, metric, include_self):
    Y = X.astype(np.float64)
    if metric == "cosine":
        Y = Y / np.linalg.norm(Y, axis=1, keepdims=True)
    d2 = (Y * Y).sum(1)[:, None] + (Y * Y).sum(1) - 2 * Y @ Y.T
    np.fill_diagonal(d2, -1.0 if include_self else np.inf)
    d2 = np.maximum(np.sort(d2, axis=1)[:, :k], 0)
    return d2 / 2 if metric == "cosine" else np.sqrt(d2)


@pytest.mark.parametrize("n,d,k,shape,metric,inc", [
    (1023, 7, 5, "clusters", "euclidean", True), (1025, 8, 20, "one", "euclidean", False),
    (2047, 50, 16, "clusters", "euclidean", True), (2048, 50, 17, "clusters", "euclidean", False),
    (2305, 9, 32, "one", "cosine", True), (4096, 61, 20, "clusters", "cosine", False),
    (5001, 64, 10, "clusters", "euclidean", True), (6145, 33, 30, "clusters", "euclidean", True)])
def test_listed_search_distances(sv, ctx, n, d, k, shape, metric, inc):
    X = _points(n, d, shape, np.random.default_rng(n + d))
    idx, dist = sv.ann(X, k, metric=metric, include_self=inc, precision="fp32", ctx=ctx)
    ref = _brute(X, k, metric, inc)
    # FP32 sums of at most 64 squared differences of coordinates up to ~30
    tol = 2e-5 * max(1.0, np.abs(X).max()) if metric == "euclidean" else 2e-6
    assert not np.any(np.abs(dist - ref) > tol + 1e-5 * ref)
    if inc:
        assert np.array_equal(idx[:, 0], np.arange(1, n + 1))
    else:
        assert not np.any(idx == np.arange(1, n + 1)[:, None])


def test_equal_points_by_index(sv, ctx):
    """More equal points than candidates: the lowest indices, as in a scan in order."""
    X = np.repeat(_points(30, 6, "clusters", np.random.default_rng(1)), 100, axis=0)
    X = X[np.random.default_rng(2).permutation(len(X))]
    idx, dist = sv.ann(X, 12, include_self=False, precision="fp32", ctx=ctx)
    _, inv = np.unique(X, axis=0, return_inverse=True)
    for i in range(0, len(X), 37):
        same = np.flatnonzero(inv.ravel() == inv.ravel()[i])
        assert np.array_equal(idx[i], same[same != i][:12] + 1)
    assert np.all(dist == 0)


def test_non_finite_points_do_not_hide_others(sv, ctx):
    X = _points(3001, 12, "clusters", np.random.default_rng(3))
    bad = np.array([5, 1500, 3000])
    X[bad[0], 3], X[bad[1], 0], X[bad[2], 11] = np.nan, np.inf, -np.inf
    ok = np.setdiff1d(np.arange(3001), bad)
    _, dist = sv.ann(X, 8, precision="fp32", ctx=ctx)
    ref = _brute(X[ok], 8, "euclidean", True)
    assert not np.any(np.abs(dist[ok] - ref) > 1e-3)


@pytest.mark.parametrize("n,d,k,shape,metric,inc", [
    (8191, 50, 16, "clusters", "euclidean", True), (8192, 50, 17, "clusters", "euclidean", False),
    (8193, 9, 32, "one", "cosine", True), (9025, 61, 20, "clusters", "cosine", False),
    (12001, 64, 8, "clusters", "euclidean", True), (12031, 33, 30, "equal", "euclidean", True)])
def test_lists_where_they_begin(sv, ctx, n, d, k, shape, metric, inc):
    """Both sides of the line (8,192 points) from which the FP32 search orders its points."""
    X = _points(n, d, shape, np.random.default_rng(n + d))
    idx, dist = sv.ann(X, k, metric=metric, include_self=inc, precision="fp32", ctx=ctx)
    rows = np.unique(np.r_[0:130, np.random.default_rng(1).integers(0, n, 600), n - 130:n])
    Y = X.astype(np.float64)
    if metric == "cosine":
        Y = Y / np.linalg.norm(Y, axis=1, keepdims=True)
    d2 = (Y[rows] ** 2).sum(1)[:, None] + (Y * Y).sum(1) - 2 * Y[rows] @ Y.T
    d2[np.arange(len(rows)), rows] = -1.0 if inc else np.inf
    d2 = np.maximum(np.sort(np.partition(d2, k, axis=1)[:, :k], axis=1), 0)
    ref = d2 / 2 if metric == "cosine" else np.sqrt(d2)
    # FP32 sums of at most 64 squared differences of coordinates up to ~30
    tol = 2e-5 * max(1.0, np.abs(X).max()) if metric == "euclidean" else 2e-6
    assert not np.any(np.abs(dist[rows] - ref) > tol + 1e-5 * ref)
    own = np.arange(1, n + 1)
    assert np.array_equal(idx[:, 0], own) if inc else not np.any(idx == own[:, None])
