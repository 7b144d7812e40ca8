"""GPU: quality control and feature selection where a gene's entries are walked by a
block, several loads at a time, and genes are ranked on the device: columns around a
block's step, all kept, none kept and some kept; equal metrics; counts beyond 15 bits."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1023, 1024, 1025, 1151, 2047, 2049, 3000]


def _matrix(n, seed):
    rng = np.random.default_rng(seed)
    cols = [np.sort(rng.choice(n, min(k, n), replace=False)) for k in LENGTHS]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])])
    val = rng.integers(1, 9, ptr[-1])
    return sp.csc_matrix((val.astype(np.int32), np.concatenate(cols), ptr), shape=(n, len(cols)))


@pytest.mark.parametrize("min_features", [0, 5, 6, 99])
def test_filter_columns(sv, ctx, min_features):
    X = _matrix(3000, 1)
    A, ci = sv.filter_cells(sv.CountMatrix.from_csc(X, ctx), min_features=min_features)
    keep = np.asarray((X > 0).sum(axis=1)).ravel() >= min_features
    assert np.array_equal(ci, keep)
    if not keep.any():
        return
    ref = X[keep].tocsc()
    ref.sort_indices()
    got = A.to_csc()
    assert np.array_equal(got.indptr, ref.indptr) and np.array_equal(got.indices, ref.indices)
    assert np.array_equal(got.data, ref.data)


@pytest.mark.parametrize("genes", [1, 2, 255, 257, 1024, 1025, 2500])
def test_ranks_of_equal_metrics(sv, ctx, genes):
    rng = np.random.default_rng(genes)
    n = 40
    pool = np.where(rng.random((n, 60)) < 0.3, rng.integers(1, 40, (n, 60)), 0)
    X = sp.csc_matrix(pool[:, rng.integers(0, 60, genes)].astype(np.int32))     # many equal genes
    f, metric = sv.find_variable_features(sv.CountMatrix.from_csc(X, ctx), genes)
    assert np.array_equal(f, np.argsort(-metric, kind="stable") + 1)
    k = max(1, genes // 3)
    assert np.array_equal(sv.find_variable_features(sv.CountMatrix.from_csc(X, ctx), k)[0], f[:k])


@pytest.mark.parametrize("factor", [1, 4000, 10**7])
def test_moments_of_small_and_large_counts(sv, ctx, O, factor):
    X = sp.csc_matrix(O.synth_counts(900, 400, -1.0, 1.5, depth=0.5, seed=4))
    X.data = X.data.astype(np.int64)
    X.data[X.indptr[100] : X.indptr[130]] *= factor             # beyond 15 bits, beyond 2^26
    X.data = np.minimum(X.data, 2**31 - 1).astype(np.int32)
    _, metric = sv.find_variable_features(sv.CountMatrix.from_csc(X, ctx), 50)
    _, ref = O.find_variable_features_vst(X, 50)
    assert np.allclose(metric, ref, rtol=1e-9, atol=1e-12)
