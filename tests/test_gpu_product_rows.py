"""GPU: the streamed products of the PCA at the edges of their group rounds: rows
that start anywhere in a group, that are empty, a group, a round (128 or 256
entries) or several rounds long and one entry off; negative values; features that
leave a task of the other product with a single one."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [2600, 24001])
@pytest.mark.parametrize("reps", [1, 9])                     # rows of one block, and of many
def test_rows_of_every_length(sv, ctx, nf, reps):
    rng = np.random.default_rng(reps + nf)
    lens = [0, 1, 3, 4, 5, 7, 8, 9, 31, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1031,
            1535, 2049, 2560] * reps
    lens = np.array(lens)[rng.permutation(len(lens))]
    cols = [np.sort(rng.choice(nf, k, replace=False)) for k in lens]
    ptr = np.concatenate([[0], np.cumsum(lens)])
    val = rng.integers(1, 9, ptr[-1]) * rng.choice([-1.0, 1.0], ptr[-1], p=[0.2, 0.8])
    X = sp.csr_matrix((val, np.concatenate(cols), ptr), shape=(len(lens), nf)).tocsc()
    mu = np.zeros(nf)
    S = sv.CenteredMatrix.from_sparse(X, mu, dtype="float32", ctx=ctx)
    U, s, V = sv.irlba(S, 3, tol=1e-9, seed=1)
    A = X.toarray()
    # U s = A V row by row.  FP32 sums of at most 2,560 terms: each product is off by
    # at most 2560 * 2^-24 = 1.5e-4 of the sum of its terms' sizes in the worst order
    # of signs; an entry missed or taken twice is 1/2560 of it on average, a group 8/2560
    err = np.abs(A @ V - U * s).max(axis=1)
    assert np.all(err <= 1.5e-4 * (np.abs(A) @ np.abs(V)).max(axis=1) + 1e-7 * s[0])
    assert np.max(np.abs(s - np.linalg.svd(A, compute_uv=False)[:3])) <= 1e-5 * s[0]
    w = rng.integers(-4, 5, len(lens)).astype(np.float64)    # exact sums
    assert np.array_equal(S.rmul(w), A.T @ w)


@pytest.mark.parametrize("nf", [1, 15, 16, 17, 33, 200])
def test_transposed_product_with_few_features(sv, ctx, nf):
    rng = np.random.default_rng(nf)
    n = 40000
    X = sp.random(n, nf, 0.2, format="csc", random_state=rng)
    X.data = rng.integers(1, 9, X.nnz).astype(np.float64)
    S = sv.CenteredMatrix.from_sparse(X, np.zeros(nf), dtype="float32", ctx=ctx)
    w = rng.integers(-4, 5, n).astype(np.float64)
    assert np.array_equal(S.rmul(w), X.T @ w)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rows_of_very_different_depth(sv, ctx, dtype):
    """Empty cells, then shallow ones, then a few with most of the entries: the ranges of rows
    that the blocks take hold as many entries each."""
    rng = np.random.default_rng(3)
    n, nf = 9001, 1500
    depth = np.r_[np.zeros(3000), np.full(5500, 0.01), np.linspace(0.02, 0.9, 501)]
    X = np.where(rng.random((n, nf)) < depth[:, None], rng.integers(1, 9, (n, nf)), 0).astype(np.int32)
    D = sv.normalize_cells(sv.CountMatrix.from_csc(sp.csc_matrix(X), ctx=ctx), scale_factor=1e3, dtype=dtype)
    S = sv.scale_features(D, scale_max=np.inf)
    U, s, V = sv.irlba(S, 3, tol=1e-8, seed=1)
    mu, _, std = S.stats()
    B = D.to_csc().toarray().astype(np.float64) / std
    A = B - mu
    # as in test_rows_of_every_length
    size = (1.5e-4 * B + 2.0 ** -40 * np.abs(mu)) @ np.abs(V) + 1e-6 * s[0] / np.sqrt(n)
    assert np.all(np.abs(A @ V - U * s) <= size.max(axis=1)[:, None] + 1e-7 * s[0])
