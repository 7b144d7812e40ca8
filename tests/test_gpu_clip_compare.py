"""GPU: the FP64 products clip as a comparison of doubles does, at clips above, among and
below the values, negative and infinite, over columns and rows around the groups of
the two kernels and with few and many cells."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale_max", [10.0, 1.0, 0.0, -0.5, -5.0, np.inf])
@pytest.mark.parametrize("n,nf", [(3, 5), (130, 257), (700, 1030), (6000, 300)])
def test_fp64_products_clip(sv, ctx, n, nf, scale_max):
    rng = np.random.default_rng(n)
    X = np.where(rng.random((n, nf)) < 0.3, rng.integers(1, 30, (n, nf)), 0)
    X[0] = 1 + np.arange(nf) % 3                              # no constant column, no empty cell
    X[1:, 0] = 2
    X[2, 1:] = 0
    D = sv.normalize_cells(sv.CountMatrix.from_csc(sp.csc_matrix(X.astype(np.int32)), ctx=ctx), scale_factor=1e4,
                           dtype="float64")
    S = sv.scale_features(D, scale_max=scale_max)
    mu, mean, std = S.stats()
    csc = sp.csc_matrix(X)
    B = np.zeros((n, nf))
    rows, cols = csc.indices, np.repeat(np.arange(nf), np.diff(csc.indptr))
    v = D.values_csc() * (1.0 / std)[cols]
    clip = scale_max + mu[cols]
    B[rows, cols] = np.where(v > clip, clip, v)
    A = B - mu
    for M, x, y in ((A, rng.normal(size=nf), None), (A.T, rng.normal(size=n), None)):
        y = S.mul(x) if M is A else S.rmul(x)
        # sums of products in another order: (terms) 2^-53 of the sum of their sizes, with
        # the product by mu apart
        size = (np.abs(B) if M is A else np.abs(B).T) @ np.abs(x) + (np.abs(mu) @ np.abs(x) if M is A else
                                                                      np.abs(mu) * np.abs(x).sum())
        assert np.all(np.abs(y - M @ x) <= 2 * max(n, nf) * 2.0 ** -53 * size + 1e-300)


def _clipped(sv, ctx, n, nf, scale_max, dtype, seed):
    """A scaled matrix over rows with gaps of more than 63 in most columns (bridged in the
    row-blocked copy), and B - mu of it in FP64 from the parameters that FP32 products use."""
    rng = np.random.default_rng(seed)
    X = np.where(rng.random((n, nf)) < rng.choice([0.004, 0.1, 0.5], nf), rng.integers(1, 30, (n, nf)), 0)
    X[0] = 1 + np.arange(nf) % 3                              # no constant column, no empty cell
    X[1:, 0] = 2
    X[n - 1, 1:] = 5
    D = sv.normalize_cells(sv.CountMatrix.from_csc(sp.csc_matrix(X.astype(np.int32)), ctx=ctx), scale_factor=1e4,
                           dtype=dtype)
    S = sv.scale_features(D, scale_max=scale_max)
    mu, _, std = S.stats()
    csc = sp.csc_matrix(X)
    B = np.zeros((n, nf))
    rows, cols = csc.indices, np.repeat(np.arange(nf), np.diff(csc.indptr))
    inv, clip = (1.0 / std).astype(np.float32)[cols], (scale_max + mu).astype(np.float32)[cols]
    B[rows, cols] = np.minimum((D.values_csc().astype(np.float32) * inv).astype(np.float64), clip)
    return D, S, B, mu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("scale_max", [10.0, 0.0, -0.5, -5.0])
@pytest.mark.parametrize("n,nf", [(130, 257), (3000, 90), (20000, 40)])
def test_row_blocked_product_clips(sv, ctx, n, nf, scale_max, dtype):
    """X^T u over the padded row-blocked copy: padding adds nothing, below any clip either."""
    _, S, B, mu = _clipped(sv, ctx, n, nf, scale_max, dtype, n)
    u = np.random.default_rng(1).normal(size=n).astype(np.float32).astype(np.float64)
    # FP32 sums of at most n products, each rounded; sum(u) and mu in FP64
    size = np.abs(B).T @ np.abs(u)
    assert np.all(np.abs(S.rmul(u) - (B - mu).T @ u) <= (n + 4) * 2.0 ** -24 * size + 1e-12 * np.abs(mu) * np.abs(u).sum())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("scale_max", [10.0, 1.0, 0.0, -0.5, -5.0])
@pytest.mark.parametrize("n,nf", [(130, 257), (3000, 1100)])
def test_irlba_products_clip(sv, ctx, n, nf, scale_max, dtype):
    """Both streamed products of the PCA are those of one matrix, the clipped one: A V = U s
    row by row, and the singular values are A's."""
    _, S, B, mu = _clipped(sv, ctx, n, nf, scale_max, dtype, nf)
    A = B - mu
    U, s, V = sv.irlba(S, 3, tol=1e-8, seed=1)
    # FP32 sums of at most nf products, each rounded; mu.x in double-float; what the
    # iteration leaves (1e-8 s)
    size = ((nf + 4) * 2.0 ** -24 * np.abs(B) + 2.0 ** -40 * np.abs(mu)) @ np.abs(V) + 1e-7 * s[0]
    assert np.all(np.abs(A @ V - U * s) <= size)
    assert np.max(np.abs(s - np.linalg.svd(A, compute_uv=False)[:3])) <= 1e-5 * s[0]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("scale_max", [1.0, -0.5])
def test_batch_products_clip(sv, ctx, scale_max, dtype):
    n, nf, off = 700, 300, np.array([0, 250, 700])
    D, _, _, _ = _clipped(sv, ctx, n, nf, scale_max, dtype, 3)
    v = sp.csr_matrix(D.to_csc())
    ok = np.ones(nf, bool)
    for a, b in zip(off, off[1:]):                            # features that vary in every sample
        ok &= v[a:b].toarray().std(axis=0) > 0
    features = np.flatnonzero(ok) + 1
    batch = sv.Batch.create(D, off, features=features, scale_max=scale_max)
    em = sv.batch_pca(batch, 3, tol=1e-8, seed=1)
    mu, _, std = batch.stats()
    for g, (a, b) in enumerate(zip(off, off[1:])):
        M = v[a:b, features - 1].toarray().astype(np.float64)
        B = np.where(M != 0, np.minimum(M / std[g], scale_max + mu[g]), 0.0)
        s = np.linalg.svd(B - mu[g], compute_uv=False)[:3]
        assert np.max(np.abs(em.stdev[g] * np.sqrt(b - a - 1) - s)) <= 1e-5 * s[0]
