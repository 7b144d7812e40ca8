"""GPU: the feature-side Lanczos step in one thread-block cluster, at the sizes
where its split changes: where it takes over (1,024 features), rows per CTA not a
multiple of 4 or 32, one, two and four threads per row, CTAs without rows, and
bases that no longer fit shared memory."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,nu,dtype", [
    (300, 1023, 3, "float64"), (500, 1024, 3, "float32"), (400, 1089, 5, "float64"), (1500, 1153, 50, "float64"),
    (700, 2049, 20, "float32"), (400, 2500, 5, "float64"), (700, 4097, 20, "float32"), (500, 8501, 50, "float64"),
    (300, 20003, 5, "float32")])
def test_feature_step_sizes(sv, ctx, m, n, nu, dtype):
    rng = np.random.default_rng(m + n)
    X = sp.random(m, n, density=0.05, random_state=rng, format="csc")
    r = nu + 3                                     # separated leading singular values
    X = sp.csc_matrix(X + sp.random(m, r, 0.5, random_state=rng) @ sp.diags(3.0 * 0.9 ** np.arange(r)) @
                      sp.random(r, n, 0.3, random_state=rng))
    X.data = X.data.astype(np.float32).astype(np.float64)
    mu = np.asarray(X.mean(axis=0)).ravel()
    S = sv.CenteredMatrix.from_sparse(X, mu, dtype=dtype, ctx=ctx)
    U, s, V = sv.irlba(S, nu, tol=1e-8, seed=3)
    A = X.toarray() - mu
    ref = np.linalg.svd(A, compute_uv=False)[:nu]
    # the products are FP64 or FP32 over rows of at most 20,003 entries
    tol = 1e-8 if dtype == "float64" else 1e-5
    assert np.max(np.abs(s - ref)) <= tol * ref[0]
    assert np.linalg.norm(V.T @ V - np.eye(nu)) <= 1e-10 and np.linalg.norm(U.T @ U - np.eye(nu)) <= 1e-10
    assert np.linalg.norm(A @ V - U * s) <= 10 * tol * ref[0]


@pytest.mark.parametrize("n,dtype", [(1200, "float64"), (3001, "float32")])
def test_fused_step_is_the_multi_block_step(sv, ctx, monkeypatch, n, dtype):
    """Bit for bit: the joined launches keep the arithmetic and the order."""
    rng = np.random.default_rng(n)
    X = sp.random(2600, n, density=0.1, random_state=rng, format="csc")
    S = sv.CenteredMatrix.from_sparse(X, np.asarray(X.mean(axis=0)).ravel(), dtype=dtype, ctx=ctx)
    out = []
    for mode in (None, "multi"):
        if mode:
            monkeypatch.setenv("SV_VSIDE", mode)
        l0 = ctx.launches()
        out.append(sv.irlba(S, 12, tol=1e-6, seed=2) + (ctx.launches() - l0,))
    (U, s, V, lf), (U2, s2, V2, lm) = out
    assert np.array_equal(s, s2) and np.array_equal(U, U2) and np.array_equal(V, V2)
    assert lf < lm                                 # the paths do differ
