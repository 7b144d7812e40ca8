"""GPU: the SVD of the projected matrix at the sizes where its split changes (one, two
and three rows per lane; an odd column without a partner; more pairs than warps),
at the end of a cycle and beside the cycle's last feature step (1,024 features on)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [200, 1100])
@pytest.mark.parametrize("work", [4, 5, 31, 32, 33, 34, 63, 64, 65, 66, 95, 96])
def test_projected_svd_sizes(sv, ctx, work, n):
    rng = np.random.default_rng(work)
    m, r = 260, 8                                  # separated leading singular values
    X = sp.random(m, n, density=0.2, random_state=rng, format="csc")
    X = sp.csc_matrix(X + sp.random(m, r, 0.5, random_state=rng) @ sp.diags(8.0 * 0.7 ** np.arange(r)) @
                      sp.random(r, n, 0.3, random_state=rng))
    mu = np.asarray(X.mean(axis=0)).ravel()
    S = sv.CenteredMatrix.from_sparse(X, mu, dtype="float64", ctx=ctx)
    U, s, V = sv.irlba(S, 2, tol=1e-9, work=work, seed=3)
    A = X.toarray() - mu
    ref = np.linalg.svd(A, compute_uv=False)[:2]
    assert np.max(np.abs(s - ref)) <= 1e-8 * ref[0]
    assert np.linalg.norm(V.T @ V - np.eye(2)) <= 1e-10 and np.linalg.norm(U.T @ U - np.eye(2)) <= 1e-10
    assert np.linalg.norm(A @ V - U * s) <= 1e-7 * ref[0]
