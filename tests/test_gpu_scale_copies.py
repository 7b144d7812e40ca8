"""GPU: the product copies of scale_features at their edges: features absent from
whole row blocks, steps between a feature's rows around the 63 that a code holds
and up to a block, last blocks of one row."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16384, 16385, 33000])
def test_row_blocked_copy_steps(sv, ctx, n):
    rng = np.random.default_rng(n)
    cols = [np.arange(0, n, st) for st in (1, 62, 63, 64, 65, 126, 127, 1000, 16383, n)]
    cols += [np.array([0, n - 1]), np.array([n - 1]), np.array([16383]), np.arange(16384, n),
             np.sort(rng.choice(n, 300, replace=False)), np.empty(0, np.int64)]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])])
    val = rng.integers(1, 255, ptr[-1]).astype(np.float64)          # exact in FP32
    X = sp.csc_matrix((val, np.concatenate(cols).astype(np.int64), ptr), shape=(n, len(cols)))
    S = sv.CenteredMatrix.from_sparse(X, np.zeros(len(cols)), dtype="float32", ctx=ctx)
    u = rng.integers(-8, 9, n).astype(np.float64)                    # exact sums in FP32
    assert np.array_equal(S.rmul(u), X.T @ u)
    v = rng.integers(-8, 9, len(cols)).astype(np.float64)
    assert np.array_equal(S.mul(v), X @ v)
