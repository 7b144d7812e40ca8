"""GPU: normalised values gathered from the table of small counts are the values
that every entry gets by itself: counts at both ends of the table and above it,
rows of odd lengths, all types and methods."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _bits(a):
    return a.view({2: np.uint16, 4: np.uint32, 8: np.uint64}[a.dtype.itemsize])


@pytest.mark.parametrize("method", ["lognormalize", "relativecounts"])
@pytest.mark.parametrize("dtype", ["float64", "float32", "bfloat16"])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_table_values_are_the_direct_ones(sv, ctx, n, dtype, method):
    rng = np.random.default_rng(n)
    genes = 1001
    X = np.where(rng.random((n, genes)) < 0.4, rng.geometric(0.2, (n, genes)), 0)
    X[:, :7] = [1, 2, 31, 32, 33, 64, 100000]
    X[0, 900:] = 0
    assert (X > 0).sum() >= 64 * n                           # dense enough for the table ...
    empty = (X > 0).sum() // 64 - n + 1
    Y = np.vstack([X, np.zeros((empty, genes), X.dtype)])    # ... and with empty cells not
    out = []
    for M in (X, Y):
        D = sv.normalize_cells(sv.CountMatrix.from_csc(sp.csc_matrix(M.astype(np.int32)), ctx=ctx),
                               method=method, scale_factor=1e4, dtype=dtype)
        out.append((D.values_csc(), D.values_csr()))
    for a, b in zip(out[0], out[1]):
        assert np.array_equal(_bits(np.asarray(a)), _bits(np.asarray(b)))
    if dtype == "float64":
        s = X.sum(1)
        cols, rows = np.nonzero(X.T)
        v = (1e4 * X[rows, cols]) / s[rows]
        ref = np.log1p(v) if method == "lognormalize" else v
        # division exact to 1/2 ulp in both, log1p within 2 ulp in both
        np.testing.assert_allclose(out[0][0], ref, rtol=4 * 2.0 ** -52, atol=0)
