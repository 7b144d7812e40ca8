"""GPU: the compressed-pattern transpose with its source segments cut into
groups, at the edges of tiles (32 output segments) and groups (64 source segments)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,genes,density", [
    (1, 1, 1.0), (31, 63, 0.5), (32, 64, 0.5), (33, 65, 0.9), (2, 5000, 0.3), (5000, 2, 0.3),
    (40, 20011, 0.05), (20011, 40, 0.05), (700, 3001, 0.1), (1000, 300, 0.0)])
def test_transpose_both_ways(sv, ctx, cells, genes, density):
    X = sp.random(cells, genes, density=density, format="csc", random_state=7,
                  data_rvs=lambda n: np.arange(1, n + 1)).astype(np.int32)
    X.sort_indices()
    R = X.tocsr()
    R.sort_indices()
    got = sv.CountMatrix.from_csc(X, ctx=ctx).to_csr()
    assert np.array_equal(got.indptr, R.indptr) and np.array_equal(got.indices, R.indices)
    assert np.array_equal(got.data, R.data)
    got = sv.CountMatrix.upload_csr(R.indptr, R.indices, R.data, R.shape, ctx=ctx).to_csc()
    assert np.array_equal(got.indptr, X.indptr) and np.array_equal(got.indices, X.indices)
    assert np.array_equal(got.data, X.data)
