"""GPU: the bank-aware order of the X v copy, put together in shared memory for rows up
to 2,048 entries and entry by entry for longer ones: rows at every offset of a group,
around both limits, with classes that overflow their slots, all in one class and too
uneven to be reordered.  The product is a sum of whole numbers: any entry lost, doubled
or with another's value shows."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("shift", [0, 1, 5])
def test_rows_keep_their_entries(sv, ctx, dtype, shift):
    nf = 6000
    rng = np.random.default_rng(shift)
    rows = [np.arange(shift)]
    for k in (1, 2, 7, 8, 9, 31, 33, 127, 129, 255, 257, 1000, 1024, 2040, 2047, 2048, 2049, 2055, 3000):
        rows.append(np.sort(rng.choice(nf, k, replace=False)))
    rows += [np.arange(0, 6000, 16)[:n] for n in (5, 100, 375)]           # one class
    rows += [np.arange(0, 6000, 8)[:n] for n in (64, 750)]                # two classes
    rows += [np.sort(np.concatenate([np.arange(0, 6000, 16), np.arange(1, 6000, 2)[:n]])) for n in (50, 1500)]
    rows += [np.empty(0, np.int64), np.arange(17), np.arange(nf)]        # the last: no constant feature
    n = len(rows)
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    X = sp.csr_matrix((rng.integers(1, 4, ptr[-1]).astype(np.int32), np.concatenate(rows), ptr), shape=(n, nf))
    C = sv.CountMatrix.from_csc(X.tocsc(), ctx=ctx)
    D = sv.normalize_cells(C, method="relativecounts", scale_factor=1.0, dtype=dtype)
    S = sv.scale_features(D)
    mu, mean, std = S.stats()
    csc = X.tocsc()
    v = rng.integers(-4, 5, nf).astype(np.float64)
    B = sp.csc_matrix((D.values_csc().astype(np.float64), csc.indices, csc.indptr), shape=(n, nf))
    w = v / std
    size = abs(B) @ abs(w)
    # a lane adds at most 6000 / 32 + 8 terms and 5 sums follow, each term rounded three
    # times: 204 roundings of 2^-24; an entry of a row of k is 1/k of the size on average
    err = np.abs(S.mul(v) - (B @ w - mu @ v))
    assert np.all(err <= 204 * 2.0 ** -24 * size + 1e-12 * (np.abs(mu) @ np.abs(v)))
