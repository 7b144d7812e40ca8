"""GPU: entries per cell of a coordinate file counted by runs: runs that end at, before
and after a warp's 32 entries, a last warp of every size, cells out of order."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["cells", "shuffled", "alternating"])
@pytest.mark.parametrize("extra", [0, 1, 31])
def test_runs_of_cells(sv, ctx, order, extra):
    genes = 70
    lens = [1, 31, 32, 33, 64, 1, 1, 30, 2, 65, 0, 7, extra]
    cell = np.repeat(np.arange(len(lens)), lens)
    gene = np.concatenate([np.arange(k) for k in lens])
    val = 1 + np.arange(len(cell)) % 9
    at = np.arange(len(cell))
    if order == "shuffled":
        at = np.random.default_rng(extra).permutation(at)
    elif order == "alternating":
        at = np.argsort(gene, kind="stable")
    text = "%%MatrixMarket matrix coordinate integer general\n" + f"{genes} {len(lens)} {len(cell)}\n"
    text += "".join(f"{gene[i] + 1} {cell[i] + 1} {val[i]}\n" for i in at)
    got = sv.CountMatrix.parse_mtx(text.encode(), ctx=ctx).to_csc()
    ref = sp.csc_matrix((val, (cell, gene)), shape=(len(lens), genes))
    assert got.shape == ref.shape and (got != ref).nnz == 0 and got.nnz == ref.nnz
