"""GPU: the pair sort behind the neighbour searches at the sizes where its larger
strides change how many go to a launch: the exact search over points ordered by it
returns the exact neighbours."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("n", [2048, 2049, 4096, 4097, 8193, 16385, 32769, 70000])
def test_neighbours_of_ordered_points(sv, ctx, n, precision):
    rng = np.random.default_rng(n)
    X = (rng.normal(0, 4, (12, 6))[rng.integers(0, 12, n)] + rng.normal(0, 1, (n, 6))).astype(np.float32)
    idx, dist = sv.ann(X, 5, precision=precision, ctx=ctx)
    rows = rng.choice(n, 40, replace=False)
    for r in rows:
        d2 = ((X.astype(np.float64) - X[r]) ** 2).sum(1)
        assert np.allclose(dist[r], np.sqrt(np.sort(d2)[:5]), rtol=1e-5, atol=1e-5)
