"""GPU: blocks too large for a context's memory pool come and go by themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_blocks_are_given_back(sv):
    c = sv.Context(0)
    free0, total = c.memory()
    nnz = []
    for _ in range(2):
        big = sv.CountMatrix.generate(200000, 8000, np.full(8000, 20.0), np.ones(200000), seed=1, ctx=c)
        nnz.append(big.nnz)
        assert 4 * big.nnz > total // 64                 # each of its arrays is such a block
        assert free0 - c.memory()[0] >= 16 * big.nnz
        del big
        assert free0 - c.memory()[0] <= total // 16 + (256 << 20)
    assert nnz[0] == nnz[1]
    held = sv.CountMatrix.generate(200000, 8000, np.full(8000, 20.0), np.ones(200000), seed=1, ctx=c)
    c.close()
    held.h, h = None, held.h                             # freed after its context
    assert c.lib.sv_counts_free(h) == 0
    d = sv.Context(0)
    assert free0 - d.memory()[0] <= 256 << 20
    d.close()
