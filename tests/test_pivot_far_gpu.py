"""Dense symmetric fronts whose Bunch-Kaufman partners lie outside the pivot kernel's block of 32 columns: every pivot a
2x2 one with a column half a front away, random ones, and rejected choices (a high threshold). Pivots, D, panels and
statistics equal the oracle's bit for bit; each row of the front is one entry of the matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import dense_panels, oracle_for

pytestmark = pytest.mark.gpu


def _far(n, rng):
    h = n // 2
    B = 0.01 * rng.uniform(-1, 1, (n, n))
    B[:h, :h] *= 0.01
    p = rng.permutation(h)
    B[np.arange(h), h + p] = 1.0 + 0.1 * rng.uniform(-1, 1, h)
    return np.triu(B) + np.triu(B, 1).T


@pytest.mark.parametrize("n", [70, 300, 385, 700, 1100])
@pytest.mark.parametrize("values,u", [("far", 0.01), ("random", 0.01), ("random", 0.5), ("random", 0.9)])
def test_partners_outside_the_block(n, values, u):
    from sdsb200.solver import DirectSolver

    rng = np.random.default_rng(n)
    if values == "far":
        B = _far(n, rng)
    else:
        B = rng.uniform(-1, 1, (n, n))
        B = B + B.T
    A = sp.csr_matrix(B)
    A.sort_indices()
    S, O, info = oracle_for(A, "S", pivot_pairs="none", pivot_threshold=u)
    ds = DirectSolver(A, "S", pivot_pairs="none", pivot_threshold=u)
    ds.execute("analysis")
    assert np.array_equal(ds.symbolic.perm, S.perm)
    assert ds.execute("factorization") == info
    assert np.array_equal(ds.stats_host(), O.stats_matrix())
    piv, kind, d = ds.pivots_host()
    assert np.array_equal(piv[:n], O.piv[:n])
    assert np.array_equal(kind[:n], O.kind[:n])
    assert np.array_equal(d[: 2 * n], O.d[: 2 * n])
    assert np.array_equal(dense_panels(S, ds.factor_host()[0]), dense_panels(S, O.factor))
