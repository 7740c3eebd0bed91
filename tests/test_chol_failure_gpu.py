"""A Cholesky front of many row tiles whose pivot fails in one of its 64-column steps: the step's CTAs, one per tile,
must leave the panel alone whether or not they learn of it from the front's info, so the panel is the same after
every factorization, and the info is the failing column's."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("position", [0, 63, 64, 100, 200, 1150])
def test_failing_step_leaves_the_panel(position, precision):
    from sdsb200.solver import DirectSolver

    n = 1200   # dense: one front
    rng = np.random.default_rng(position)
    B = np.triu(rng.uniform(-1, 1, (n, n)), 1)
    B = B + B.T + 4 * n * np.eye(n)
    ds = DirectSolver(sp.csr_matrix(B), "SPD", factor_precision=precision)
    ds.execute("analysis")
    bad = int(ds.symbolic.perm[position]) - 1
    B[bad, bad] = -1.0
    A = sp.csr_matrix(B)
    ds.update(A.data)
    assert ds.execute("factorization") == bad + 1
    want = ds.factor_host()[0]
    for _ in range(30):
        assert ds.execute("refactorization") == bad + 1
        assert np.array_equal(ds.factor_host()[0], want)
