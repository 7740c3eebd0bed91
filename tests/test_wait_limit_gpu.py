"""A pivot kernel's CTAs that wait too long for one another end the factorization with SDSB200_TIMEOUT, and the next
call starts afresh. The limit is set to 0, so that the first wait that looks at the clock gives up: the helper
clusters of a front of 900 columns wait for each of its blocks. Nothing faults or hangs: every wait returns."""
import numpy as np
import pytest

from sdsb200 import matrices as M
from test_front_edges_gpu import _arrow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("structure", ["S", "G"])
def test_factorization_gives_up_and_recovers(structure, precision):
    from sdsb200 import capi
    from sdsb200._native import numeric_lib
    from sdsb200.solver import DirectSolver

    lib = numeric_lib()
    A = _arrow(900, 40, structure, 3)
    ds = DirectSolver(A, structure, pivot_pairs="none", factor_precision=precision)
    ds.execute("analysis")
    assert ds.execute("factorization") == 0
    want = (*ds.factor_host(), *ds.pivots_host())
    b = M.rhs(A.shape[0], 1, seed=1)
    x = ds.execute("solve", None, b).cpu().numpy()
    for _ in range(2):   # the second time the launches are a replayed graph's
        assert lib.sdsb200_set_wait_limit(ds._plan, 0) == capi.OK
        with pytest.raises(Exception, match="gave up"):
            ds.execute("refactorization")
        assert lib.sdsb200_solve(ds._plan, None, 0, None, 0, 1, None, None, None, None) == capi.PHASE_ORDER
        assert lib.sdsb200_set_wait_limit(ds._plan, 2_000_000_000) == capi.OK
        assert ds.execute("refactorization") == 0
        for got, w in zip((*ds.factor_host(), *ds.pivots_host()), want):
            assert (got is None and w is None) or np.array_equal(got, w)
        assert np.array_equal(ds.execute("solve", None, b).cpu().numpy(), x)
        assert ds.plan_stat("solve_status") == 0
    assert lib.sdsb200_set_wait_limit(ds._plan, -1) == capi.INVALID_VALUE
