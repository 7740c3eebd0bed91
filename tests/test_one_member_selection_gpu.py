"""``ubatch_index`` = 0 and ``ubatch_mask`` = [1] on a single system select its only member: every call must do
what it does without a selection, also where one launch takes several groups of 8 right-hand sides."""
import numpy as np
import pytest

from helpers import small_kkt
from sdsb200 import matrices as M

pytestmark = pytest.mark.gpu


def _matrix(structure):
    return {"SPD": lambda: M.lap3d(13, 12, 11, seed=6), "S": lambda: small_kkt(20, 20, 150, seed=2),
            "G": lambda: M.convection_diffusion3d(11, 10, 9, seed=6)}[structure]()


@pytest.mark.parametrize("structure", ["SPD", "S", "G"])
@pytest.mark.parametrize("nrhs", [1, 8, 16, 33])
def test_solve_of_the_selected_member(structure, nrhs):
    from sdsb200.solver import DirectSolver

    A = _matrix(structure)
    b = np.random.default_rng(5).uniform(-1, 1, (A.shape[0], nrhs))
    for ir in (0, 1):
        ds = DirectSolver(A, structure, reordering_alg="nd", max_nrhs=nrhs, ir_n_steps=ir)
        ds.execute("analysis")
        assert ds.execute("factorization") == 0
        modes = (0, 1) if structure == "G" else (0,)

        def solve(mode):
            ds.setparam("solve_mode", mode)
            x = np.full((A.shape[0], nrhs), 7.0)
            ds.execute("solve", x, b)
            return x

        want = [solve(m) for m in modes]
        for name, value, off in (("ubatch_index", 0, -1), ("ubatch_mask", [1], None)):
            ds.setparam(name, value)
            for m in modes:   # the same tasks on the same factor: the same bits
                assert np.array_equal(solve(m), want[m]), (name, ir, m)
            ds.setparam(name, off)
        assert ds.plan_stat("solve_status") == 0


@pytest.mark.parametrize("structure", ["S", "G"])
def test_factorization_of_the_selected_member(structure):
    """The same kernels: equal pivots and factors would also come from the one-CTA pivot kernel that batches use,
    ten times slower on these fronts (up to 400 columns), so the pivot launches' time is compared too."""
    from sdsb200._native import numeric_lib
    from sdsb200.solver import DirectSolver

    A = M.convection_diffusion3d(20, 20, 20, seed=6) if structure == "G" else M.lap3d(20, 20, 20, seed=6)
    ds = DirectSolver(A, structure, reordering_alg="nd")
    ds.execute("analysis")

    def factor():
        assert ds.execute("refactorization") == 0
        numeric_lib().sdsb200_set_profiling(ds._plan, 1)   # resets the totals
        assert ds.execute("refactorization") == 0
        ms = ds.plan_stat("prof_ms:pivot")
        numeric_lib().sdsb200_set_profiling(ds._plan, 0)
        return ms, ds.factor_host(), ds.pivots_host()

    assert ds.execute("factorization") == 0
    ms, fac, piv = factor()
    for name, value, off in (("ubatch_index", 0, -1), ("ubatch_mask", [1], None)):
        ds.setparam(name, value)
        ms_sel, fac_sel, piv_sel = factor()
        ds.setparam(name, off)
        assert all(np.array_equal(x, y) for x, y in zip(fac + piv, fac_sel + piv_sel) if x is not None)
        assert ms_sel <= 2.0 * ms + 0.5, (name, ms_sel, ms)
