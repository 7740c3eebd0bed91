"""More right-hand sides than one group of the one-launch solve takes (8): groups as members of one launch,
up to four per launch, the last one short. Each column must equal the same column solved alone to rounding,
for A and A^T, with and without refinement."""
import numpy as np
import pytest

from helpers import small_kkt
from sdsb200 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("structure", ["SPD", "S", "G"])
@pytest.mark.parametrize("nrhs", [9, 16, 31, 33])
def test_groups_match_single_columns(structure, nrhs):
    from sdsb200.solver import DirectSolver

    A = {"SPD": lambda: M.lap3d(13, 12, 11, seed=6), "S": lambda: small_kkt(20, 20, 150, seed=2),
         "G": lambda: M.convection_diffusion3d(11, 10, 9, seed=6)}[structure]()
    n = A.shape[0]
    b = np.random.default_rng(5).uniform(-1, 1, (n, nrhs))
    for ir in (0, 1):
        ds = DirectSolver(A, structure, reordering_alg="nd", max_nrhs=nrhs, ir_n_steps=ir)
        ds.execute("analysis")
        assert ds.execute("factorization") == 0
        for tr in ((False, True) if structure == "G" else (False,)):
            ds.setparam("solve_mode", int(tr))
            x = ds.execute("solve", None, b).cpu().numpy()
            # the same tasks in another instance of the kernel: sums in another order at most, a few n eps
            for c in (0, 7, 8, nrhs - 1):
                one = ds.execute("solve", None, b[:, c]).cpu().numpy()
                assert np.abs(x[:, c] - one).max() <= 1e-10 * np.abs(one).max(), (tr, ir, c)
            AA = A.T.tocsr() if tr else A
            assert M.scaled_backward_error(AA, x, b) <= 1e-12
        assert ds.plan_stat("solve_status") == 0
