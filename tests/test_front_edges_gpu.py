"""Fronts at the edges of the factorization kernels' blocks: 32 columns of a pivot block, 64 columns of a Cholesky
step, 64 / 128 rows of an update tile, 32 rows of a register chunk, the lines between the kernels (64 and 96
rows) and between one CTA and a cluster (384 rows). Two dense blocks of w columns that share a dense separator
of s: two fronts of (w + s, w) and one of (s, s), or what amalgamation makes of them.

"S" and "G": pivots, D, panels and statistics equal the oracle's bit for bit, with diagonals small enough for
interchanges, 2x2 pivots and pivots from outside the block. "SPD": panels within 1e-10 of the oracle, as
everywhere: sums of at most 1000 products in another order, condition below 10, are off by a few 1e-13."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import dense_panels, oracle_for, rel_max_diff
from sdsb200 import matrices as M

pytestmark = pytest.mark.gpu

SIZES = [(1, 0), (2, 1), (31, 1), (32, 0), (33, 31), (48, 17), (63, 1), (64, 0), (65, 0), (64, 33), (95, 1), (96, 0),
         (97, 31), (127, 2), (129, 65), (160, 160), (353, 33), (385, 127), (511, 1), (513, 70), (900, 40)]


def _arrow(w, s, structure, seed):
    rng = np.random.default_rng(seed)
    n = 2 * w + s
    mask = np.ones((n, n), bool)
    mask[:w, w:2 * w] = mask[w:2 * w, :w] = False
    B = rng.uniform(-1, 1, (n, n)) * mask
    if structure != "G":
        B = (B + B.T) / 2
    if structure == "SPD":
        B += n * np.eye(n)
    else:   # most diagonals lose against their column, some are zero
        B[np.arange(n), np.arange(n)] *= rng.choice([0.0, 0.05, 30.0], n, p=[0.2, 0.4, 0.4])
    i, j = np.nonzero(mask)
    A = sp.csr_matrix((B[i, j], (i, j)), shape=(n, n))
    A.sort_indices()
    return A


@pytest.mark.parametrize("structure", ["SPD", "S", "G"])
@pytest.mark.parametrize("w,s", SIZES)
def test_front_edges(structure, w, s):
    from sdsb200.solver import DirectSolver

    A = _arrow(w, s, structure, 7 * w + s)
    pairs = {} if structure == "SPD" else dict(pivot_pairs="none")
    S, O, info = oracle_for(A, structure, **pairs)
    ds = DirectSolver(A, structure, **pairs)
    ds.execute("analysis")
    assert np.array_equal(ds.symbolic.perm, S.perm)
    assert ds.execute("factorization") == info
    assert np.array_equal(ds.stats_host(), O.stats_matrix())
    fac, ufac = ds.factor_host()
    if structure == "SPD":
        assert rel_max_diff(dense_panels(S, fac), dense_panels(S, O.factor)) <= 1e-10
    else:
        piv, kind, d = ds.pivots_host()
        assert np.array_equal(piv[: S.n], O.piv[: S.n])
        assert np.array_equal(kind[: S.n], O.kind[: S.n])
        assert np.array_equal(d[: (2 if structure == "S" else 1) * S.n], O.d[: (2 if structure == "S" else 1) * S.n])
        assert np.array_equal(dense_panels(S, fac), dense_panels(S, O.factor))
        if structure == "G":
            assert np.array_equal(ufac, O.ufactor)
    b = M.rhs(A.shape[0], 1, seed=1)
    x = ds.execute("solve", None, b).cpu().numpy()
    if structure == "SPD":
        assert M.scaled_backward_error(A, x, b) <= 1e-12
    elif not (kind[: S.n] == 4).any():   # no perturbed pivot
        # both solutions come from the same factor: as many roundings of the same sizes, in another order
        xo = O.solve(b)
        assert M.scaled_backward_error(A, x, b) <= 1e3 * M.scaled_backward_error(A, xo, b) + 1e-13
