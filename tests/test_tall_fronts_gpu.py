"""The kernels that wide LDLT / LU fronts take by their height: clusters of 8 CTAs with a copy of the block's rows (up to
3840 rows below the first block), without it, clusters of 16 (from 4097 rows), the cooperative kernel (from 8193), and
the one-CTA kernel of uniform batches. A few columns over a tall separator that is the Schur complement, so that
only the tall front is factored: pivots, D, statistics and panels equal the oracle's bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import dense_panels, oracle_for
from test_front_edges_gpu import _arrow

pytestmark = pytest.mark.gpu


def _tall(w, s, structure, seed):
    rng = np.random.default_rng(seed)
    B11 = rng.uniform(-1, 1, (w, w))
    B12 = rng.uniform(-1, 1, (w, s))
    B21 = rng.uniform(-1, 1, (s, w)) if structure == "G" else B12.T
    if structure != "G":
        B11 = B11 + B11.T
    np.fill_diagonal(B11, rng.choice([0.0, 0.05, 30.0], w, p=[0.2, 0.4, 0.4]))
    A = sp.bmat([[sp.csr_matrix(B11), sp.csr_matrix(B12)], [sp.csr_matrix(B21), sp.diags(rng.uniform(1, 2, s))]], format="csr")
    A.sort_indices()
    return A


@pytest.mark.parametrize("structure", ["S", "G"])
@pytest.mark.parametrize("w,s", [(70, 3700), (40, 3860), (33, 4100), (70, 5000), (40, 8160)])
def test_tall_front(structure, w, s):
    from sdsb200.solver import DirectSolver

    A = _tall(w, s, structure, w + s)
    flags = np.zeros(w + s, np.int8)
    flags[w:] = 1
    S, O, info = oracle_for(A, structure, pivot_pairs="none", user_schur_indices=flags)
    ds = DirectSolver(A, structure, pivot_pairs="none", schur_mode=1, user_schur_indices=flags)
    ds.execute("analysis")
    assert np.array_equal(ds.symbolic.perm, S.perm)
    f = int(S.front_nrows[0])
    assert f >= s + 1 and int(S.front_ncols[0]) == f - s        # the tall front, first
    assert ds.execute("factorization") == info
    assert np.array_equal(ds.stats_host()[0], O.stats_matrix()[0])
    piv, kind, d = ds.pivots_host()
    n, n1 = w + s, f - s
    assert np.array_equal(piv[:n1], O.piv[:n1])
    assert np.array_equal(kind[:n1], O.kind[:n1])
    assert np.array_equal(d[:n1], O.d[:n1]) and (structure == "G" or np.array_equal(d[n: n + n1], O.d[n: n + n1]))
    for got, want in zip(ds.factor_host(), (O.factor, O.ufactor if structure == "G" else None)):
        if want is not None:
            P, Q = (x[: f * n1].reshape(n1, f).T for x in (got, want))
            assert all(np.array_equal(P[j:, j], Q[j:, j]) for j in range(n1))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("structure", ["S", "G"])
@pytest.mark.parametrize("w,s", [(200, 33), (353, 70), (700, 40)])
def test_panel_kernel_against_one_cta(structure, w, s, precision):
    """A uniform batch of the same matrix twice: the one-CTA kernel's pivots and panels."""
    from sdsb200.solver import DirectSolver

    A = _arrow(w, s, structure, w + s)
    one = DirectSolver(A, structure, pivot_pairs="none", factor_precision=precision)
    two = DirectSolver((A.indptr, A.indices, np.concatenate([A.data, A.data]), A.shape[0]), structure,
                       pivot_pairs="none", factor_precision=precision)
    for ds in (one, two):
        ds.execute("analysis")
    info = one.execute("factorization")
    assert list(two.execute("factorization")) == [info, info]
    for x, y in zip(one.pivots_host(), two.pivots_host(1)):
        assert np.array_equal(x, y)
    for x, y in zip(one.factor_host(), two.factor_host(1)):
        assert (x is None) == (y is None)
        if x is not None:
            assert np.array_equal(dense_panels(one.symbolic, x), dense_panels(two.symbolic, y))
