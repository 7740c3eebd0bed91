"""Cholesky pivots over the exponent range: the reciprocal square root's fast form is used from 2^-99 up to 2^100, rsqrt()
beyond. The shared-memory, warp and 64-column step kernels, FP64 and FP32."""
import numpy as np
import pytest
import scipy.sparse as sp

from helpers import dense_panels, oracle_for
from sdsb200 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,lo,hi,ulp", [("fp64", -1000, 1000, 2.0 ** -52), ("fp32", -120, 120, 2.0 ** -23)])
@pytest.mark.parametrize("n", [300, 20000])   # CTA per front, warp per front
def test_diagonal(n, precision, lo, hi, ulp):
    """Fronts of one column: L = sqrt(d), whose correction leaves one unit in the last place."""
    from sdsb200.solver import DirectSolver

    rng = np.random.default_rng(n)
    d = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n))
    d[:6] = np.ldexp([1.0, 2.0 - 2.0 ** -20, 1.0, 2.0 - 2.0 ** -20, 1.0, 1.0], [-99, -100, 100, 99, lo, hi - 1])
    if precision == "fp32":
        d = d.astype(np.float32).astype(np.float64)
    A = sp.diags(d).tocsr()
    ds = DirectSolver(A, "SPD", pivot_epsilon=0.0, factor_precision=precision)
    ds.execute("analysis")
    assert ds.execute("factorization") == 0
    L = ds.factor_host()[0][ds.symbolic.front_ptr[:-1] - 1]
    want = np.sqrt(d[ds.symbolic.perm - 1])
    assert np.abs(L / want - 1).max() <= ulp


@pytest.mark.parametrize("precision,exps,tol", [("fp64", (-960, -240, -100, -98, 0, 96, 100, 240, 900), 1e-12),
                                                ("fp32", (-110, -98, 0, 96, 110), 1e-4)])
@pytest.mark.parametrize("n", [24, 90, 200])   # fronts in registers (32 and 96 rows), 64-column steps
def test_scaled_dense(n, precision, exps, tol):
    """A 2^k (k even) has the factor L 2^(k/2). Sums of at most 200 products, condition below 3: the largest relative
    difference is a few 200 eps."""
    from sdsb200.solver import DirectSolver

    rng = np.random.default_rng(n)
    B = rng.uniform(-1, 1, (n, n))
    B = (B + B.T) / 2 + n * np.eye(n)
    S, O, info = oracle_for(sp.csr_matrix(B), "SPD", pivot_epsilon=0.0)
    want = dense_panels(S, O.factor)
    ds = DirectSolver(sp.csr_matrix(B), "SPD", pivot_epsilon=0.0, factor_precision=precision)
    ds.execute("analysis")
    for k in exps:
        ds.update(np.ldexp(sp.csr_matrix(B).data, k))
        assert ds.execute("factorization") == 0
        got = np.ldexp(dense_panels(ds.symbolic, ds.factor_host()[0]), -k // 2)
        assert np.abs(got - want).max() <= tol * np.abs(want).max(), k


def test_scaled_batch():
    """The warp kernel's fronts of several columns: 256 members, each at its own scale, against the unscaled member."""
    from sdsb200.solver import DirectSolver

    A = M.lap2d_shifted(16, 16, seed=1)
    n, nb = A.shape[0], 256
    k = 2 * np.random.default_rng(0).integers(-240, 240, nb)
    vals = np.ldexp(np.tile(A.data, (nb, 1)), k[:, None])
    ds = DirectSolver((A.indptr, A.indices, vals.reshape(-1), n), "SPD", pivot_epsilon=0.0)
    ds.execute("analysis")
    assert list(ds.execute("factorization")) == [0] * nb
    S, O, _ = oracle_for(A, "SPD", pivot_epsilon=0.0)
    want = dense_panels(S, O.factor)
    for m in range(0, nb, 5):
        got = np.ldexp(dense_panels(ds.symbolic, ds.factor_host(m)[0]), -k[m] // 2)
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
