"""A symbolic factorization made by hand, whose child lists its rows below the pivot block in another order than its
parent has them: the shared-memory kernel takes any order, so fronts that fit it must go there, whatever the
line between the kernels is for the analysis' own plans. "G" only: a symmetric front's stored triangle fixes the
order."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdsb200 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [40, 80, 120, 150])   # rows of the parent
def test_unordered_child_rows(s):
    from sdsb200.solver import DirectSolver

    rng = np.random.default_rng(s)
    w, leaves = 10, 3
    n = leaves * w + s
    mask = np.zeros((n, n), bool)
    mask[leaves * w:, leaves * w:] = True
    for q in range(leaves):
        own = np.arange(q * w, (q + 1) * w)
        rows = leaves * w + rng.choice(s, 35, replace=False)
        mask[np.ix_(own, own)] = mask[np.ix_(own, rows)] = mask[np.ix_(rows, own)] = True
    B = rng.uniform(-1, 1, (n, n)) * mask + n * np.eye(n)
    A = sp.csr_matrix(B)
    A.sort_indices()
    b = M.rhs(n, 2, seed=1)
    ds = DirectSolver(A, "G", max_nrhs=2)
    ds.execute("reordering")
    m = ds.symbolic.maps
    fptr, sptr, rptr = m["front_ptr"] - 1, m["super_ptr"] - 1, m["rowptr"] - 1
    done = 0
    for c in range(ds.symbolic.ns):
        f, wc = rptr[c + 1] - rptr[c], sptr[c + 1] - sptr[c]
        if m["child_ptr"][c + 1] > m["child_ptr"][c] or m["snparent"][c] <= 0 or f - wc < 2:
            continue
        to = rng.permutation(f - wc)            # row t goes to place to[t]
        for name, begin in (("rowval", rptr[c] + wc), ("relind", m["relind_ptr"][c] - 1)):
            v = m[name][begin: begin + f - wc].copy()
            m[name][begin + to] = v
        for k in range(m["amap_ptr"][c] - 1, m["amap_ptr"][c + 1] - 1):
            p = m["amap_src"][k] - 1
            loc = abs(m["amap"][p]) - 1 - fptr[c]
            i, j = loc % f, loc // f
            if i >= wc:
                m["amap"][p] = np.sign(m["amap"][p]) * (fptr[c] + wc + to[i - wc] + j * f + 1)
        done += 1
    assert done >= 2
    ds.execute("symbolic_factorization")
    assert ds.execute("factorization") == 0
    x = ds.execute("solve", None, b).cpu().numpy()
    assert M.scaled_backward_error(A, x, b) <= 1e-12
