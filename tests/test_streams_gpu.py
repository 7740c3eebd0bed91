"""One plan called on two streams in turn, with no wait between the calls: they share the plan's working vectors, so
each must wait for the last, whether its launches go out directly (the one-launch solve, a first factorization) or
as a recorded graph (the per-level solve, a repeated factorization)."""
import numpy as np
import pytest

from sdsb200 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ir", [0, 1])
@pytest.mark.parametrize("structure", ["SPD", "G"])
def test_solves_on_two_streams(structure, ir):
    import torch

    from sdsb200._native import numeric_lib
    from sdsb200.solver import DirectSolver

    A = M.lap3d(24, 24, 24, seed=6) if structure == "SPD" else M.convection_diffusion3d(18, 18, 18, seed=6)
    n, nrhs = A.shape[0], 8
    ds = DirectSolver(A, structure, reordering_alg="nd", max_nrhs=nrhs, ir_n_steps=ir)
    ds.execute("analysis")
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    b = [torch.from_numpy(np.random.default_rng(q).uniform(-1, 1, (n, nrhs))).cuda() for q in range(2)]
    torch.cuda.synchronize()
    lib = numeric_lib()
    want = {}
    for mode in (1, 0):
        lib.sdsb200_set_persistent(ds._plan, mode)
        assert ds.execute("factorization") == 0
        for q in range(2):
            want[mode, q] = ds.execute("solve", None, b[q]).clone()
            torch.cuda.synchronize()
    got = []
    for rep in range(12):
        for q, mode in ((0, 1), (1, 1), (0, 0), (1, 1), (0, 1), (1, 0)):
            lib.sdsb200_set_persistent(ds._plan, mode)
            with torch.cuda.stream(streams[q]):
                got.append((mode, q, ds.execute("solve", None, b[q])))
                got[-1][2].record_stream(streams[q])
        with torch.cuda.stream(streams[rep % 2]):
            assert ds.execute("refactorization") == 0   # the same values, the same factor
    torch.cuda.synchronize()
    for mode, q, x in got:
        assert torch.equal(x, want[mode, q]), (mode, q)


def test_repeated_solves_record_a_graph():
    """The one-launch solve launches directly, then (32 calls in a row with the same buffers) as a graph; other buffers
    in between, a refinement step and another stream change nothing."""
    import torch

    from sdsb200.solver import DirectSolver

    A = M.lap3d(12, 12, 12, seed=6)
    n = A.shape[0]
    ds = DirectSolver(A, "SPD", reordering_alg="nd", max_nrhs=2, ir_n_steps=1)
    ds.execute("analysis")
    assert ds.execute("factorization") == 0
    b = [torch.from_numpy(np.random.default_rng(q).uniform(-1, 1, (n, 2))).cuda() for q in range(2)]
    x = [torch.empty_like(v) for v in b]
    want = [ds.execute("solve", None, v).clone() for v in b]
    other = torch.cuda.Stream()
    for q in [0] * 40 + [1] * 5 + [0] * 3 + [1] * 40 + [0, 1] * 4:
        x[q].fill_(7.0)
        torch.cuda.synchronize()
        with torch.cuda.stream(other if q else torch.cuda.current_stream()):
            ds.execute("solve", x[q], b[q])
        torch.cuda.synchronize()
        assert torch.equal(x[q], want[q])
