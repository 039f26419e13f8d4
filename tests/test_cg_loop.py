"""The solver's host loop: without a times array an iteration is queued ahead
and the state read from pinned memory, with one the host waits for each
iteration.  Both must stop at the same iteration with the same bits, wherever
the stop falls: at the initial residual, in the first iterations, at max_iter,
at the tolerance.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STOPS = [(0, 1e-10), (1, 1e-10), (2, 1e-10), (3, 1e-10), (500, 1e-10), (500, 0.999), (4, 0.0),
         (500, 1.0)]


def problem(kind):
    from hpcg_b200 import Problem
    if kind != "general":
        P = Problem(16, 8, 24, levels=3)
        P.generate("varcoef", seed=3, sigma=0.5)
        return P
    n = 300                    # a path graph's Laplacian + I
    P = Problem.general(levels=1)
    i = np.arange(n)
    cols = np.stack([np.maximum(i - 1, 0), i, np.minimum(i + 1, n - 1)], 1)
    vals = np.tile([-1.0, 3.0, -1.0], (n, 1))
    nnz = np.full(n, 3, np.uint8)
    cols[0, :2], vals[0, :2], nnz[0] = [0, 1], [3.0, -1.0], 2
    nnz[-1] = 2
    P.load_level_general(0, nnz, cols, vals)
    return P


@pytest.mark.parametrize("kind", ["fp64", "plain", "mixed", "general"])
def test_stops(kind):
    from hpcg_b200 import HPCGXError
    P = problem(kind)
    b = P.fill_uniform(5, -1.0, 1.0)

    def go(rhs, max_iter, tol, times):
        x = torch.zeros_like(rhs)
        if kind == "mixed":
            return P.cg_mixed(rhs, x, max_iter, tol, times=times), x
        return P.cg(rhs, x, max_iter, tol, precond=kind != "plain", times=times), x

    for rhs in (b, torch.zeros_like(b)):
        for max_iter, tol in STOPS:
            (k, nr, nr0), x = go(rhs, max_iter, tol, None)
            (k2, mr, mr0), y = go(rhs, max_iter, tol, np.zeros(6))
            assert (k, nr, nr0) == (k2, mr, mr0) and torch.equal(x, y)
            assert k <= max_iter
    bad = b.clone()
    bad[7] = float("nan")
    for times in (None, np.zeros(6)):
        with pytest.raises(HPCGXError):
            go(bad, 500, 1e-10, times)
    (k, nr, nr0), _ = go(b, 500, 1e-10, None)      # usable afterwards
    assert 0 < k < 500 and nr <= 1e-10 * nr0
    P.close()
