"""Matrices whose rows leave out entries of existing neighbours.

The host loaders accept a stencil row that skips slots.  Columns are not
stored, so such a slot is told from a coupling of value 0 by the level's
"holes" flag: it must read the row itself, as a slot without a neighbour does,
also where the neighbour's entry is not finite.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def with_holes(lev, seed, share):
    """A copy of a level with a random symmetric set of couplings left out."""
    rng = np.random.default_rng(seed)
    n = lev.nrow
    cols, vals, nnz = lev.cols.reshape(n, 27).copy(), lev.vals.reshape(n, 27).copy(), lev.nnz.copy()
    gone = {(i, int(c)) for i in range(n) for c in cols[i, :nnz[i]] if c > i and rng.random() < share}
    for i in range(n):
        keep = [j for j in range(nnz[i])
                if (min(i, cols[i, j]), max(i, cols[i, j])) not in gone]
        m = len(keep)
        cols[i, :m], vals[i, :m] = cols[i, keep], vals[i, keep]
        cols[i, m:], vals[i, m:], nnz[i] = i, 0.0, m
    return nnz, cols, vals


def product(nnz, cols, vals, x):
    """Row sums from 0 over the entries in order (src/ComputeSPMV_ref.cpp:64-70)."""
    y = np.zeros(len(nnz))
    for j in range(27):
        on = j < nnz
        y[on] = y[on] + vals[on, j] * x[cols[on, j]]
    return y


@pytest.mark.parametrize("dims", [(16, 8, 8), (9, 7, 5), (33, 5, 4)])
def test_left_out_entries(oracle, dims):
    from hpcg_b200 import Problem
    L, _, _, _ = oracle.hierarchy(*dims, levels=1)
    nnz, cols, vals = with_holes(L[0], 3, 0.2)
    n = L[0].nrow
    P = Problem(*dims, levels=1)
    P.load_level(0, nnz, cols.reshape(-1), vals.reshape(-1))
    x = oracle.uniform(4, n, -1.0, 1.0)
    assert (P.spmv(torch.from_numpy(x).cuda()).cpu().numpy() == product(nnz, cols, vals, x)).all()
    c = P.get_values(0)[1].cpu().numpy()
    for i in range(n):   # the row's own entries, and the row itself in every other slot
        assert sorted(c[i][c[i] != i]) == sorted(j for j in cols[i, :nnz[i]] if j != i)
    # an infinite x reaches the rows that have an entry for it and no other
    i = n // 2
    x[i] = np.inf
    y = P.spmv(torch.from_numpy(x).cuda()).cpu().numpy()
    want = np.isfinite(product(nnz, cols, vals, x))
    assert (np.isfinite(y) == want).all()
    # values written later fill the whole stencil again
    full = Problem(*dims, levels=1)
    full.generate("hpcg")
    P.set_values(full.get_values(0)[0].reshape(-1), level=0)
    assert torch.equal(P.get_values(0)[1], full.get_values(0)[1])
