"""Matrices whose rows leave out entries of existing neighbours.

The host loaders accept a stencil row that skips slots, and one that stores a
coupling of value 0.  Columns are not stored; the level keeps which slots a row
leaves out.  A left-out slot reads the row itself, as a slot without a neighbour
does, also where the neighbour's entry is not finite; a stored 0 keeps its
column, in the products (0 times infinity), in get_values and in the gradient.
"""
import copy

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


def edit(lev, leave_out=(), zero=()):
    """A copy of a level without the couplings in leave_out and with value 0 for
    those in zero, both sets of pairs i < j."""
    n, out = lev.nrow, copy.copy(lev)
    cols, vals, nnz = lev.cols.reshape(n, 27).copy(), lev.vals.reshape(n, 27).copy(), lev.nnz.copy()
    diag = lev.diag.copy()
    for i in range(n):
        pair = [(min(i, int(c)), max(i, int(c))) for c in cols[i, :nnz[i]]]
        vals[i, [j for j, e in enumerate(pair) if e in zero]] = 0.0
        keep = [j for j, e in enumerate(pair) if e not in leave_out]
        m = len(keep)
        cols[i, :m], vals[i, :m] = cols[i, keep], vals[i, keep]
        cols[i, m:], vals[i, m:], nnz[i] = i, 0.0, m
        diag[i] = keep.index(diag[i])
    out.cols, out.vals, out.nnz, out.diag = cols.reshape(-1), vals.reshape(-1), nnz, diag
    return out


def couplings(lev):
    n = lev.nrow
    cols = lev.cols.reshape(n, 27)
    return [(i, int(c)) for i in range(n) for c in cols[i, :lev.nnz[i]] if c > i]


def slots(lev):
    """Columns and presence of every slot: the row itself where it has no entry."""
    n = lev.nrow
    c, there = np.repeat(np.arange(n)[:, None], 27, 1), np.zeros((n, 27), bool)
    for i in range(n):
        for j in lev.cols.reshape(n, 27)[i, :lev.nnz[i]]:
            dz, dy, dx = (int(a) - int(b) for a, b in
                          zip(np.unravel_index(j, (lev.nz, lev.ny, lev.nx)),
                              np.unravel_index(i, (lev.nz, lev.ny, lev.nx))))
            s = (dz + 1) * 9 + (dy + 1) * 3 + dx + 1
            c[i, s], there[i, s] = j, True
    return c, there


def same(got, want):
    return np.array_equal(got.cpu().numpy(), want, equal_nan=True)


# even and odd lines; lines in chunks, whose last class is swept a second time
@pytest.mark.parametrize("dims", [(16, 8, 8), (9, 7, 5), (514, 4, 4)])
def test_stored_zeros_beside_left_out_entries(oracle, dims):
    from hpcg_b200 import Problem
    L, _, _, _ = oracle.hierarchy(*dims, levels=1, varcoef=(5, 0.5))
    oracle.colour_order(L)
    n = L[0].nrow
    rng = np.random.default_rng(7)
    kinds = [(e, rng.random()) for e in couplings(L[0])]
    gone = {e for e, u in kinds if u < 0.1}
    zero = {e for e, u in kinds if 0.1 <= u < 0.3}
    lev = edit(L[0], gone, zero)
    P = Problem(*dims, levels=1)
    P.load_level(0, lev.nnz, lev.cols, lev.vals)
    c, there = slots(lev)
    assert np.array_equal(P.get_values(0)[1].cpu().numpy(), c)
    # the gradient: the neighbour's entry where the row has one, the row's own
    # where it leaves it out, 0 where there is no neighbour
    lam, x = oracle.uniform(8, n, -1.0, 1.0), oracle.uniform(9, n, -1.0, 1.0)
    want = np.where(there | slots(L[0])[1], -(lam[:, None] * x[c]), 0.0)
    dlam, dx = torch.from_numpy(lam).cuda(), torch.from_numpy(x).cuda()
    assert same(P.adjoint_grad(dlam, dx), want)
    assert same(P.spmv(dx), oracle.spmv(lev, x))
    y = dx.clone()
    assert same(P.symgs(dlam, y), oracle.symgs(lev, lam, x, coloured=True))
    for i in rng.integers(0, n, 3):
        x[i] = np.inf
    want = oracle.spmv(lev, x)
    assert not np.isfinite(want).all() and same(P.spmv(torch.from_numpy(x).cuda()), want)
    P.close()


@pytest.mark.parametrize("iz", [2, 3])      # a line of class 1, and of class 3
@pytest.mark.parametrize("dims", [(16, 8, 8), (514, 4, 4), (12, 12, 12)])
def test_sweeps_keep_to_the_entries(oracle, dims, iz):
    """Three rows cut off from all others by left-out entries, two of them coupled
    by a stored 0: what is not finite there stays there."""
    from hpcg_b200 import Problem
    L, _, _, _ = oracle.hierarchy(*dims, levels=2)
    oracle.colour_order(L)
    nx, ny, nz = dims
    a = (iz * ny + 3) * nx + nx // 2 + 1
    rows = (a, a + 1, a - 4)
    gone = {e for e in couplings(L[0]) if (e[0] in rows or e[1] in rows) and e != (a, a + 1)}
    fine = edit(L[0], gone, {(a, a + 1)})
    P = Problem(*dims, levels=2)
    for l, lev in enumerate((fine, L[1])):
        P.load_level(l, lev.nnz, lev.cols, lev.vals)
    n = fine.nrow
    r, x = oracle.uniform(3, n, -1.0, 1.0), oracle.uniform(4, n, -1.0, 1.0)
    x[a] = x[a - 4] = np.inf
    want = oracle.symgs(fine, r, x, coloured=True)
    assert sorted(np.flatnonzero(~np.isfinite(want))) == sorted(rows)
    assert same(P.symgs(torch.from_numpy(r).cuda(), torch.from_numpy(x).cuda()), want)
    # the V-cycle from a right-hand side that is not finite there
    r[a] = np.inf
    want = oracle.mg([fine, L[1]], r, coloured=True)
    assert sorted(np.flatnonzero(~np.isfinite(want))) == [a, a + 1]
    assert same(P.mg(torch.from_numpy(r).cuda()), want)
    P.close()


@pytest.mark.parametrize("times", [False, True], ids=["ahead", "timed"])
def test_a_solve_follows_the_matrix(oracle, times):
    """One Problem, loaded with full and with holed matrices in turn: its captured
    iteration has the kernels of the matrix that is loaded.  iteration_bytes tells
    them apart: those of a holed level read 4 B per row and launch more."""
    from hpcg_b200 import Problem
    from hpcg_b200._lib import CG_MG
    dims = (16, 8, 8)
    full, _, _, _ = oracle.hierarchy(*dims, levels=2)
    n = full[0].nrow
    some = couplings(full[0])[::5]
    holed = [edit(full[0], set(some)), full[1]]
    b = torch.from_numpy(oracle.uniform(3, n, -1.0, 1.0)).cuda()

    def load(p, levels):
        for l, lev in enumerate(levels):
            p.load_level(l, lev.nnz, lev.cols, lev.vals)
        return p

    def solve(p):
        x = torch.zeros_like(b)
        out = p.cg(b, x, 50, 1e-10, times=np.zeros(6) if times else None)
        return out, x, p.iteration_bytes(CG_MG)

    P = Problem(*dims, levels=2)
    got = [solve(load(P, levels)) for levels in (full, holed, full, holed)]
    for k in (0, 1):
        fresh = solve(load(Problem(*dims, levels=2), (full, holed)[k]))
        for g in got[k::2]:
            assert g[0] == fresh[0] and torch.equal(g[1], fresh[1]) and g[2] == fresh[2]
    # two sweeps in which classes 0..2 (a quarter of the rows each) are launched
    # twice and class 3 once, and the SpMV
    assert got[1][2] - got[0][2] == 4 * n * (2 * 1.75 + 1)
    P.generate("hpcg")
    assert solve(P)[2] == got[0][2]
    P.close()
