"""General-pattern rows around the kernels' chunk of 27 entries: rows of 1 to 70
entries in one matrix, levels smaller than a slice and not a multiple of one,
an injection in any order.

SpMV, SYMGS and the V-cycle bit-exact against the oracle's restatement of
src/ComputeSPMV_ref.cpp:58-71, src/ComputeSYMGS_ref.cpp:67-100 (colour order of
src/OptimizeProblem.cpp:50-79) and src/ComputeMG_ref.cpp:39-63 -- here in numpy,
since the oracle's rows hold 27 entries at most.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def random_level(n, most, seed):
    """Symmetric weighted graph Laplacian + I with up to `most` entries per row."""
    rng = np.random.default_rng(seed)
    nb = [dict() for _ in range(n)]
    hubs = rng.choice(n, size=max(1, n // 10), replace=False)
    for i in range(n):
        want = int(rng.integers(0, most)) if i in hubs else int(rng.integers(0, 4))
        for j in rng.integers(0, n, size=want):
            if j != i and len(nb[i]) < most - 1 and len(nb[j]) < most - 1:
                nb[i][int(j)] = nb[j][i] = float(rng.uniform(0.5, 2.0))
    w = max(len(r) for r in nb) + 1
    cols, vals = np.zeros((n, w), np.int32), np.zeros((n, w))
    nnz = np.zeros(n, np.uint8)
    for i in range(n):
        row = sorted(list(nb[i]) + [i])
        nnz[i] = len(row)
        cols[i, :len(row)] = row
        vals[i, :len(row)] = [1.0 + sum(nb[i].values()) if j == i else -nb[i][j] for j in row]
    return nnz, cols, vals


def spmv(A, x):
    nnz, cols, vals = A
    y = np.zeros(len(nnz))
    for i in range(len(nnz)):
        s = 0.0
        for j in range(nnz[i]):
            s += vals[i, j] * x[cols[i, j]]
        y[i] = s
    return y


def colours(A):
    nnz, cols, _ = A
    c = np.zeros(len(nnz), int)
    for i in range(1, len(nnz)):
        used = {c[j] for j in cols[i, :nnz[i]] if j < i}
        c[i] = next(k for k in range(i + 1) if k not in used)
    return c


def symgs(A, r, x):
    nnz, cols, vals = A
    x, c = x.copy(), colours(A)
    order = np.argsort(c, kind="stable")
    for i in list(order) + list(order[::-1]):
        s = r[i]
        for j in range(nnz[i]):
            s -= vals[i, j] * x[cols[i, j]]
        d = vals[i, list(cols[i, :nnz[i]]).index(i)]
        s += x[i] * d
        x[i] = s / d
    return x


def mg(levels, l, r):
    A, f2c = levels[l]
    x = symgs(A, r, np.zeros(len(r)))
    if l + 1 < len(levels):
        rc = r[f2c] - spmv(A, x)[f2c]
        xc = mg(levels, l + 1, rc)
        x[f2c] = x[f2c] + xc
        x = symgs(A, r, x)
    return x


@pytest.mark.parametrize("sizes,most", [((1,), 1), ((31,), 5), ((33, 7), 27), ((500, 61, 9), 28),
                                        ((1200, 200), 70), ((2049, 2048, 300), 40)])
def test_rows(sizes, most):
    from hpcg_b200 import Problem
    rng = np.random.default_rng(sum(sizes) + most)
    levels = []
    for l, n in enumerate(sizes):
        f2c = None
        if l + 1 < len(sizes):
            f2c = rng.choice(n, size=sizes[l + 1], replace=False).astype(np.int32)
        levels.append((random_level(n, most, 10 * l + n), f2c))
    P = Problem.general(levels=len(sizes))
    for l, ((nnz, cols, vals), f2c) in enumerate(levels):
        P.load_level_general(l, nnz, cols, vals, f2c)
    for l, (A, _) in enumerate(levels):
        n = sizes[l]
        x, r = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        assert (P.spmv(torch.from_numpy(x).cuda(), level=l).cpu().numpy() == spmv(A, x)).all()
        y = torch.from_numpy(x).cuda()
        P.symgs(torch.from_numpy(r).cuda(), y, level=l)
        assert (y.cpu().numpy() == symgs(A, r, x)).all()
    r = rng.uniform(-1, 1, sizes[0])
    assert (P.mg(torch.from_numpy(r).cuda()).cpu().numpy() == mg(levels, 0, r)).all()
    P.close()
