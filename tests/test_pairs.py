"""The row-pair kernels where they can go wrong: lines longer than a block
(taken in chunks), lines at the edges of a block, odd lines, and vectors whose
data starts at an odd element (no two-element loads).

SpMV, SYMGS (FP64 and BF16/FP32) and the V-cycles bit-exact against the
oracle's restatement of src/ComputeSPMV_ref.cpp:64-70,
src/ComputeSYMGS_ref.cpp:67-100 and src/ComputeMG_ref.cpp:39-63 in colour order.
Variable coefficients, so that a value taken from a wrong slot shows.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# x-lines of 255, 256, 257, 258 and 516 pairs, even and odd; one line; ragged;
# classes of more than 100,000 pairs, even and odd; many long lines, in chunks of
# 64 (FP64; BF16 one chunk), 128 (256), 64 (160) and 64 (192) pairs
GRIDS = [(510, 3, 3, 1), (511, 2, 3, 1), (512, 4, 2, 2), (514, 4, 4, 2), (1031, 3, 2, 1),
         (1032, 2, 2, 2), (513, 1, 1, 1), (34, 6, 10, 2), (256, 2, 6, 2),
         (130, 101, 100, 1), (131, 101, 101, 1),
         (384, 48, 48, 1), (700, 32, 32, 1), (514, 64, 64, 1), (1025, 46, 46, 1)]


def view(a, odd):
    """a on the device; odd: starting one element into its allocation."""
    t = torch.empty(len(a) + 1, dtype=torch.from_numpy(a[:1]).dtype, device="cuda")
    v = t[1:] if odd else t[:-1]
    v.copy_(torch.from_numpy(a))
    return v


def host(t):
    return t.detach().cpu().numpy()


@pytest.mark.parametrize("odd", [False, True], ids=["even", "odd"])
@pytest.mark.parametrize("dims", GRIDS, ids=lambda d: "x".join(map(str, d[:3])))
def test_pairs(oracle, dims, odd):
    from hpcg_b200 import Problem
    nx, ny, nz, levels = dims
    L, _, _, _ = oracle.hierarchy(nx, ny, nz, levels=levels, varcoef=(5, 0.5))
    oracle.colour_order(L)
    P = Problem(nx, ny, nz, levels=levels)
    for l, lev in enumerate(L):
        P.load_level(l, lev.nnz, lev.cols, lev.vals)
    P.build_mixed()
    n = L[0].nrow
    r, x0 = oracle.uniform(3, n, -1.0, 1.0), oracle.uniform(4, n, 1.0, 2.0)
    y = view(r, odd)
    assert (host(P.spmv(view(x0, odd), y=y)) == oracle.spmv(L[0], x0)).all()
    x = view(x0, odd)
    P.symgs(view(r, odd), x)
    assert (host(x) == oracle.symgs(L[0], r, x0, coloured=True)).all()
    x32 = x0.astype(np.float32)
    assert (host(P.spmv_mixed(view(x32, odd))) == oracle.spmv32(L[0], x32)).all()
    x = view(x32, odd)
    P.symgs_mixed(view(r, odd), x)
    assert (host(x) == oracle.symgs32(L[0], r, x32)).all()
    x = view(np.full(n, np.nan), odd)      # the first sweep reads nothing of x
    assert (host(P.mg(view(r, odd), x)) == oracle.mg(L, r, coloured=True)).all()
    x = view(np.full(n, np.nan, np.float32), odd)
    assert (host(P.mg_mixed(view(r, odd), x)) == oracle.mg32(L, r)).all()
    P.close()
