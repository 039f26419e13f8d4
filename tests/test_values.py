"""Row-major values in and out of the device layout on ragged grids: blocks of 64
rows that end inside a line, lines of odd length, grids smaller than a block.

set_values -> get_values returns the input wherever the stencil has a neighbour
and 0 elsewhere, with the neighbour (or the row itself) as column; the adjoint
gradient is -lambda_i x_j there and 0 elsewhere, bit for bit; coarse levels take
the injected edges; the BF16 copy is torch's rounding of the values.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,levels", [((1, 1, 1), 1), ((3, 1, 2), 1), ((5, 7, 3), 1), ((64, 2, 2), 2),
                                         ((65, 3, 2), 1), ((33, 9, 5), 1), ((16, 24, 8), 4),
                                         ((130, 6, 4), 2), ((1, 40, 30), 1), ((130, 1, 4), 1),
                                         ((70, 33, 1), 1), ((1, 1, 200), 1)])
def test_values(dims, levels):
    from hpcg_b200 import Problem
    nx, ny, nz = dims
    n = nx * ny * nz
    g = torch.Generator(device="cuda").manual_seed(n)
    v = torch.empty(n, 27, dtype=torch.float64, device="cuda").uniform_(-2, -1, generator=g)
    P = Problem(nx, ny, nz, levels=levels)
    P.set_values(v.reshape(-1), level=0, recoarsen=True)     # nothing generated before
    row = torch.arange(n, device="cuda")
    ix, iy, iz = row % nx, (row // nx) % ny, row // (nx * ny)
    has, col = torch.zeros(n, 27, dtype=torch.bool, device="cuda"), row[:, None].repeat(1, 27)
    for s in range(27):
        dx, dy, dz = s % 3 - 1, (s // 3) % 3 - 1, s // 9 - 1
        has[:, s] = ((ix + dx >= 0) & (ix + dx < nx) & (iy + dy >= 0) & (iy + dy < ny) &
                     (iz + dz >= 0) & (iz + dz < nz))
        col[:, s] = torch.where(has[:, s], row + (dz * ny + dy) * nx + dx, row)
    want = torch.where(has, v, 0.0)
    out, cols = P.get_values(0)
    assert torch.equal(out, want) and torch.equal(cols, col.to(torch.int32))
    lam = torch.empty(n, dtype=torch.float64, device="cuda").uniform_(-1, 1, generator=g)
    x = torch.empty(n, dtype=torch.float64, device="cuda").uniform_(-1, 1, generator=g)
    assert torch.equal(P.adjoint_grad(lam, x), torch.where(has, -(lam[:, None] * x[col]), 0.0))
    # BF16 values through the product with a unit vector per colour of rows
    P.build_mixed()
    e = torch.zeros(n, dtype=torch.float32, device="cuda")
    e[n // 2] = 1.0
    y = P.spmv_mixed(e)
    hit = (col == n // 2) & has
    assert torch.equal(y, torch.where(hit, want.to(torch.bfloat16).to(torch.float32), 0.0).sum(1))
    # coarse levels: an edge takes the value of the edge that leaves its lower
    # injected point in its direction; no slot is left unwritten
    for l in range(levels - 1):
        fine, (cv, cc) = P.get_values(l)[0], P.get_values(l + 1)
        mx, my, mz = P.level_dims(l + 1)
        fx, fy, _ = P.level_dims(l)
        r = torch.arange(mx * my * mz, device="cuda")
        jx, jy, jz = r % mx, (r // mx) % my, r // (mx * my)
        f = (2 * jz * fy + 2 * jy) * fx + 2 * jx
        total = torch.zeros(r.numel(), dtype=torch.float64, device="cuda")
        for s in range(27):
            if s == 13:
                continue
            there = cc[:, s] != r
            src = f if s > 13 else f[torch.where(there, cc[:, s].long(), r)]
            w = torch.where(there, fine[src, s if s > 13 else 26 - s], 0.0)
            assert torch.equal(cv[:, s], w)
            total += w.abs()
        assert torch.equal(cv[:, 13], total + 2.0)
    P.close()
