"""hpcgx_iteration_bytes against a count of its own: the values that each launch
of an iteration multiplies (a zero-guess class launch those of the lower colours
and the diagonal), and the rows of the vectors that it updates.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def colour_counts(nx, ny, nz):
    """Per colour: rows, values, and values of the diagonal and the lower colours."""
    iz, iy, ix = (a.reshape(-1) for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx),
                                                     indexing="ij"))
    colour = (ix & 1) + 2 * (iy & 1) + 4 * (iz & 1)
    out = np.zeros((8, 3), np.int64)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                x, y, z = ix + dx, iy + dy, iz + dz
                there = (x >= 0) & (x < nx) & (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
                other = (x & 1) + 2 * (y & 1) + 4 * (z & 1)
                low = there & ((other < colour) | ((dx == 0) & (dy == 0) & (dz == 0)))
                for c in range(8):
                    out[c, 1] += (there & (colour == c)).sum()
                    out[c, 2] += (low & (colour == c)).sum()
    for c in range(8):
        out[c, 0] = (colour == c).sum()
    return out


def sweep_bytes(cnt, value, vec, rhs, zero, transfer):
    """A symmetric sweep in its 7 launches: classes 0, 1, 2, the last class in both
    directions, classes 2, 1, 0.  transfer: colour 0 reads or writes one vector
    more (restriction, prolongation)."""
    total = 0
    for q, first in ((0, zero), (1, zero), (2, zero), (3, False), (2, False), (1, False), (0, False)):
        for c in (2 * q, 2 * q + 1):
            rows, values, low = cnt[c]
            total += value * (low if first else values) + rows * (rhs + vec)
            # the row's own entry is read unless the sweep starts from zero
            total += 0 if (first or (q == 3 and zero)) else rows * vec
    return total + (cnt[0][0] * vec if transfer else 0)


def vcycle_bytes(dims, levels, value, vec):
    total = 0
    for l in range(levels):
        cnt = colour_counts(*(d >> l for d in dims))
        last = l + 1 == levels
        total += sweep_bytes(cnt, value, vec, vec, True, not last)
        if not last:
            total += sweep_bytes(cnt, value, vec, vec, False, True)
    return total


@pytest.mark.parametrize("dims,levels", [((16, 8, 8), 1), ((16, 24, 8), 3), ((9, 7, 5), 1)])
def test_iteration_bytes(dims, levels):
    from hpcg_b200 import Problem
    from hpcg_b200._lib import CG_MG, CG_MIXED, CG_PLAIN
    P = Problem(*dims, levels=levels)
    P.generate("hpcg")
    b = P.fill_uniform(3, -1.0, 1.0)
    n = P.rows()
    nnz = int(colour_counts(*dims)[:, 1].sum())
    spmv = 8 * nnz + 16 * n
    x = torch.zeros_like(b)
    P.cg(b, x, 2, 1e-10, precond=False)
    P.cg(b, x, 2, 1e-10)
    P.cg_mixed(b, x, 2, 1e-10)
    # per row: z = r; r.z; p = z + beta p with the deferred x += alpha p; r -= alpha Ap
    assert P.iteration_bytes(CG_PLAIN) == spmv + n * (16 + 16 + 40 + 24)
    assert P.iteration_bytes(CG_MG) == spmv + n * (16 + 40 + 24) + vcycle_bytes(dims, levels, 8, 8)
    # z in FP32, z.Ap as well, and r's FP32 copy
    assert P.iteration_bytes(CG_MIXED) == spmv + n * (20 + 36 + 28) + vcycle_bytes(dims, levels, 2, 4)
    P.close()
