"""The vector kernels at the edges of their tiles (1024 elements, four per
thread) and of the grid (592 blocks, above 2^23 elements 1184 and 740 for the dot
product; 1024 for the residual), with vectors on and off a two-element
boundary: WAXPBY bit-exact in its three branches
(src/ComputeWAXPBY_ref.cpp:52-67), in place as well; dot products
(src/ComputeDotProduct_ref.cpp:48-63) to 1e-13 of the exactly rounded sum of
products, the same bits wherever the vectors start; the residual exact.
"""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# more than 2^23 elements: the larger grid, at its edge and with several tiles a block
LARGE = [1 << 23, (1 << 23) + 1, 740 * 1024 * 12 + 1, 1184 * 1024 * 8 - 1,
         1184 * 1024 * 8 + 513]
SIZES = [1, 2, 255, 1023, 1024, 1025, 2047, 2051, 592 * 1024 - 1, 592 * 1024 + 1,
         1024 * 1024 - 1, 1024 * 1024 + 1, 1184 * 1024 + 513]


@pytest.fixture(scope="module")
def P():
    from hpcg_b200 import Problem
    p = Problem(128, 128, 80, levels=1)
    yield p
    p.close()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("odd", [(0, 0, 0), (1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)],
                         ids=lambda o: "".join(map(str, o)))
def test_vectors(P, n, odd):
    g = torch.Generator(device="cuda").manual_seed(n)
    buf = [torch.empty(n + 2, dtype=torch.float64, device="cuda").uniform_(-1, 1, generator=g)
           for _ in odd]
    x, y, w = (b[o:o + n] for b, o in zip(buf, odd))
    hx, hy = x.cpu().numpy(), y.cpu().numpy()
    for a, b in ((1.0, 0.3), (-0.7, 1.0), (0.7, -1.3), (1.0, 1.0)):
        edge = [t.clone() for t in buf]
        want = (hx if a == 1.0 else a * hx) + (b * hy if b != 1.0 or a == 1.0 else hy)
        P.waxpby(a, x, b, y, w=w)
        assert (w.cpu().numpy() == want).all()
        assert torch.equal(buf[2][:odd[2]], edge[2][:odd[2]])
        assert torch.equal(buf[2][odd[2] + n:], edge[2][odd[2] + n:])
    z = x.clone()
    P.waxpby(0.7, z, -1.3, y, w=z)
    assert (z.cpu().numpy() == 0.7 * hx + -1.3 * hy).all()
    want = math.fsum((hx * hy).tolist())
    # each product and the running sums of at most n / 256 terms round once
    got = P.dot(x, y)
    assert abs(got - want) <= 1e-13 * np.abs(hx * hy).sum()
    # the order of the sum is the length's, not that of where the vectors start
    assert got == P.dot(x.clone(), y.clone())
    assert P.residual(x, y) == np.abs(hx - hy).max()


@pytest.fixture(scope="module")
def large():
    from hpcg_b200 import Problem
    p = Problem(256, 256, 160, levels=1)
    yield p
    p.close()


@pytest.mark.parametrize("n", LARGE)
def test_large_vectors(large, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    x, y, w = (torch.empty(n + 2, dtype=torch.float64, device="cuda").uniform_(-1, 1, generator=g)
               for _ in range(3))
    hx, hy = x.cpu().numpy(), y.cpu().numpy()
    # sums of at most n / (740 * 256) + 1 products a thread, and of the threads'
    want = float(np.sum(hx[:n].astype(np.longdouble) * hy[1:n + 1]))
    bound = 1e-13 * float(np.abs(hx[:n] * hy[1:n + 1]).sum())
    got = large.dot(x[:n], y[1:n + 1])
    assert abs(got - want) <= bound
    assert got == large.dot(x[:n], y[1:n + 1].clone())
    for odd in (0, 1):
        v, end = w[odd:odd + n], w.clone()
        large.waxpby(0.7, x[:n], -1.3, y[odd:odd + n], w=v)
        assert (v.cpu().numpy() == 0.7 * hx[:n] - 1.3 * hy[odd:odd + n]).all()
        assert torch.equal(w[:odd], end[:odd]) and torch.equal(w[odd + n:], end[odd + n:])
    assert large.residual(x[:n], y[1:n + 1]) == np.abs(hx[:n] - hy[1:n + 1]).max()
