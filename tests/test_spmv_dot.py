"""CG's SpMV with its dot product (p.Ap, src/CG.cpp:119) on both sides of the row
count from which a launch of its own sums it, on even and odd grids, on one rank
and over slabs: the step length of the first unpreconditioned iteration,
alpha = b.b / b.Ab from x = 0, seen in x = alpha b.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

# 2^25 rows: 512 x 256 x 256 is the first with the launch, 508 the last without;
# odd lines, ragged groups and turns; and one plane of a little more
GRIDS = [(512, 256, 256), (508, 256, 256), (515, 257, 255), (514, 257, 254), (33, 17, 9)]


def step(b, x):
    """alpha of x = alpha b, the same for every entry that is not tiny."""
    i = int(b.abs().argmax())
    a = float(x[i] / b[i])
    assert torch.equal(x, a * b) or float((x - a * b).abs().max()) <= 1e-15 * abs(a) * float(b.abs().max())
    return a


@pytest.mark.parametrize("dims", GRIDS, ids=lambda d: "x".join(map(str, d)))
def test_one_rank(dims):
    from hpcg_b200 import Problem
    P = Problem(*dims, levels=1)
    P.generate("hpcg")
    b = P.fill_uniform(3, -1.0, 1.0)
    Ab = P.spmv(b)
    want = float(b @ b) / float(b @ Ab)
    seen = set()
    for _ in range(2):
        x = torch.zeros_like(b)
        k, _, nr0 = P.cg(b, x, 1, 1e-30, precond=False)
        assert k == 1 and abs(nr0 ** 2 / float(b @ b) - 1) <= 1e-13
        seen.add(step(b, x))
    # sums of up to 1e4 terms a block in FP64: a few 1e-14
    assert len(seen) == 1 and abs(seen.pop() / want - 1) <= 1e-13
    P.close()


def test_slabs():
    from hpcg_b200 import Group, Problem
    ps = [Problem(512, 512, 128, nranks=2, rank=r, levels=1) for r in range(2)]
    for p in ps:
        p.generate("hpcg")
    g = Group(ps)
    bs = [torch.rand(p.rows(), dtype=torch.float64, device="cuda") - 0.5 for p in ps]
    Ab = g.spmv(bs)
    want = sum(float(b @ b) for b in bs) / sum(float(b @ y) for b, y in zip(bs, Ab))
    xs = [torch.zeros_like(b) for b in bs]
    assert g.cg(bs, xs, 1, 1e-30, mode=0)[0] == 1
    for b, x in zip(bs, xs):
        assert abs(step(b, x) / want - 1) <= 1e-13
    g.close()
