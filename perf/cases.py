"""The work whose speed this repository is judged by: listed cases, and draws from the same ranges.

A user of the framework solves HPCG systems (FP64 and mixed precision, to a tolerance or for a fixed
number of iterations), applies its operators one by one, differentiates through a solve, and solves
systems whose matrix has no grid order.  A case is a dict of plain values:

  op        "cg" (MG-PCG), "mg" (one V-cycle), "operators" (SpMV, a smoothing step, a dot product and a
            WAXPBY, called one after another), "gradient" (a solve and its adjoint through autograd)
  matrix    "hpcg" (26 / -1), "varcoef" (a_ij = -exp(sigma z) per edge, diagonal sum|a_ij| + 2) or
            "renumbered" (the HPCG hierarchy with every level's rows in a random order, a general-pattern
            problem)
  nx ny nz  the finest grid, coarsened levels - 1 times
  mixed     BF16/FP32 V-cycle (inside FP64 CG) instead of the FP64 one
  max_iter, tol   the solver's arguments; tol = 0 runs max_iter iterations
"""
import math

import numpy as np
import torch

from hpcg_b200 import Problem, solve

OFFSETS = [(s // 9 - 1, (s // 3) % 3 - 1, s % 3 - 1) for s in range(27)]   # (dz, dy, dx) of slot s
DIAG = 13


def case(name, op, dims, matrix="hpcg", mixed=False, levels=4, sigma=0.0, max_iter=0, tol=0.0):
    c = {"op": op, "matrix": matrix, "nx": dims[0], "ny": dims[1], "nz": dims[2], "levels": levels,
         "mixed": mixed, "sigma": sigma, "max_iter": max_iter, "tol": tol}
    return dict(c, name=name) if name else c


def listed():
    return [
        # HPCG's smallest local grid, solved to 1e-10: what a unit test or a coarse inner solve costs
        case("solve-16", "cg", (16, 16, 16), max_iter=500, tol=1e-10),
        # HPCG's default local grid, one timed set of the benchmark: 50 iterations at tolerance 0
        case("set-104", "cg", (104, 104, 104), max_iter=50),
        # one timed set on the grid that the drop-in and the operator tests use at full size
        case("set-256", "cg", (256, 256, 256), max_iter=50),
        # a small system through the mixed-precision solver, to the benchmark's tolerance
        case("mixed-solve-64", "cg", (64, 64, 64), mixed=True, max_iter=500, tol=1e-10),
        # the benchmark's solver on a grid of the benchmark's kind (b = A u, x0 = 0, tolerance 1e-10),
        # stopped after 25 iterations
        case("mixed-384", "cg", (384, 384, 384), mixed=True, max_iter=25, tol=1e-10),
        # the preconditioner alone, for a Krylov method of the user's own: FP64, variable coefficients
        case("vcycle-192x160x128", "mg", (192, 160, 128), matrix="varcoef", sigma=0.5),
        # the same in mixed precision on the grid that the sweep profiles use
        case("mixed-vcycle-256x256x128", "mg", (256, 256, 128), mixed=True),
        # operator by operator: a ragged single-level grid, where a call's latency is what counts
        case("operators-65x13x11", "operators", (65, 13, 11), levels=1),
        # operator by operator on an ordinary grid with variable coefficients
        case("operators-128", "operators", (128, 128, 128), matrix="varcoef", sigma=0.5),
        # the differentiable solve, FP64: forward, adjoint and both gradients
        case("gradient-128", "gradient", (128, 128, 128), matrix="varcoef", sigma=0.5, max_iter=2000,
             tol=1e-12),
        # the same in mixed precision on a rougher medium and a grid of unequal sides
        case("mixed-gradient-192x160x96", "gradient", (192, 160, 96), matrix="varcoef", mixed=True,
             sigma=1.0, max_iter=2000, tol=1e-10),
        # a system without grid order: the general sparse path
        case("renumbered-48", "cg", (48, 48, 48), matrix="renumbered", max_iter=500, tol=1e-10),
    ]


def draw(rng):
    """One more case of the listed ones' ranges: any grid whose rows lie between a few hundred and the
    listed largest of its kind, sides up to 8 : 1, odd sides where it isn't coarsened."""
    kinds = [("cg", "hpcg", False, 256), ("cg", "hpcg", True, 384), ("cg", "varcoef", False, 160),
             ("mg", "hpcg", False, 224), ("mg", "varcoef", False, 192), ("mg", "hpcg", True, 224),
             ("operators", "hpcg", False, 192), ("operators", "varcoef", False, 160),
             ("gradient", "varcoef", False, 128), ("gradient", "varcoef", True, 144),
             ("cg", "renumbered", False, 48)]
    op, matrix, mixed, top = rng.choice(kinds)
    levels = rng.choice([4, 4, 4, 3, 2, 1]) if op in ("cg", "mg") and matrix != "renumbered" else 4
    if op == "operators":
        levels = rng.choice([1, 1, 4])
    unit = 1 << (levels - 1)
    side = math.exp(rng.uniform(math.log(16), math.log(top)))
    a, b = rng.uniform(-1, 1) * math.log(2), rng.uniform(-1, 1) * math.log(2)
    shape = [side * math.exp(v) for v in (a, b, -a - b)]
    dims = [max(1, int(v / unit)) * unit for v in shape]   # rounded down: never above the top
    sigma = rng.choice([0.25, 0.5, 1.0]) if matrix == "varcoef" else 0.0
    if op == "gradient":
        return case(None, op, dims, matrix, mixed, levels, sigma, 2000, 1e-10)
    if op == "cg":
        cap = 25 if side > 256 else 50
        fixed = rng.random() < 0.5
        return case(None, op, dims, matrix, mixed, levels, sigma, cap, 0.0 if fixed and side > 64 else 1e-10)
    return case(None, op, dims, matrix, mixed, levels, sigma)


# ------------------------------------------------------------------ inputs

def generator(seed, salt, device):
    return torch.Generator(device=device).manual_seed(1000003 * int(seed) + salt)


def uniform(seed, salt, n, device, lo=-1.0, hi=1.0):
    return torch.rand(n, dtype=torch.float64, device=device,
                      generator=generator(seed, salt, device)) * (hi - lo) + lo


def level_dims(c):
    return [(c["nx"] >> l, c["ny"] >> l, c["nz"] >> l) for l in range(c["levels"])]


def box(dims, s):
    """The rows that have a neighbour in slot s, and those neighbours, as slices of (z, y, x)."""
    rows, nbs = [], []
    for d, m in zip(OFFSETS[s], (dims[2], dims[1], dims[0])):
        lo, hi = max(0, -d), max(max(0, -d), m - max(0, d))
        rows.append(slice(lo, hi))
        nbs.append(slice(lo + d, hi + d))
    return tuple(rows), tuple(nbs)


def varcoef_values(c, seed, device):
    """(n, 27) values of a symmetric matrix: -exp(sigma z) per edge, diagonal sum|a_ij| + 2."""
    dims = (c["nx"], c["ny"], c["nz"])
    shape = dims[::-1]
    v = torch.zeros(shape + (27,), dtype=torch.float64, device=device)
    gen = generator(seed, 1, device)
    for s in range(14, 27):
        rows, nbs = box(dims, s)
        w = -torch.exp(c["sigma"] * torch.randn(shape, dtype=torch.float64, device=device, generator=gen))
        v[rows + (s,)] = w[rows]
        v[nbs + (26 - s,)] = w[rows]
    v[..., DIAG] = v.abs().sum(-1) + 2.0
    return v.view(-1, 27)


def renumbered_levels(c, seed):
    """Host arrays (nnz, cols, vals, f2c) of every level, rows in a random order: row order[i] of the
    grid becomes row i."""
    rng = np.random.default_rng(int(seed))
    dims = level_dims(c)
    new = [rng.permutation(a * b * d) for a, b, d in dims]    # grid row -> row
    out = []
    for l, (nx, ny, nz) in enumerate(dims):
        n = nx * ny * nz
        iz, iy, ix = np.unravel_index(np.arange(n), (nz, ny, nx))
        cols = np.zeros((n, 27), np.int64)
        there = np.zeros((n, 27), bool)
        for s, (dz, dy, dx) in enumerate(OFFSETS):
            there[:, s] = ((iz + dz >= 0) & (iz + dz < nz) & (iy + dy >= 0) & (iy + dy < ny) &
                           (ix + dx >= 0) & (ix + dx < nx))
            cols[:, s] = np.arange(n) + (dz * ny + dy) * nx + dx
        vals = np.where(np.arange(27) == DIAG, 26.0, -1.0)[None, :].repeat(n, 0)
        first = np.argsort(~there, axis=1, kind="stable")      # present entries first, in slot order
        cols = np.take_along_axis(np.where(there, cols, np.arange(n)[:, None]), first, 1)
        vals = np.take_along_axis(np.where(there, vals, 0.0), first, 1)
        old = np.argsort(new[l])                               # row -> grid row
        f2c = None
        if l + 1 < len(dims):
            nxc, nyc, nzc = dims[l + 1]
            jz, jy, jx = np.unravel_index(np.argsort(new[l + 1]), (nzc, nyc, nxc))
            f2c = new[l][(2 * jz * ny + 2 * jy) * nx + 2 * jx].astype(np.int32)
        out.append((there.sum(1)[old].astype(np.uint8), new[l][cols[old]].astype(np.int32), vals[old], f2c))
    return out


def prepare(c, seed):
    dims, dev = (c["nx"], c["ny"], c["nz"]), torch.device("cuda", 0)
    n = dims[0] * dims[1] * dims[2]
    s = {"case": c}
    if c["matrix"] == "renumbered":
        P = Problem.general(levels=c["levels"])
        for l, (nnz, cols, vals, f2c) in enumerate(renumbered_levels(c, seed)):
            P.load_level_general(l, nnz, cols, vals, f2c)
    else:
        P = Problem(*dims, levels=c["levels"])
        P.generate("hpcg")
        if c["matrix"] == "varcoef":
            vals = varcoef_values(c, seed, dev)
            P.set_values(vals.reshape(-1), level=0, recoarsen=True)
            if c["op"] == "gradient":
                s["vals"] = vals
        if c["mixed"]:
            P.build_mixed()
    s["P"] = P
    u = uniform(seed, 2, n, dev)
    if c["op"] == "cg":
        s["b"] = P.spmv(u)
    elif c["op"] == "gradient":
        s["b"] = uniform(seed, 3, n, dev, 0.0, 1.0)
        s["g"] = torch.randn(n, dtype=torch.float64, device=dev, generator=generator(seed, 4, dev))
    elif c["op"] == "mg":
        s["r"] = u
    else:
        s["x"], s["r"] = u, uniform(seed, 5, n, dev)
        s["z"] = torch.empty_like(u)
    return s


def run(s):
    c, P = s["case"], s["P"]
    if c["op"] == "cg":
        x = torch.zeros_like(s["b"])
        if c["mixed"]:
            k, nr, nr0 = P.cg_mixed(s["b"], x, c["max_iter"], c["tol"])
        else:
            k, nr, nr0 = P.cg(s["b"], x, c["max_iter"], c["tol"])
        return {"x": x, "iterations": k, "normr": nr, "normr0": nr0}
    if c["op"] == "mg":
        return P.mg_mixed(s["r"]) if c["mixed"] else P.mg(s["r"])
    if c["op"] == "gradient":
        vals, b = s["vals"].detach().requires_grad_(True), s["b"].detach().requires_grad_(True)
        x = solve(vals, b, P, tol=c["tol"], max_iter=c["max_iter"], mixed=c["mixed"])
        gv, gb = torch.autograd.grad(x, (vals, b), s["g"])
        return {"x": x.detach(), "grad_vals": gv, "grad_b": gb}
    z = s["z"].copy_(s["x"])
    y = P.spmv(s["x"])
    P.symgs(s["r"], z)
    d = P.dot(s["x"], y)
    w = P.waxpby(0.75, y, -1.25, z)
    return {"y": y, "z": z, "dot": d, "w": w}


# ------------------------------------------------------------------ work

def iterations(c):
    """About how many iterations a solve takes (to 1e-10: 16 at 16^3, 169 at 256^3, 302 at 512^3; some
    twenty on any grid where the variable coefficients' diagonal dominates)."""
    if c["tol"] == 0.0:
        return c["max_iter"]
    side = (c["nx"] * c["ny"] * c["nz"]) ** (1.0 / 3.0)
    digits = -math.log10(c["tol"]) / 10.0
    k = 20 * digits if c["matrix"] == "varcoef" else 16 * digits * (max(side, 4.0) / 16.0) ** 0.85
    return max(1, min(c["max_iter"], round(k)))


def work(c):
    """Bytes: a matrix pass reads 8 B (BF16: 2 B; a general pattern: 12 B) per nonzero, the second half
    of a symmetric sweep is a pass of its own and the sweep from zero skips half of its first one; each
    vector of a step is read and written once.  Whatever the caches hold between steps is counted."""
    levels = [(a * b * d, (3 * a - 2) * (3 * b - 2) * (3 * d - 2)) for a, b, d in level_dims(c)]
    n, nnz = levels[0]
    per = 12.0 if c["matrix"] == "renumbered" else 8.0
    vb, xb = (2.0, 4.0) if c["mixed"] else (per, 8.0)

    def vcycle():
        by = fl = 0.0
        for l, (m, z) in enumerate(levels):
            by += 1.5 * z * vb + 2 * m * xb
            fl += 3.0 * z
            if l + 1 < len(levels):
                by += 2.0 * z * vb + 3 * m * xb
                fl += 4.0 * z + 2.0 * z / 8
        return by, fl

    def solver():
        by, fl = vcycle()
        return iterations(c) * (by + per * nnz + 16.0 * n + (8 + xb + xb + 16 + 16 + 24) * n), iterations(c) * (fl + 2.0 * nnz + 12.0 * n)

    if c["op"] == "cg":
        by, fl = solver()
    elif c["op"] == "mg":
        by, fl = vcycle()
    elif c["op"] == "gradient":
        by, fl = solver()
        by, fl = 2 * by + 3 * 216.0 * n, 2 * fl + 27.0 * n
    else:
        by, fl = 8.0 * nnz + 16.0 * n + 16.0 * nnz + 24.0 * n + 16.0 * n + 24.0 * n, 6.0 * nnz + 5.0 * n
    return {"bytes": by, "flops": fl}


def tolerance(c):
    """About four times what the paths were seen off exact() (64 bits, sums in another order) over the
    listed cases and some twenty draws."""
    if c["op"] == "cg":
        # seen: x 1e-15, the last residual norm 3e-13; mixed: x 1e-10 where capped, the norm 4e-6 (it
        # lies ten digits below the first one, and the FP32 V-cycle's rounding shows in it)
        return {"rel": 2e-5} if c["mixed"] else {"rel": 2e-12}
    if c["op"] == "gradient":
        # seen: 3e-16; mixed: 4e-11, the solves' own tolerance
        return {"rel": 5e-10} if c["mixed"] else {"rel": 1e-14}
    # seen: 2e-16 and 5e-16; the mixed V-cycle 1e-7
    return {"rel": 5e-7} if c["mixed"] else {"rel": 2e-15}


# ------------------------------------------------------------------ 64-bit reference (plain torch)

class Grid:
    """One level's operator in FP64: values per slot on the (z, y, x) grid."""

    def __init__(self, dims, vals, coarse=None):
        self.dims, self.vals, self.coarse = dims, vals, coarse
        nx, ny, nz = dims
        self.shape = (nz, ny, nx)
        self.colours = [tuple(slice(p, None, 2) for p in (q >> 2, (q >> 1) & 1, q & 1)) for q in range(8)]

    def padded(self, x):
        return torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))

    def window(self, xp, s, colour=(slice(None),) * 3):
        """x's neighbours in slot s of the rows of a colour."""
        cut = []
        for d, m, c in zip(OFFSETS[s], self.shape, colour):
            cut.append(slice((c.start or 0) + 1 + d, m + 1 + d, c.step))
        return xp[tuple(cut)]

    def spmv(self, x):
        xp, y = self.padded(x), torch.zeros_like(x)
        for s in range(27):
            y += self.vals[s] * self.window(xp, s)
        return y

    def symgs(self, r, x):
        xp = self.padded(x)
        for q in list(range(8)) + list(range(7, -1, -1)):
            at = self.colours[q]
            t = r[at].clone()
            if not t.numel():
                continue
            for s in range(27):
                if s != DIAG:
                    t -= self.vals[s][at] * self.window(xp, s, at)
            self.window(xp, DIAG, at).copy_(t / self.vals[DIAG][at])
        return xp[1:-1, 1:-1, 1:-1].contiguous()

    def mg(self, r):
        x = self.symgs(r, torch.zeros_like(r))
        if self.coarse is not None:
            rc = (r - self.spmv(x))[::2, ::2, ::2].contiguous()
            x[::2, ::2, ::2] += self.coarse.mg(rc)
            x = self.symgs(r, x)
        return x


class Rows:
    """One level's operator in FP64 on rows in any order: the greedy colouring in row order, and one
    sparse matrix for each colour."""

    def __init__(self, nnz, cols, vals, f2c, device, coarse=None):
        n = len(nnz)
        colour, lists, counts = [0] * n, cols.tolist(), nnz.tolist()
        for i in range(n):
            used = {colour[j] for j in lists[i][:counts[i]] if j < i}
            k = 0
            while k in used:
                k += 1
            colour[i] = k
        mask = np.arange(cols.shape[1])[None, :] < nnz[:, None].astype(np.int64)
        colour = np.asarray(colour)

        def csr(rows):
            m = mask[rows]
            start = np.concatenate([[0], np.cumsum(m.sum(1))])
            return torch.sparse_csr_tensor(torch.from_numpy(start), torch.from_numpy(cols[rows][m].astype(np.int64)),
                                           torch.from_numpy(vals[rows][m]), size=(len(rows), n)).to(device)

        torch.sparse.check_sparse_tensor_invariants.disable()
        self.all, self.coarse = csr(np.arange(n)), coarse
        diag = np.where((cols == np.arange(n)[:, None]) & mask, vals, 0.0).sum(1)
        self.parts = []
        for k in range(colour.max() + 1):
            rows = np.flatnonzero(colour == k)
            self.parts.append((torch.from_numpy(rows).to(device), csr(rows), torch.from_numpy(diag[rows]).to(device)))
        self.f2c = None if f2c is None else torch.from_numpy(f2c.astype(np.int64)).to(device)

    def spmv(self, x):
        return self.all @ x

    def symgs(self, r, x):
        x = x.clone()
        for rows, A, d in self.parts + self.parts[::-1]:
            x[rows] += (r[rows] - A @ x) / d
        return x

    def mg(self, r):
        x = self.symgs(r, torch.zeros_like(r))
        if self.coarse is not None:
            rc = (r - self.spmv(x))[self.f2c]
            x[self.f2c] += self.coarse.mg(rc)
            x = self.symgs(r, x)
        return x


def hierarchy(c, seed, device):
    """The levels' operators, finest first."""
    if c["matrix"] == "renumbered":
        top = None
        for nnz, cols, vals, f2c in reversed(renumbered_levels(c, seed)):
            top = Rows(nnz, cols, vals, f2c, device, top)
        return top
    dims, per_level = level_dims(c), []
    for l, d in enumerate(dims):
        shape = d[::-1]
        if c["matrix"] == "hpcg":
            v = torch.zeros((27,) + shape, dtype=torch.float64, device=device)
            for s in range(27):
                v[(s,) + box(d, s)[0]] = 26.0 if s == DIAG else -1.0
        elif l == 0:
            v = varcoef_values(c, seed, device).view(shape + (27,)).permute(3, 0, 1, 2).contiguous()
        else:
            # an edge takes the finer level's value of the edge that leaves its lower point in its direction
            f, v = per_level[-1], torch.zeros((27,) + shape, dtype=torch.float64, device=device)
            for s in range(14, 27):
                rows, nbs = box(d, s)
                w = f[s][::2, ::2, ::2]
                v[(s,) + rows] = w[rows]
                v[(26 - s,) + nbs] = w[rows]
            v[DIAG] = v.abs().sum(0) + 2.0
        per_level.append(v)
    top = None
    for d, v in zip(reversed(dims), reversed(per_level)):
        top = Grid(d, v, top)
    return top


def conjugate_gradients(A, b, max_iter, tol, flexible):
    x, r, p, Ap = torch.zeros_like(b), b.clone(), None, None
    dot = lambda u, v: float((u * v).sum())  # noqa: E731
    normr0 = normr = math.sqrt(dot(r, r))
    k = 0
    rtz = pAp = 0.0
    while k < max_iter and normr / normr0 > tol:
        k += 1
        z = A.mg(r)
        old, rtz = rtz, dot(r, z)
        if k == 1:
            p = z.clone()
        else:
            beta = -dot(z, Ap) / pAp if flexible else rtz / old
            p = z + beta * p
        Ap = A.spmv(p)
        pAp = dot(p, Ap)
        alpha = rtz / pAp
        x += alpha * p
        r -= alpha * Ap
        normr = math.sqrt(dot(r, r))
    return x, k, normr, normr0


def exact(c, seed):
    device = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    n = c["nx"] * c["ny"] * c["nz"]
    solves = {"cg": iterations(c), "gradient": 2 * iterations(c)}.get(c["op"], 1)
    if n * solves > 1.2e9 or n > 60e6 or (c["matrix"] == "renumbered" and n > 120e3):
        return None     # over about 20 seconds
    A = hierarchy(c, seed, device)
    shape = (n,) if c["matrix"] == "renumbered" else A.shape
    flat = lambda v: v.reshape(-1)  # noqa: E731
    u = uniform(seed, 2, n, device).view(shape)
    if c["op"] == "cg":
        b = A.spmv(u)
        x, k, nr, nr0 = conjugate_gradients(A, b, c["max_iter"], c["tol"], c["mixed"])
        # the count is a whole number and the last residual that of a stopping rule: no 64-bit value
        return {"x": flat(x), "iterations": None, "normr": None, "normr0": nr0}
    if c["op"] == "mg":
        return flat(A.mg(u))
    if c["op"] == "gradient":
        b = uniform(seed, 3, n, device, 0.0, 1.0).view(shape)
        g = torch.randn(n, dtype=torch.float64, device=device, generator=generator(seed, 4, device)).view(shape)
        x = conjugate_gradients(A, b, c["max_iter"], c["tol"], c["mixed"])[0]
        lam = conjugate_gradients(A, g, c["max_iter"], c["tol"], c["mixed"])[0]
        xp, gv = A.padded(x), torch.empty(shape + (27,), dtype=torch.float64, device=device)
        for s in range(27):
            gv[..., s] = -lam * A.window(xp, s)
        return {"x": flat(x), "grad_vals": gv.view(n, 27), "grad_b": flat(lam)}
    r = uniform(seed, 5, n, device).view(shape)
    y, z = A.spmv(u), A.symgs(r, u)
    return {"y": flat(y), "z": flat(z), "dot": float((u * y).sum()), "w": flat(0.75 * y - 1.25 * z)}
