"""Performance cases of the numeric factorize-and-solve path.

Each case is work that a program using this package repeats on a handle it
keeps, through the public classes ``Solver`` and ``Server``:

* ``step``: new values on a known pattern, then a solve with new right-hand
  sides, both from host arrays (``Solver.refactor`` + ``Solver.solve``): a
  time step or a Newton iteration;
* ``batch``: the same on a batch of independent matrices in one handle;
* ``solve``: right-hand sides that are on the GPU against factors that stay
  resident (``Solver.solve_device``);
* ``serve``: a burst of refactor and solve requests on several resident
  matrices (``Server``).

Matrices are the generators' grids: the lognormal 2D and 3D Laplacians of the
serving stream and the batched workload, 3D convection-diffusion, the 3D
27-point stencil and the perturbed 2D Laplacian.  The values of a pass are
those of a refactor request of the serving stream: every off-diagonal entry
rescaled, the diagonal following so that the rows keep their dominance.
"""
import functools
import math

import numpy as np
import torch

import snusolver_b200 as snu
from snusolver_b200 import generators
from snusolver_b200.server import Server, rescale_values

_PREC = {"fp64": snu.FP64, "mixed": snu.FP32_IR}


def listed():
    return [
        # the smallest call: a 24 x 24 grid factored and solved in FP64;
        # launches and host work are all of it
        dict(name="step_2d_24_fp64", op="step", grid="2d_perturbed", nx=24,
             ny=24, nz=1, leaves=4, precision="fp64", nrhs=1, pinned=False),
        # a plain FP64 step of a 128 x 128 grid, one right-hand side
        dict(name="step_2d_128_fp64", op="step", grid="2d_perturbed", nx=128,
             ny=128, nz=1, leaves=8, precision="fp64", nrhs=1, pinned=False),
        # a ragged 2D grid in mixed precision, more leaves
        dict(name="step_2d_301x187_mixed", op="step", grid="2d", nx=301,
             ny=187, nz=1, leaves=16, precision="mixed", nrhs=3, pinned=False),
        # the benchmark's workload: 64^3 convection-diffusion, 4 right-hand
        # sides, mixed precision, page-locked host arrays (the largest case)
        dict(name="step_3d_64_mixed", op="step", grid="3d_convdiff", nx=64,
             ny=64, nz=64, leaves=8, precision="mixed", nrhs=4, pinned=True),
        # plain FP64 in 3D at an odd size
        dict(name="step_3d_41_fp64", op="step", grid="3d_convdiff", nx=41,
             ny=41, nz=41, leaves=8, precision="fp64", nrhs=3, pinned=True),
        # the 27-point stencil with 16 right-hand sides
        dict(name="step_27pt_33_mixed", op="step", grid="3d_27pt", nx=33,
             ny=33, nz=33, leaves=8, precision="mixed", nrhs=16, pinned=True),
        # a batch of independent 2D grids of 32..256 points a side
        dict(name="batch_40_mixed", op="batch", grid="2d", nx=32, ny=256,
             nz=40, leaves=8, precision="mixed", nrhs=1, pinned=False),
        # one right-hand side on resident factors of a 2D grid
        dict(name="solve_2d_400_mixed_1", op="solve", grid="2d", nx=400,
             ny=400, nz=1, leaves=8, precision="mixed", nrhs=1, pinned=False),
        # many right-hand sides on resident factors of a 3D grid
        dict(name="solve_3d_54_mixed_64", op="solve", grid="3d", nx=54, ny=54,
             nz=54, leaves=8, precision="mixed", nrhs=64, pinned=False),
        # FP64 factors, a ragged count of columns
        dict(name="solve_3d_37_fp64_13", op="solve", grid="3d", nx=37, ny=37,
             nz=37, leaves=8, precision="fp64", nrhs=13, pinned=False),
        # a server's burst: two refactors and twelve solves of 1..64 columns
        # on three resident matrices
        dict(name="serve_3_mixed", op="serve", grid="2d", nx=100, ny=224,
             nz=22, leaves=8, precision="mixed", nrhs=64, pinned=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any operation, grids from 16 to 400 points a side in 2D
    and 8 to 56 in 3D, both precisions, 1 to 64 right-hand sides."""
    op = rng.choice(["step", "step", "step", "solve", "solve", "solve",
                     "batch", "serve"])
    c = dict(op=op, leaves=8, precision=rng.choice(["fp64", "mixed"]),
             nrhs=_log(rng, 1, 64), pinned=rng.random() < 0.5, nz=1)
    if op == "batch":
        lo = rng.randint(16, 64)
        c.update(grid="2d", nx=lo, ny=rng.randint(lo + 16, 256),
                 nz=_log(rng, 4, 40), nrhs=_log(rng, 1, 8), pinned=False,
                 precision="mixed")
    elif op == "serve":
        c.update(grid="2d", nx=rng.randint(50, 160), ny=rng.randint(100, 240),
                 nz=rng.randint(10, 26), nrhs=_log(rng, 4, 64), pinned=False,
                 precision="mixed")
    else:
        c["grid"] = rng.choice(["2d", "2d", "2d_perturbed", "3d",
                                "3d_convdiff", "3d_27pt"])
        if c["grid"] in ("2d", "2d_perturbed"):
            c.update(nx=_log(rng, 16, 400), ny=_log(rng, 16, 400))
        elif c["grid"] == "3d":
            m = _log(rng, 8, 56)
            c.update(nx=m, ny=max(8, m - rng.randint(0, 7)),
                     nz=max(8, m - rng.randint(0, 7)))
        else:
            m = _log(rng, 8, 52 if c["grid"] == "3d_convdiff" else 34)
            c.update(nx=m, ny=m, nz=m)
        c["leaves"] = (4 if c["nx"] * c["ny"] * c["nz"] < 2000
                       else rng.choice([4, 8, 16]))
    return c


@functools.lru_cache(maxsize=24)
def _grid(kind, nx, ny, nz):
    """Pattern and first values of a grid: (rowptr, colidx, vals)."""
    if kind == "2d":
        return generators.laplace2d_lognormal(nx, ny, seed=1000 + nx)
    if kind == "2d_perturbed":
        return generators.laplace2d_perturbed(nx, ny, seed=0)
    if kind == "3d":
        return generators.laplace3d_lognormal(nx, ny, nz, seed=1000 + nx)
    if kind == "3d_convdiff":
        return generators.convdiff3d(nx)
    if kind == "3d_27pt":
        return generators.stencil27_lognormal(nx, seed=4)[:3]
    raise KeyError(kind)


def _grids(case):
    """Every matrix of the case as (kind, nx, ny, nz)."""
    if case["op"] == "batch":  # nz grids, sides drawn from nx..ny
        rng = np.random.default_rng(3)
        sides = rng.integers(case["nx"], case["ny"] + 1, size=(case["nz"], 2))
        return [("2d", int(a), int(b), 1) for a, b in sides]
    if case["op"] == "serve":  # two 2D grids and a 3D grid
        return [("2d", case["nx"], case["nx"], 1),
                ("2d", case["ny"], case["ny"], 1),
                ("3d", case["nz"], case["nz"], case["nz"])]
    return [(case["grid"], case["nx"], case["ny"], case["nz"])]


def _inputs(case, seed):
    """(matrices, refactor values per matrix, right-hand sides): the same
    from prepare() and exact()."""
    mats = [_grid(*g) for g in _grids(case)]
    rng = np.random.default_rng([seed, 17])
    n = [len(m[0]) - 1 for m in mats]
    if case["op"] == "serve":
        # the 2D grids are refactored; every matrix takes solves of 1..nrhs
        # columns, the first more of them after its refactor
        vals = [rescale_values(*mats[0], rng), rescale_values(*mats[1], rng),
                None]
        most = case["nrhs"]
        cols = [1, 1, max(1, most // 4), most, 1, max(1, most // 2),
                max(1, most // 8), most, 1, 2, max(1, most // 3), most]
        on = [0, 1, 2, 0, 0, 2, 1, 1, 2, 0, 2, 0]
        rhs = [(m, np.asfortranarray(rng.uniform(-1, 1, (k, n[m])).T))
               for m, k in zip(on, cols)]
        return mats, vals, rhs
    vals = [rescale_values(*m, rng) for m in mats]
    rhs = np.asfortranarray(rng.uniform(-1, 1, (case["nrhs"], sum(n))).T)
    return mats, vals, rhs


def _host(a, pinned):
    """A host array (Fortran order kept) in page-locked memory if asked."""
    if not pinned:
        return a
    t = torch.from_numpy(np.ascontiguousarray(a.T)).pin_memory()
    return t.numpy().T


def prepare(case, seed):
    mats, vals, rhs = _inputs(case, seed)
    prec = _PREC[case["precision"]]
    if case["op"] == "serve":
        s = Server(slots=4, nleaves=case["leaves"], precision=prec)
        ids = [s.factor(*m)[0] for m in mats]
        bad = [c for c in s.drain() if c["status"]]
        if bad:
            raise RuntimeError("factor request failed: %r" % bad[0])
        out = [np.empty_like(b, order="F") for _, b in rhs]
        return dict(op="serve", s=s, ids=ids, vals=vals, rhs=rhs, out=out)
    s = snu.Solver(nleaves=case["leaves"], precision=prec)
    if case["op"] == "batch":
        s.construct_batch(mats)
    else:
        s.construct(*mats[0])
    s.factorize()
    v = np.concatenate(vals)
    if case["op"] == "solve":
        s.refactor(v)
        b = torch.from_numpy(np.ascontiguousarray(rhs.T)).cuda()
        return dict(op="solve", s=s, b=b, x=torch.empty_like(b))
    return dict(op="step", s=s, vals=_host(v, case["pinned"]),
                b=_host(rhs, case["pinned"]),
                x=_host(np.zeros_like(rhs, order="F"), case["pinned"]))


def run(state):
    s = state["s"]
    if state["op"] == "step":
        s.refactor(state["vals"])
        return s.solve(state["b"], out=state["x"])
    if state["op"] == "solve":
        b, x = state["b"], state["x"]
        s.solve_device(b.data_ptr(), x.data_ptr(), b.shape[0], b.shape[1],
                       torch.cuda.current_stream().cuda_stream)
        return x
    for m, v in zip(state["ids"], state["vals"]):
        if v is not None:
            s.refactor(m, v)
    for (m, b), x in zip(state["rhs"], state["out"]):
        s.solve(state["ids"][m], b, out=x)
    bad = [c for c in s.drain() if c["status"]]
    if bad:
        raise RuntimeError("request failed: %r" % bad[0])
    return state["out"]


@functools.lru_cache(maxsize=96)
def _plan(grid, leaves):
    """(n, nnz, factor entries, factorization flops) of a grid's front plan,
    without a GPU."""
    rp, ci, _ = _grid(*grid)
    with snu.Solver(nleaves=leaves) as s:
        st = s.analyze(rp, ci).plan().stats()
    return len(rp) - 1, len(ci), st["factor_entries"], st["factor_flops"]


def work(case):
    """The values and right-hand sides read, the factors written by a
    factorization and read once by a solve, the solutions written; the
    factorization's flops and two per factor entry and column.  Refinement
    steps and work vectors are not counted."""
    es = 8 if case["precision"] == "fp64" else 4
    plans = [_plan(g, case["leaves"]) for g in _grids(case)]
    n, nnz, entries, flops = (sum(p[k] for p in plans) for k in range(4))
    if case["op"] == "serve":
        _, _, rhs = _inputs(case, 0)
        by = sum(8 * p[1] + es * p[2] for p in plans[:2])
        fl = sum(p[3] for p in plans[:2])
        for m, b in rhs:
            fl += 2.0 * plans[m][2] * b.shape[1]
            by += 16.0 * b.size + es * plans[m][2]
        return dict(bytes=by, flops=fl)
    r = case["nrhs"]
    by = 16.0 * n * r + es * entries
    fl = 2.0 * entries * r
    if case["op"] != "solve":
        by += 8.0 * nnz + es * entries
        fl += flops
    return dict(bytes=by, flops=fl)


def tolerance(case):
    """FP64: the rounding of an LU without pivoting on diagonally dominant
    systems (up to 6e-15 seen against the exact solutions).  Mixed:
    refinement stops at a backward error of 1e-10, which the condition of the
    grid amplifies in the solution (up to 1.4e-7 seen on lognormal 2D grids,
    2e-9 in 3D)."""
    if case["precision"] == "fp64":
        return dict(rel=1e-13, max=1e-12)
    if case["grid"] == "2d":
        return dict(rel=1e-6, max=1e-5)
    return dict(rel=2e-8, max=2e-7)


# ----------------------------------------------------- the exact solutions

def _bicgstab(A, d, b, tol, most):
    """Jacobi-preconditioned BiCGSTAB (van der Vorst, 1992) on every column
    of b at once; columns that have converged or broken down stay put."""
    x = torch.zeros_like(b)
    r = b.clone()
    rt = r.clone()
    p = torch.zeros_like(b)
    v = torch.zeros_like(b)
    one = torch.ones(b.shape[1], dtype=b.dtype, device=b.device)
    rho, alpha, om = one, one, one
    stop = tol * b.norm(dim=0)

    def over(a, c):
        return torch.where(c != 0, a / torch.where(c != 0, c, one), 0 * a)

    for it in range(most):
        rn = (rt * r).sum(0)
        beta = over(rn, rho) * over(alpha, om)
        p = r + beta * (p - om * v)
        y = p / d
        v = A @ y
        alpha = over(rn, (rt * v).sum(0))
        s = r - alpha * v
        z = s / d
        t = A @ z
        om = over((t * s).sum(0), (t * t).sum(0))
        x += alpha * y + om * z
        r = s - om * t
        rho = rn
        if it % 16 == 15 and bool((r.norm(dim=0) <= stop).all()):
            break
    return x


def _solve64(mat, vals, b):
    """A^-1 b in 64 bits: BiCGSTAB restarted on the true residual until the
    residual is at rounding level; None if it does not get there."""
    rp, ci, _ = mat
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = len(rp) - 1
    rows = np.repeat(np.arange(n), np.diff(rp))
    diag = np.zeros(n)
    diag[rows[rows == ci]] = vals[rows == ci]
    A = torch.sparse_csr_tensor(torch.from_numpy(rp.astype(np.int64)),
                                torch.from_numpy(ci.astype(np.int64)),
                                torch.from_numpy(np.asarray(vals)),
                                size=(n, n)).to(dev)
    d = torch.from_numpy(diag)[:, None].to(dev)
    B = torch.from_numpy(np.ascontiguousarray(b)).to(dev)
    an = float(np.bincount(rows, np.abs(vals), n).max())
    x = torch.zeros_like(B)
    for _ in range(40):
        r = B - A @ x
        be = (r.abs().amax(0) / (an * x.abs().amax(0) + B.abs().amax(0))).max()
        if float(be) < 4e-16:
            break
        x += _bicgstab(A, d, r, 1e-6, 600)
    return x.cpu().numpy() if float(be) < 4e-15 else None


def exact(case, seed):
    mats, vals, rhs = _inputs(case, seed)
    if case["op"] == "serve":
        return [_solve64(mats[m], mats[m][2] if vals[m] is None else vals[m], b)
                for m, b in rhs]
    if case["op"] == "batch":
        out, at = [], 0
        for m, v in zip(mats, vals):
            k = len(m[0]) - 1
            x = _solve64(m, v, rhs[at:at + k])
            if x is None:
                return None
            out.append(x)
            at += k
        return np.concatenate(out)
    x = _solve64(mats[0], vals[0], rhs)
    return x.T if case["op"] == "solve" and x is not None else x
