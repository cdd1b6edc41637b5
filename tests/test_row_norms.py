"""Row norms of new values where rows are long: the backward error that a
solve reports against the same formula on the host, for rows on both sides of
the length that a block takes over, and the time of a refactor."""
import time

import numpy as np
import pytest
import scipy.sparse as sp

import snusolver_b200 as snu
from snusolver_b200 import generators


def _csr(A):
    A = sp.csr_matrix(A)
    A.sort_indices()
    return A.indptr, A.indices, A.data.copy()


def _border(nx, ny, row, col):
    """A grid with one more unknown whose row and column hold `row` and `col`
    entries (the first ones)."""
    rp, ci, v = generators.laplace2d_lognormal(nx, ny, seed=nx)
    n = nx * ny
    G = sp.csr_matrix((v, ci, rp), shape=(n, n)) + sp.diags(np.full(n, 2e-3))
    r, c = np.zeros(n), np.zeros(n)
    r[:row], c[:col] = -0.5, -1e-3
    return _csr(sp.bmat([[G, sp.csr_matrix(c[:, None])],
                         [sp.csr_matrix(r[None, :]), [[0.6 * n + 10.0]]]]))


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [(63, 64), (255, 256), (257, 1000), (0, 899)])
def test_backward_error_counts_long_rows(gpu, rows):
    # one matrix, and a batch with one: stopping after the FP32 solve leaves
    # a residual far above the rounding of the sums compared here
    mats = [_border(30, 30, min(r, 900), 5) for r in rows]
    mats.append(generators.laplace2d_perturbed(11, 9, seed=1))
    rng = np.random.default_rng(0)

    def want(ms, x, b):
        be, at = 0.0, 0
        for rp, ci, v in ms:
            n = len(rp) - 1
            A = sp.csr_matrix((v, ci, rp), shape=(n, n))
            xs, bs = x[at:at + n], b[at:at + n]
            den = abs(A).sum(1).max() * abs(xs).max() + abs(bs).max()
            be, at = max(be, abs(bs - A @ xs).max() / den), at + n
        return be

    for ms in ([mats[0]], [mats[1]], mats):
        with snu.Solver(nleaves=2, precision=snu.FP32_IR, ir_tol=1e-3) as s:
            if len(ms) == 1:
                s.construct(*ms[0])
            else:
                s.construct_batch(ms)
            b = rng.uniform(-1, 1, s.n)
            x = s.factorize().solve(b)
            # (sums of 1e3 terms in 64 bits against a residual near 1e-7)
            assert s.stats()["backward_error"] == pytest.approx(
                want(ms, x, b), rel=1e-5)


@pytest.mark.gpu
def test_refactor_time_of_a_long_row(gpu):
    # a dense row against a dense column: the same fronts and as many values,
    # so the times differ by the norm of the row (250 000 entries; 8.2 ms
    # when one thread sums it)
    t = []
    for row, col in ((0, 250000), (250000, 0)):
        m = _border(500, 500, row, col)
        with snu.Solver(nleaves=8, precision=snu.FP32_IR) as s:
            s.construct(*m).factorize()
            ts = []
            for _ in range(7):
                t0 = time.perf_counter()
                s.refactor(m[2])
                ts.append(time.perf_counter() - t0)
            t.append(min(ts))
    assert t[1] < t[0] + 2e-3, t
