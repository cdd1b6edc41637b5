"""FP64 Schur updates of batches too small to fill the device run in 32 x 32
tiles: fronts whose update matrices end inside a tile, on one tile and on
several, against the dense solution."""
import numpy as np
import pytest

import snusolver_b200 as snu
from snusolver_b200 import generators


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(5, 5), (17, 3), (31, 33), (40, 23), (64, 9)])
@pytest.mark.parametrize("nleaves", [2, 8])
def test_small_fp64_updates(gpu, shape, nleaves):
    rp, ci, v = generators.laplace2d_perturbed(*shape, seed=sum(shape))
    n = len(rp) - 1
    A = np.zeros((n, n))
    A[np.repeat(np.arange(n), np.diff(rp)), ci] = v
    b = np.random.default_rng(4).uniform(-1, 1, (n, 2))
    with snu.Solver(nleaves=nleaves) as s:
        x = s.construct(rp, ci, v).factorize().solve(b)
    ref = np.linalg.solve(A, b)
    # forward error of a backward stable solve: cond(A) times a small
    # multiple of the rounding of the longest sums (front sizes below 200)
    tol = np.linalg.cond(A) * 200 * 2.0 ** -53
    assert np.abs(x - ref).max() <= tol * np.abs(ref).max()
