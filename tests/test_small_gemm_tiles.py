"""FP64 Schur updates of batches of at most two rounds of 32 x 32 tiles run in
those: fronts whose update matrices end inside a tile, on one tile and
on several, and batches on both sides of that size, against the dense
solution."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("copies,above", [(4, False), (500, True)])
def test_fp64_updates_on_both_sides_of_the_rule(gpu, copies, above):
    mats = [generators.laplace2d_perturbed(31, 33, seed=k % 3)
            for k in range(copies)]
    n = len(mats[0][0]) - 1
    b = np.random.default_rng(5).uniform(-1, 1, n * copies)
    with snu.Solver(nleaves=8) as s:
        s.construct_batch(mats)
        fp = s.front_plan()
        tiles = np.zeros(fp["nlevels"], int)  # 32 x 32 tiles of each level
        np.add.at(tiles, fp["level"], ((fp["q"] + 31) // 32) ** 2)
        # (1480: two rounds of five blocks on each of 148 SMs)
        assert tiles.max() > 1480 if above else tiles.max() <= 1480
        x = s.factorize().solve(b)
    for k in range(3):
        rp, ci, v = mats[k]
        A = np.zeros((n, n))
        A[np.repeat(np.arange(n), np.diff(rp)), ci] = v
        B = b.reshape(copies, n)[k::3].T
        ref = np.linalg.solve(A, B)
        tol = np.linalg.cond(A) * 200 * 2.0 ** -53  # (as above)
        assert np.abs(x.reshape(copies, n)[k::3].T - ref).max() <= tol * np.abs(ref).max()
