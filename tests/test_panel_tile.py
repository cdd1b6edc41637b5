"""The diagonal-tile factorization at the edges of its tiles and steps: dense
fronts whose pivots end inside a step of four, a tile of 64 or an outer block
of 256, and FP32 pivots near the ends of the exponent range, whose reciprocals
take the scaled path."""
import numpy as np
import pytest

import snusolver_b200 as snu


def _dense(n, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1, 1, (n, n)) + 2.0 * n * np.eye(n)
    A *= scale
    rp = np.arange(0, n * n + 1, n)
    ci = np.tile(np.arange(n), n)
    return A, rp, ci, A.ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 5, 9, 63, 64, 65, 67, 130, 191, 256, 259])
@pytest.mark.parametrize("precision", [snu.FP64, snu.FP32_IR])
def test_dense_fronts(gpu, n, precision):
    A, rp, ci, v = _dense(n, n)
    b = np.random.default_rng(1).uniform(-1, 1, (n, 3))
    with snu.Solver(nleaves=2, precision=precision) as s:
        x = s.construct(rp, ci, v).factorize().solve(b)
        be = s.stats()["backward_error"]
    ref = np.linalg.solve(A, b)
    # rows dominate by at least 2n - n: the condition number is below 3, so
    # the forward error is at most a few times n eps (FP64) or the backward
    # error that refinement stops at (mixed)
    tol = 8 * n * 2.0 ** -53 if precision == snu.FP64 else 4 * 1e-10
    assert be <= (8 * n * 2.0 ** -53 if precision == snu.FP64 else 1e-10)
    assert np.abs(x - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [7, 40, 64])
@pytest.mark.parametrize("exponent", [-128, -126, 113, 118])
def test_fp32_pivots_near_the_exponent_range(gpu, n, exponent):
    # diagonal near 2n 2^exponent: below 2^-118 or above 2^117 (the static
    # pivot off, which would replace the small ones)
    A, rp, ci, v = _dense(n, 3, 2.0 ** exponent)
    # (right-hand sides and solutions stay normal FP32 numbers)
    b = np.random.default_rng(2).uniform(-1, 1, n) * 2.0 ** max(exponent, 0)
    with snu.Solver(nleaves=2, precision=snu.FP32_IR, pivot_eps=0.0) as s:
        x = s.construct(rp, ci, v).factorize().solve(b)
        assert s.stats()["fp64_fallback"] == 0
    ref = np.linalg.solve(A, b)
    assert np.abs(x - ref).max() <= 4 * 1e-10 * np.abs(ref).max()
