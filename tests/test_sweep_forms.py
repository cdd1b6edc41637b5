"""The solve's vectors in elimination order against the per-front work vectors
(the bit-reproducible mode): every register-group width, ragged groups and
passes, pivot blocks of one and of several chunks."""
import numpy as np
import pytest

import snusolver_b200 as snu
from snusolver_b200 import generators


def _solver(monkeypatch, mat, precision, **env):
    for k in ("SNU_DETERMINISTIC", "SNU_SOLVE_FUSED"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    return snu.Solver(nleaves=4, precision=precision).construct(*mat).factorize()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [snu.FP64, snu.FP32_IR])
@pytest.mark.parametrize("grid", [(37, 29), (13, 14, 15)])
def test_forms_agree(gpu, monkeypatch, precision, grid):
    mat = (generators.laplace2d_perturbed(*grid, seed=2) if len(grid) == 2
           else generators.laplace3d_lognormal(*grid, seed=2))
    n = len(mat[0]) - 1
    rng = np.random.default_rng(7)
    level = _solver(monkeypatch, mat, precision, SNU_SOLVE_FUSED="0")
    tree = _solver(monkeypatch, mat, precision, SNU_SOLVE_FUSED="1")
    work = _solver(monkeypatch, mat, precision, SNU_DETERMINISTIC="1")
    # FP64: the forms differ in the order of their sums only; mixed: all
    # refine to a backward error of 1e-10, which the condition of these grids
    # (below 1e4) amplifies
    tol = 1e-11 if precision == snu.FP64 else 1e-6
    for nrhs in (1, 2, 3, 5, 8, 13, 16, 17, 33, 64, 65):
        b = np.asfortranarray(rng.uniform(-1, 1, (nrhs, n)).T)
        ref = work.solve(b)
        for s in (level, tree):
            x = s.solve(b)
            assert s.stats()["backward_error"] <= 1e-10
            assert np.abs(x - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("fused", ["0", "1"])
def test_nan_right_hand_side_with_every_bit_set(gpu, monkeypatch, fused):
    # the pattern that marks an unsolved element is no result: a NaN column
    # ends as NaN, its neighbours are untouched and nothing waits
    mat = generators.laplace2d_perturbed(20, 17, seed=2)
    n = len(mat[0]) - 1
    b = np.asfortranarray(np.random.default_rng(3).uniform(-1, 1, (2, n)).T)
    s = _solver(monkeypatch, mat, snu.FP64, SNU_SOLVE_FUSED=fused)
    ref = s.solve(b)
    c = b.copy(order="F")
    c[:, 1].view(np.uint64)[:] = np.uint64(0xFFFFFFFFFFFFFFFF)
    x = s.solve(c)
    assert np.isnan(x[:, 1]).all()
    assert np.abs(x[:, 0] - ref[:, 0]).max() <= 1e-12 * np.abs(ref[:, 0]).max()
