"""The damped step's exact digit products, Cholesky panels and LU fallback at
the sizes where they can go wrong: parameters around the tensor-core tiles (64
columns, 128 rows) and the panels (64), rows around the 32-row stages and
their read-back windows, columns of very different magnitude, systems that
are not positive definite.

TOLERANCES as in test_lm_gpu.py: J^T J 1e-13 of sqrt(JJ_ii JJ_jj) (the FP64
sum's own error at these row counts), trial models 1e-9 of the step."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

DM = np.array([[1e-3, 1e-3], [0.1, 1e-2], [1.0, 1.0]])


def problem(nrows, ncols, seed, spread=1.0):
    rng = np.random.default_rng(seed)
    J = rng.normal(size=(nrows, ncols)) * 10.0 ** rng.uniform(-spread, spread, ncols)[None, :]
    return (J, rng.normal(size=nrows), rng.normal(size=ncols),
            10.0 ** rng.uniform(-spread, spread, ncols), DM)


def check(ctx, J, r, b, sig, dm):
    B, JJ = ctx.lm_steps(J, r, b, sig, dm, return_jtj=True)
    Bref, JJref = oracle.lm_steps(J, r, b, sig, dm)
    s = np.sqrt(np.diag(JJref))
    assert np.max(np.abs(JJ - JJref) / np.outer(s, s)) <= 1e-13
    assert np.array_equal(JJ, JJ.T)
    for d in range(len(dm)):
        step = Bref[d] - b
        assert np.max(np.abs((B[d] - b) - step)) <= 1e-9 * np.max(np.abs(step)), d


@pytest.mark.parametrize("nrows,ncols", [(1, 1), (40, 2), (31, 63), (260, 64), (33, 65), (700, 127),
                                         (129, 128), (4100, 129), (257, 192), (900, 257)])
def test_tile_and_panel_edges(ctx, nrows, ncols):
    check(ctx, *problem(nrows, ncols, seed=nrows + ncols))


def test_columns_of_very_different_magnitude(ctx):
    """Six decades between the columns (and their uncertainties)."""
    check(ctx, *problem(500, 150, seed=3, spread=3.0))
    J, r, b, sig, dm = problem(300, 70, seed=4)
    JJ = ctx.lm_steps(np.ldexp(J, 400), r, b, sig, dm, return_jtj=True)[1]
    assert np.array_equal(JJ, np.ldexp(ctx.lm_steps(J, r, b, sig, dm, return_jtj=True)[1], 800))


@pytest.mark.parametrize("ncols", [50, 150])
def test_systems_that_are_not_positive_definite(ctx, ncols):
    """Negative damping makes the second system indefinite (pivoted LU); the
    first and third stay on Cholesky."""
    J, r, b, sig, _ = problem(400, ncols, seed=5)
    sig = np.ones(ncols)
    mid = np.median(np.diag(J.T @ J))
    check(ctx, J, r, b, sig, np.array([[0.1, 0.1], [0.0, -0.7 * mid], [1.0, 0.1]]))


def test_not_finite_jacobian_entries(ctx):
    J, r, b, sig, dm = problem(200, 90, seed=6)
    J[7, 11] = np.nan
    J[9, 40] = np.inf
    JJ = ctx.lm_steps(J, r, b, sig, dm, return_jtj=True)[1]
    odd = np.zeros(90, bool)
    odd[[11, 40]] = True
    assert not np.any(np.isfinite(JJ[odd])) and not np.any(np.isfinite(JJ[:, odd]))
    ok = JJ[np.ix_(~odd, ~odd)]
    ref = J[:, ~odd].T @ J[:, ~odd]
    assert np.max(np.abs(ok - ref)) <= 1e-13 * np.max(np.abs(ref))
