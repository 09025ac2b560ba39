"""Densities of tensor-core trials as two TF32 parts: formed from the double's
bits in the middle of the range, by conversions outside.  Scaling all densities
by a power of two, which moves them from one to the other, scales the field
exactly, so a difference shows a wrong part (2^-11 of a density or 2^-11 of its
low part).  Densities with ties of both roundings, powers of two and zeros.

TOLERANCE: 1e-12 of the largest value (nothing is rounded differently but sums
in another order)."""
import numpy as np
import pytest

import ztm_gb300

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [-82, -74, -60, 30, 90])
def test_scaled_trials(ctx, shift):
    rng = np.random.default_rng(11)
    mesh = ztm_gb300.make_mesh(20, 17, 9, 1000.0, 1000.0, 500.0)
    rho = rng.normal(0.0, 1.0, (32, 20 * 17 * 9))
    rho[rng.random(rho.shape) < 0.2] = 0.0
    pick = rng.random(rho.shape)
    sign = np.where(rng.random(rho.shape) < 0.5, -1.0, 1.0)
    two = 2.0 ** rng.integers(-2, 3, rho.shape)
    for p, v in enumerate((1.0, 1.0 + 2.0 ** -11, 1.0 + 2.0 ** -24, 1.0 + 3 * 2.0 ** -24,
                           2.0 - 2.0 ** -12, 1.0 + 2.0 ** -10 + 2.0 ** -22, 1.0 - 2.0 ** -53)):
        at = (pick >= 0.05 * p) & (pick < 0.05 * (p + 1))
        rho[at] = (sign * two * v)[at]
    st = np.stack([rng.uniform(0.0, 20e3, 70), rng.uniform(0.0, 17e3, 70),
                   rng.uniform(100.0, 2000.0, 70)], axis=1)
    ref = ctx.batch([(mesh, rho, st)])[0]
    out = ctx.batch([(mesh, rho * 2.0 ** shift, st)])[0] * 2.0 ** -shift
    assert np.max(np.abs(out - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_near_limits_on_cell_centres(ctx):
    """Cells of 2 x 1 x 2 km (half-diagonal 1.5 km) and a near radius of 8
    half-diagonals: centres exactly on the limit, which float cannot decide.
    TOLERANCE: 1e-6, that of the mixed method."""
    mesh = ztm_gb300.make_mesh(24, 40, 20, 2000.0, 1000.0, 2000.0)
    rho = np.random.default_rng(3).normal(0.0, 300.0, 24 * 40 * 20)
    st = np.array([[2000.0 * i + 1000.0, 1000.0 * j + 500.0, z]
                   for i, j in ((0, 0), (11, 20), (23, 39), (5, 33)) for z in (-1000.0, 1000.0, 11000.0)])
    st[:, :2] += np.arange(len(st))[:, None] % 2 * 1e-9
    a = ctx.prism(mesh, rho, st, precision="mixed", near_q=8.0)
    b = ctx.prism(mesh, rho, st, precision="fp64")
    assert np.max(np.abs(a - b)) <= 1e-6 * np.max(np.abs(b))
