"""The double point-mass sums by levels (pm64.cuh) against the oracle, at the
sizes where they can go wrong: rows shorter and longer than a warp, station
counts around a block of 128, one level and many, refined grids, node lists
with repetitions; stations very near nodes and very far above them (the
integer r^-3 over its range and the library's beyond it).

TOLERANCE: 1e-12 normwise, that of the point-mass tests."""
import numpy as np
import pytest

import oracle
import ztm_gb300
from helpers import rel_err

pytestmark = pytest.mark.gpu


def inputs(di, dj, dk, fh, fv, seed, lift=0.37):
    rng = np.random.default_rng(seed)
    n = ((di - 1) * fh + 1) * ((dj - 1) * fh + 1) * ((dk - 1) * fv + 1)
    drho = rng.normal(0.0, 0.1, n)
    drho[rng.random(n) < 0.4] = 0.0
    return drho, (dk - 1) + lift + 0.2 * rng.random(di * dj), rng.normal(0.0, 1.0, di * dj)


DIMS = [(12, 11, 2, 1, 1, 0), (33, 5, 3, 1, 3, 0), (65, 9, 7, 1, 2, 3), (18, 19, 5, 2, 3, 2),
        (16, 8, 1, 1, 1, 0), (43, 3, 2, 1, 1, 0), (20, 20, 290, 1, 2, 5), (3, 2, 600, 1, 1, 0)]


@pytest.mark.parametrize("dims", DIMS)
def test_forward_and_adjoint(ctx, dims):
    g = ztm_gb300.make_grid(*dims)
    drho, surf, w = inputs(*dims[:5], seed=sum(dims))
    assert rel_err(ctx.pointmass(g, drho, surf), oracle.pointmass_tfm(g, drho, surf)) <= 1e-12
    for kw in ({}, {"drho": drho}):
        assert rel_err(ctx.pointmass_adjoint(g, surf, w, **kw),
                       oracle.pointmass_adjoint(g, surf, w, **kw)) <= 1e-12
    nn = np.random.default_rng(1).integers(0, drho.size, drho.size // 2).astype(np.int32)
    nn[: nn.size // 4] = nn[0]
    drho[nn] += 0.3
    assert rel_err(ctx.pointmass(g, drho, surf, nn=nn), oracle.pointmass_tfm(g, drho, surf, nn=nn)) <= 1e-12
    assert rel_err(ctx.pointmass_adjoint(g, surf, w, nn=nn),
                   oracle.pointmass_adjoint(g, surf, w, nn=nn)) <= 1e-12


@pytest.mark.parametrize("lift", [1e-9, 1e-3, 40.0, 1e6, 1e100])
def test_distances(ctx, lift):
    """Stations a billionth of a grid unit above the top nodes up to distances
    beyond the integer form's range."""
    g = ztm_gb300.make_grid(9, 8, 3, 1, 2, 0)
    drho, surf, _ = inputs(9, 8, 3, 1, 2, seed=2)
    surf = np.full(surf.size, 2.0 + lift)
    assert rel_err(ctx.pointmass(g, drho, surf), oracle.pointmass_tfm(g, drho, surf)) <= 1e-12


def test_a_station_on_a_node_is_not_finite(ctx):
    g = ztm_gb300.make_grid(9, 8, 3, 1, 2, 0)
    drho, surf, _ = inputs(9, 8, 3, 1, 2, seed=3)
    drho[:] = 0.2
    surf[10] = 2.0
    out = ctx.pointmass(g, drho, surf)
    assert not np.isfinite(out[10]) and np.all(np.isfinite(np.delete(out, 10)))


@pytest.mark.parametrize("lift", [1e-3, 0.5, 7.3, 33.0, 1e3, 1.04e6, 1.06e6, 3e6])
def test_every_pair(ctx, lift):
    """Single pairs, element by element, over a wide grid: r^2 in fixed point,
    near pairs whose r^2 is added in double instead, and heights around the
    fixed point's limit (2^20 spacings).  TOLERANCE: 5e-15, r^-3 to 1e-15 and
    three products here, as much again in the oracle."""
    g = ztm_gb300.make_grid(121, 47, 2, 1, 2, 0)
    n = 121 * 47 * 3
    surf = np.full(121 * 47, 1.0 + lift)
    w = np.zeros(121 * 47)
    for node, station in ((0, 5686), (121 * 47 + 121 * 20 + 60, 121 * 23 + 57), (n - 1, 0)):
        drho = np.zeros(n)
        drho[node] = 0.7
        ref = oracle.pointmass_tfm(g, drho, surf)
        assert np.all(np.abs(ctx.pointmass(g, drho, surf) - ref) <= 5e-15 * np.abs(ref))
        w[:] = 0.0
        w[station] = 1.3
        ref = oracle.pointmass_adjoint(g, surf, w)
        assert np.all(np.abs(ctx.pointmass_adjoint(g, surf, w) - ref) <= 5e-15 * np.abs(ref))
