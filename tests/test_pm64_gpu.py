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
