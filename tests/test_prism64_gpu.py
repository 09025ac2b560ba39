"""The double prism forward and adjoint with the far field in float pairs
(prism64.cu) against the oracle: odd column counts (a half-empty column
pair), layer counts off the adjoint's groups of 8, one and many station
tiles, odd station counts, stations on, in and below the mesh, far outside
it, and inputs of extreme magnitude.

TOLERANCE: 1e-10 normwise (the oracle's own 8-corner sums in double, whose
cancellation grows like (R/a)^3, as in the other double prism tests)."""
import numpy as np
import pytest

import oracle
import ztm_gb300
from helpers import awkward_stations, rel_err

pytestmark = pytest.mark.gpu


def mesh_and_density(nx, ny, nz, dx, dy, dz, seed):
    rng = np.random.default_rng(seed)
    mesh = ztm_gb300.make_mesh(nx, ny, nz, dx, dy, dz, x0=-3000.0, y0=1500.0, z_top=200.0)
    rho = rng.normal(0.0, 200.0, nx * ny * nz)
    rho[rng.random(rho.size) < 0.1] = 0.0
    return mesh, rho


SHAPES = [(41, 37, 19, 1000.0, 1000.0, 500.0), (64, 33, 16, 2000.0, 1600.0, 500.0),
          (35, 35, 33, 500.0, 500.0, 500.0), (127, 29, 9, 1000.0, 800.0, 1000.0)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("n_random", [0, 24, 151])
def test_forward_and_adjoint_match_oracle(ctx, shape, n_random):
    mesh, rho = mesh_and_density(*shape, seed=7)
    st = awkward_stations(mesh, n_random=n_random)[:-1 if n_random == 24 else None]
    assert rel_err(ctx.prism(mesh, rho, st, precision="fp64"), oracle.prism_mesh(mesh, rho, st)) <= 1e-10
    r = np.random.default_rng(8).normal(0.0, 10.0, len(st))
    r[::7] = 0.0
    assert rel_err(ctx.adjoint(mesh, st, r, precision="fp64"), oracle.mesh_adjoint(mesh, st, r)) <= 1e-10


def test_extreme_magnitudes_and_distances(ctx):
    """Densities and residuals beyond float's range scale out exactly; a
    station a million cells away (beyond every form's powers) stays finite
    and is the point mass there to the ratio of sizes."""
    mesh, rho = mesh_and_density(41, 37, 19, 1000.0, 1000.0, 500.0, seed=9)
    st = awkward_stations(mesh, n_random=20)
    g = ctx.prism(mesh, rho, st, precision="fp64")
    r = np.random.default_rng(10).normal(0.0, 1.0, len(st))
    a = ctx.adjoint(mesh, st, r, precision="fp64")
    for e in (600, -600):
        assert np.array_equal(ctx.prism(mesh, np.ldexp(rho, e), st, precision="fp64"), np.ldexp(g, e))
        assert rel_err(np.ldexp(ctx.adjoint(mesh, st, np.ldexp(r, e), precision="fp64"), -e), a) <= 1e-14
    far = np.array([[1.0e9, 2.0e9, 5.0e8], [2.0e4, 2.0e4, 3.0e9], [2.0e4, 2.0e4, 3000.0]])
    g = ctx.prism(mesh, np.abs(rho), far, precision="fp64")
    mass = np.abs(rho).sum() * mesh.dx * mesh.dy * mesh.dz
    c = np.array([mesh.x0 + 20.5e3, mesh.y0 + 18.5e3, mesh.z_top - 4750.0])
    d = far[:2] - c
    pm = ztm_gb300.DEFAULT_G * 1e5 * mass * d[:, 2] / np.sum(d * d, 1) ** 1.5
    assert np.all(np.abs(g[:2] / pm - 1.0) <= 1e-3)  # the mass's offset from the centre over d


def test_not_finite_inputs_reach_the_results(ctx):
    mesh, rho = mesh_and_density(41, 37, 19, 1000.0, 1000.0, 500.0, seed=11)
    st = awkward_stations(mesh, n_random=20)
    rho[rho.size // 2] = np.nan
    assert np.all(np.isnan(ctx.prism(mesh, rho, st, precision="fp64")))
    r = np.ones(len(st))
    r[3] = np.inf
    assert not np.any(np.isfinite(ctx.adjoint(mesh, st, r, precision="fp64")))


@pytest.mark.parametrize("n_random", [1, 40, 3000])
def test_mixed_near_regions_in_parts(ctx, n_random):
    """The mixed forward with a station's near vertices split over several
    warps (few stations) and whole (many) against the double forward."""
    mesh, rho = mesh_and_density(33, 29, 14, 1000.0, 800.0, 500.0, seed=12)
    st = awkward_stations(mesh, n_random=n_random)
    assert rel_err(ctx.prism(mesh, rho, st, precision="mixed"),
                   ctx.prism(mesh, rho, st, precision="fp64")) <= 1e-6
