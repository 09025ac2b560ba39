"""The mixed forward of few stations over a small mesh (far_split_kernel) gives
the bits of the persistent kernel, which a context that counts forms runs:
station counts around a warp and a block, layer counts around 8, 16, 32 and 64
(sums per column), columns that end inside a stage, far column pairs, near
columns, stations beside and below the mesh.

TOLERANCE: none (bitwise)."""
import numpy as np
import pytest

import ztm_gb300

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("nx,ny,nz,ns", [(33, 29, 14, 63), (1, 1, 1, 1), (5, 7, 8, 32),
                                         (64, 64, 33, 100), (97, 3, 24, 65), (200, 5, 64, 31),
                                         (16, 16, 40, 129), (33, 31, 9, 600), (300, 9, 16, 33),
                                         (12, 10, 130, 40)])
def test_bits_of_the_persistent_kernel(nx, ny, nz, ns, precision):
    rng = np.random.default_rng(nx + ny + nz + ns)
    mesh = ztm_gb300.make_mesh(nx, ny, nz, 1000.0, 1200.0, 400.0, x0=-50.0, y0=30.0, z_top=100.0)
    rho = rng.normal(0.0, 300.0, nx * ny * nz)
    rho[rng.random(rho.size) < 0.2] = 0.0
    st = np.stack([rng.uniform(-0.3, 1.3, ns) * nx * 1000.0, rng.uniform(-0.3, 1.3, ns) * ny * 1200.0,
                   rng.uniform(-500.0, 4000.0, ns)], axis=1)
    with ztm_gb300.GravityContext(0) as a, ztm_gb300.GravityContext(0) as b:
        b.count_forms(True)
        assert np.array_equal(a.prism(mesh, rho, st, precision=precision),
                              b.prism(mesh, rho, st, precision=precision))


@pytest.mark.parametrize("ns", [1, 2, 33, 511, 512, 513])
def test_station_order_by_counting(ctx, ns):
    """Up to 512 stations are ordered by counting, more by the library's sort:
    stations that share cells, lie outside the mesh or twice in the list.
    TOLERANCE: 1e-6 of the largest value against double, that of the mixed
    method."""
    rng = np.random.default_rng(ns)
    mesh = ztm_gb300.make_mesh(23, 31, 12, 900.0, 1100.0, 500.0, z_top=50.0)
    rho = rng.normal(0.0, 300.0, 23 * 31 * 12)
    st = np.stack([rng.uniform(-0.5, 1.5, ns) * 23 * 900.0, rng.uniform(-0.5, 1.5, ns) * 31 * 1100.0,
                   rng.uniform(60.0, 3000.0, ns)], axis=1)
    st[ns // 2:][: ns // 4] = st[: ns // 4]
    a = ctx.prism(mesh, rho, st, precision="mixed")
    b = ctx.prism(mesh, rho, st, precision="fp64")
    assert np.max(np.abs(a - b)) <= 1e-6 * np.max(np.abs(b))
