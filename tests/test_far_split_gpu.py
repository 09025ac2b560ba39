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
