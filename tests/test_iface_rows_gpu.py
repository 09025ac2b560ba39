"""The mixed interface kernels where a block's or a tile's columns lie in one
row, in the adjoint's table of rows (64 columns in x and more) and in more rows,
with odd station counts around a tile of 256 (padding stations), and the misfit
whose residual comes out of the forward's last kernel.

TOLERANCE: 1e-6 normwise between mixed and double, that of the interface tests;
the misfit call against its parts 1e-12 (the same kernels; near pairs meet in
double atomics)."""
import numpy as np
import pytest

import ztm_gb300
from helpers import rel_err

pytestmark = pytest.mark.gpu


def case(nx, ny, ns, seed):
    rng = np.random.default_rng(seed)
    dx, dy = 2000.0, 1500.0
    im = ztm_gb300.make_imesh(nx, ny, dx, dy, -45000.0, x0=-300.0, y0=120.0)
    depth = 30000.0 + 4000.0 * rng.normal(size=nx * ny).clip(-2.0, 2.0)
    depth[rng.random(nx * ny) < 0.1] = 500.0  # tops close to the stations
    rho = rng.normal(300.0, 100.0, nx * ny)
    st = np.stack([rng.uniform(-0.1, 1.1, ns) * nx * dx, rng.uniform(-0.1, 1.1, ns) * ny * dy,
                   rng.uniform(10.0, 3000.0, ns)], axis=1)
    return im, depth, rho, st, rng.normal(size=ns)


@pytest.mark.parametrize("nx,ny,ns", [(5, 30, 33), (31, 9, 257), (62, 5, 1), (63, 5, 40),
                                      (64, 7, 259), (65, 4, 255), (127, 3, 300), (128, 2, 2),
                                      (130, 5, 513), (300, 1, 65)])
def test_rows(ctx, nx, ny, ns):
    im, depth, rho, st, r = case(nx, ny, ns, seed=nx + ny + ns)
    gz = ctx.interface(im, depth, rho, st, precision="mixed")
    ref = ctx.interface(im, depth, rho, st, precision="fp64")
    assert rel_err(gz, ref) <= 1e-6
    v = np.random.default_rng(1).normal(0.0, 100.0, nx * ny)
    assert rel_err(ctx.interface_jvp(im, depth, rho, st, v, precision="mixed"),
                   ctx.interface_jvp(im, depth, rho, st, v, precision="fp64")) <= 1e-6
    for a, b in zip(ctx.interface_adjoint(im, depth, rho, st, r, precision="mixed"),
                    ctx.interface_adjoint(im, depth, rho, st, r, precision="fp64")):
        assert rel_err(a, b) <= 1e-6
    for p in ("mixed", "fp64"):
        g0 = gz if p == "mixed" else ref
        mis, g, gr, gd = ctx.interface_misfit(im, depth, rho, st, g0 - r, precision=p)
        assert np.array_equal(g, g0)
        res = g0 - (g0 - r)
        assert mis == pytest.approx(0.5 * np.sum(res ** 2), rel=1e-12)
        ar, ad = ctx.interface_adjoint(im, depth, rho, st, res, precision=p)
        assert rel_err(gr, ar) <= 1e-12 and rel_err(gd, ad) <= 1e-12
