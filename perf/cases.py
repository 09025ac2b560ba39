"""The work that users of the gravity library have it do, case by case.

Every case goes through a public call of `ztm_gb300.GravityContext` with
inputs drawn from a seed: smooth random density fields, draped or levelled
stations, TFM-like grids.  Sizes are those of the library's own benchmark
workloads and tests, or ordinary odd ones between them.

The kinds of work:
  pointmass  the reference's point-mass field (what the optimiser's C++ driver
             calls for every model), host or device arrays, node list or
             threshold, double or float
  misfit     that field's misfit with its density gradient (one forward and
             one transposed sum: what replaces the finite-difference Jacobian)
  prism      the closed-form prism forward, mixed precision or plain double
  adjoint    its density gradient J^T r
  step       a forward, the residual and the gradient: one inversion step
  interface  misfit and both gradients of an interface (Moho) model
  batch      line-search trials on one mesh beside independent regional meshes
  lm         the damped Gauss-Newton trial models of one optimiser iteration
  invert     a whole interface inversion on host arrays
"""
import math

import numpy as np
import torch

import ztm_gb300

G5 = ztm_gb300.DEFAULT_G * 1.0e5  # m/s^2 -> mGal
_context = None


def _ctx():
    """The program's context: one for its life, as a caller keeps it."""
    global _context
    if _context is None:
        _context = ztm_gb300.GravityContext(0)
    return _context


# ---------------------------------------------------------------------------
# the cases
def _pm(kind, precision, di, dj, dk, fh, fv, bfr, arrays, use_list):
    return {"kind": kind, "precision": precision, "di": di, "dj": dj, "dk": dk, "fh": fh, "fv": fv,
            "bfr": bfr, "arrays": arrays, "list": use_list}


def _mesh(kind, precision, nx, ny, nz, dx, dy, dz, nsx, nsy, relief):
    """relief: station heights 0..relief metres on a fractal surface; 0: a
    level 100 m above the mesh."""
    return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "dx": dx, "dy": dy,
            "dz": dz, "nsx": nsx, "nsy": nsy, "relief": relief}


def listed():
    return [
        # the drop-in call of the C++ optimiser: its own 61 x 61 x 33 grid,
        # double, host vectors, its list of selected nodes
        dict(_pm("pointmass", "fp64", 61, 61, 33, 1, 2, 10, "host", True), name="tfm_forward"),
        # the same grid's misfit and density gradient in one call
        dict(_pm("misfit", "fp64", 61, 61, 33, 1, 2, 10, "host", False), name="tfm_gradient"),
        # the point-mass field in float (the reference's GPU arithmetic) on a
        # larger survey, every node a station
        dict(_pm("pointmass", "fp32", 128, 128, 33, 1, 2, 0, "device", False), name="survey_fp32"),
        # plain double prism forward, 64 x 64 x 32 prisms, 32 x 32 stations
        dict(_mesh("prism", "fp64", 64, 64, 32, 2000.0, 2000.0, 1000.0, 32, 32, 0.0),
             name="plain_64x64x32"),
        # one double inversion step (forward and gradient) on an odd regional mesh
        dict(_mesh("step", "fp64", 61, 47, 23, 1000.0, 1000.0, 500.0, 27, 25, 1500.0),
             name="regional_step_fp64"),
        # the flagship: mixed precision, draped stations over a 256 x 256 x 64 mesh
        dict(_mesh("prism", "mixed", 256, 256, 64, 1000.0, 1000.0, 500.0, 128, 128, 3000.0),
             name="draped_256x256x64"),
        # its density gradient
        dict(_mesh("adjoint", "mixed", 256, 256, 64, 1000.0, 1000.0, 500.0, 128, 128, 3000.0),
             name="draped_adjoint"),
        # a small local model with a few stations: a call's latency
        dict(_mesh("prism", "mixed", 33, 29, 14, 1000.0, 800.0, 500.0, 9, 7, 800.0),
             name="local_33x29x14"),
        # misfit and gradients of a 256 x 256 Moho under 128 x 128 stations
        {"name": "moho_256", "kind": "interface", "precision": "mixed", "nx": 256, "ny": 256,
         "cell": 1000.0, "nsx": 128, "nsy": 128},
        # a line search: 32 trial models on the draped mesh and 16 regional
        # meshes of uneven size, in one call
        {"name": "trials_32_regions_16", "kind": "batch", "nx": 256, "ny": 256, "nz": 64,
         "nsx": 128, "nsy": 128, "trials": 32, "regions": 16},
        # the trial models of a damped Gauss-Newton iteration, 4 damping pairs
        {"name": "lm_12000x2700", "kind": "lm", "rows": 12000, "cols": 2700, "pairs": 4},
        # a short whole inversion for the depth of an interface
        {"name": "invert_128", "kind": "invert", "nx": 128, "ny": 128, "cell": 1000.0, "nsx": 64,
         "nsy": 64, "iterations": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid_dims(rng, most):
    """Fine-grid dims of a point-mass case within `most` node-station pairs."""
    while True:
        di, dj, dk = _log(rng, 21, 128), _log(rng, 21, 128), rng.randint(9, 40)
        fh, fv = (2, rng.choice([1, 2])) if rng.random() < 0.2 else (1, rng.choice([1, 2, 2, 3]))
        bfr = rng.randint(0, 8)
        nodes = ((di - 1) * fh + 1) * ((dj - 1) * fh + 1) * ((dk - 1) * fv + 1)
        if nodes * (di - 2 * bfr) * (dj - 2 * bfr) <= most:
            return di, dj, dk, fh, fv, bfr


def _mesh_dims(rng, most):
    """Mesh and station dims within `most` prism-station pairs."""
    while True:
        nx, ny, nz = _log(rng, 17, 256), _log(rng, 17, 256), _log(rng, 9, 80)
        nsx, nsy = _log(rng, 5, 128), _log(rng, 5, 128)
        if nx * ny * nz * nsx * nsy <= most:
            dx = rng.choice([500.0, 1000.0, 2000.0])
            dy = dx * rng.choice([0.8, 1.0, 1.0])
            dz = dx * rng.choice([0.25, 0.5, 0.5, 1.0])
            return nx, ny, nz, dx, dy, dz, nsx, nsy, rng.choice([0.0, 800.0, 3000.0])


def draw(rng):
    kind = rng.choice(["pointmass", "pointmass", "misfit", "prism", "prism", "prism", "adjoint",
                       "step", "interface", "batch", "lm", "invert"])
    if kind in ("pointmass", "misfit"):
        precision = rng.choice(["fp64", "fp64", "fp32"])
        dims = _grid_dims(rng, 2.0e9 if precision == "fp64" else 2.0e10)
        return _pm(kind, precision, *dims, rng.choice(["host", "device"]), rng.random() < 0.5)
    if kind in ("prism", "adjoint", "step"):
        precision = rng.choice(["mixed", "mixed", "fp64"])
        return _mesh(kind, precision, *_mesh_dims(rng, 2.0e8 if precision == "fp64" else 6.0e10))
    if kind == "interface":
        return {"kind": kind, "precision": "mixed", "nx": _log(rng, 24, 256),
                "ny": _log(rng, 24, 256), "cell": rng.choice([500.0, 1000.0, 2000.0]),
                "nsx": _log(rng, 9, 128), "nsy": _log(rng, 9, 128)}
    if kind == "batch":
        return {"kind": kind, "nx": _log(rng, 40, 160), "ny": _log(rng, 40, 160),
                "nz": rng.randint(20, 64), "nsx": _log(rng, 16, 96), "nsy": _log(rng, 16, 96),
                "trials": rng.randint(2, 32), "regions": rng.randint(0, 6)}
    if kind == "lm":
        cols = _log(rng, 60, 2000)
        return {"kind": kind, "rows": cols * rng.randint(2, 5) + rng.randint(0, 99), "cols": cols,
                "pairs": rng.randint(1, 4)}
    return {"kind": "invert", "nx": _log(rng, 48, 128), "ny": _log(rng, 48, 128),
            "cell": rng.choice([500.0, 1000.0]), "nsx": _log(rng, 24, 64),
            "nsy": _log(rng, 24, 64), "iterations": rng.randint(4, 10)}


# ---------------------------------------------------------------------------
# inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _smooth(g, shape, spacing, corr):
    """Unit-variance Gaussian random field with a Gaussian correlation."""
    f = torch.fft.rfftn(_randn(g, *shape))
    for ax, (n, d) in enumerate(zip(shape, spacing)):
        last = ax == len(shape) - 1
        k = (torch.fft.rfftfreq if last else torch.fft.fftfreq)(n, d, device="cuda",
                                                                 dtype=torch.float64)
        w = torch.exp(-0.5 * (math.pi * corr * k) ** 2)
        f *= w.reshape([-1 if a == ax else 1 for a in range(len(shape))])
    out = torch.fft.irfftn(f, s=shape)
    out = out - out.mean()
    return out / out.std()


def _fractal(g, ny, nx):
    """Fractal surface (H = 0.8) scaled to 0..1."""
    f = torch.fft.rfft2(_randn(g, ny, nx))
    ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = math.inf
    s = torch.fft.irfft2(f * k ** -1.8, s=(ny, nx))
    return (s - s.min()) / (s.max() - s.min())


def _stations(g, lx, ly, nsx, nsy, relief, z0=0.0):
    """A regular survey over lx x ly metres, draped or level."""
    xs = (torch.arange(nsx, device="cuda", dtype=torch.float64) + 0.5) * (lx / nsx)
    ys = (torch.arange(nsy, device="cuda", dtype=torch.float64) + 0.5) * (ly / nsy)
    z = _fractal(g, nsy, nsx) * relief if relief else torch.full((nsy, nsx), 100.0, device="cuda",
                                                                 dtype=torch.float64)
    X, Y = xs[None, :].expand(nsy, nsx), ys[:, None].expand(nsy, nsx)
    return torch.stack([X, Y, z + z0], dim=-1).reshape(-1, 3).contiguous()


def _density(g, c, amplitude=100.0):
    """Density contrasts of a mesh (kg/m^3): correlated over five cells, and
    a few boxes of one density."""
    shape = (c["nz"], c["ny"], c["nx"])
    f = _smooth(g, shape, (c["dz"], c["dy"], c["dx"]), 5.0 * c["dx"]) * amplitude
    lo = torch.rand(8, 3, generator=g, device="cuda").tolist()
    for i, u in enumerate(lo):
        b = [slice(int(a * n), int(a * n) + max(1, n // 8)) for a, n in zip(u, shape)]
        f[b[0], b[1], b[2]] += 300.0 if i % 2 else -300.0
    return f.reshape(-1)


def _pm_inputs(c, g):
    """drho (g/cc) over the fine grid and the station heights: correlated
    contrasts at depth, nothing within one grid unit of the surface, a third
    of the nodes without a contrast, as the density builder leaves them."""
    ii, jj = (c["di"] - 1) * c["fh"] + 1, (c["dj"] - 1) * c["fh"] + 1
    kk = (c["dk"] - 1) * c["fv"] + 1
    f = _smooth(g, (kk, jj, ii), (1.0 / c["fv"], 1.0 / c["fh"], 1.0 / c["fh"]), 4.0) * 0.1
    f[torch.abs(f) < 0.04] = 0.0
    surf = (c["dk"] - 3) + 0.3 + 0.3 * _fractal(g, c["dj"], c["di"]).reshape(-1)
    k = torch.arange(kk, device="cuda", dtype=torch.float64) / c["fv"]
    f[k > float(surf.min()) - 1.0] = 0.0
    return f.reshape(-1).contiguous(), surf.contiguous()


def _moho(c, g):
    """Column tops between 20 and 45 km (bases at 45 km), contrast -400."""
    f = _smooth(g, (c["ny"], c["nx"]), (c["cell"], c["cell"]), 40000.0)
    depth = 20000.0 + (f - f.min()) / (f.max() - f.min()) * 25000.0
    rho = torch.full((c["nx"] * c["ny"],), -400.0, device="cuda", dtype=torch.float64)
    st = _stations(g, c["nx"] * c["cell"], c["ny"] * c["cell"], c["nsx"], c["nsy"], 0.0, -100.0)
    return depth.reshape(-1).contiguous(), rho, st


def _line_columns(c, depth, rho, st):
    """Data of an inversion: the columns as vertical lines of mass."""
    x = (torch.arange(c["nx"], device="cuda", dtype=torch.float64) + 0.5) * c["cell"]
    y = (torch.arange(c["ny"], device="cuda", dtype=torch.float64) + 0.5) * c["cell"]
    h2 = ((x[None, None, :] - st[:, 0, None, None]) ** 2 +
          (y[None, :, None] - st[:, 1, None, None]) ** 2).reshape(st.shape[0], -1)
    zt, zb = st[:, 2, None] + depth[None, :], st[:, 2, None] + 45000.0
    return G5 * c["cell"] ** 2 * (((h2 + zt * zt).rsqrt() - (h2 + zb * zb).rsqrt()) @ rho)


def _mesh_of(c):
    return ztm_gb300.make_mesh(c["nx"], c["ny"], c["nz"], c["dx"], c["dy"], c["dz"])


def _imesh_of(c):
    return ztm_gb300.make_imesh(c["nx"], c["ny"], c["cell"], c["cell"], -45000.0)


def prepare(case, seed):
    c, g, s = case, _gen(seed), {"case": case, "ctx": _ctx()}
    if c["kind"] in ("pointmass", "misfit"):
        s["grid"] = ztm_gb300.make_grid(c["di"], c["dj"], c["dk"], c["fh"], c["fv"], c["bfr"])
        s["drho"], s["surf"] = _pm_inputs(c, g)
        s["data"] = 20.0 * _randn(g, c["di"] * c["dj"])
        s["nn"] = torch.nonzero(torch.abs(s["drho"]) > 0.001).reshape(-1).to(torch.int32) \
            if c["list"] else None
        if c["arrays"] == "host":
            for k in ("drho", "surf", "data", "nn"):
                s[k] = s[k].cpu().numpy() if s[k] is not None else None
    elif c["kind"] in ("prism", "adjoint", "step"):
        s["mesh"] = _mesh_of(c)
        s["rho"] = _density(g, c)
        s["st"] = _stations(g, c["nx"] * c["dx"], c["ny"] * c["dy"], c["nsx"], c["nsy"],
                            c["relief"])
        s["data"] = 20.0 * _randn(g, s["st"].shape[0])
    elif c["kind"] == "interface":
        s["mesh"] = _imesh_of(c)
        s["depth"], s["rho"], s["st"] = _moho(c, g)
        s["data"] = -150.0 + 20.0 * _randn(g, s["st"].shape[0])
    elif c["kind"] == "batch":
        cells = {"dx": 1000.0, "dy": 1000.0, "dz": 500.0}
        main = dict(c, **cells)
        m, p = _density(g, main), _smooth(g, (c["nz"], c["ny"], c["nx"]), (500.0, 1000.0, 1000.0),
                                          10000.0).reshape(-1) * 30.0
        alpha = torch.linspace(0.0, 2.0, c["trials"], device="cuda", dtype=torch.float64)
        s["jobs"] = [(_mesh_of(main), m[None, :] + alpha[:, None] * p[None, :],
                      _stations(g, c["nx"] * 1000.0, c["ny"] * 1000.0, c["nsx"], c["nsy"], 3000.0))]
        for r in _regions(c):
            s["jobs"].append((_mesh_of(r), _density(g, r)[None, :].contiguous(),
                              _stations(g, r["nx"] * 1000.0, r["ny"] * 1000.0, r["nsx"], r["nsy"],
                                        2000.0)))
    elif c["kind"] == "lm":
        n = c["cols"]
        s["J"] = _randn(g, c["rows"], n) * (0.1 + 9.9 * _rand(g, n))[None, :]
        s["r"], s["b"] = _randn(g, c["rows"]), _randn(g, n)
        s["sig"] = 0.05 + 1.95 * _rand(g, n)
        s["damping"] = torch.tensor([[1e-3, 1e-4], [1e-2, 1e-3], [0.1, 1e-2], [1.0, 1.0]],
                                    device="cuda", dtype=torch.float64)[:c["pairs"]].contiguous()
    elif c["kind"] == "invert":
        s["mesh"] = _imesh_of(c)
        depth, rho, st = _moho(c, g)
        data = _line_columns(c, depth, rho, st) + 0.05 * _randn(g, st.shape[0])
        s["depth0"] = np.full(depth.numel(), float(depth.mean()))
        s["rho"], s["st"], s["data"] = (t.cpu().numpy() for t in (rho, st, data))
    return s


def _regions(c):
    """The regional meshes of a batch: uneven sizes fixed by the case."""
    k = min(1.0, c["nx"] / 256.0)
    out = []
    for i in range(c["regions"]):
        u, v, w = (0.618 * i) % 1.0, (0.755 * i) % 1.0, (0.57 * i) % 1.0
        out.append({"nx": int(k * (64 + 128 * u)), "ny": int(k * (64 + 128 * v)),
                    "nz": max(8, int(k * (48 + 17 * w))), "dx": 1000.0, "dy": 1000.0, "dz": 500.0,
                    "nsx": max(4, int(k * (32 + 96 * w))), "nsy": max(4, int(k * (32 + 96 * u)))})
    return out


# ---------------------------------------------------------------------------
# one pass
def run(state):
    s, c = state, state["case"]
    ctx, kind = s["ctx"], c["kind"]
    if kind == "pointmass":
        return ctx.pointmass(s["grid"], s["drho"], s["surf"], nn=s["nn"], precision=c["precision"])
    if kind == "misfit":
        ssq, res, field, g, g0 = ctx.pointmass_misfit(s["grid"], s["drho"], s["surf"], s["data"],
                                                      g0=1.5, gsig=2.0, nn=s["nn"],
                                                      precision=c["precision"])
        return {"ssq": ssq, "res": res, "G": field, "g_drho": g, "g_g0": g0}
    if kind == "prism":
        return ctx.prism(s["mesh"], s["rho"], s["st"], precision=c["precision"])
    if kind == "adjoint":
        return ctx.adjoint(s["mesh"], s["st"], s["data"], precision=c["precision"])
    if kind == "step":
        gz = ctx.prism(s["mesh"], s["rho"], s["st"], precision=c["precision"])
        return gz, ctx.adjoint(s["mesh"], s["st"], gz - s["data"], precision=c["precision"])
    if kind == "interface":
        return ctx.interface_misfit(s["mesh"], s["depth"], s["rho"], s["st"], s["data"],
                                    precision=c["precision"])
    if kind == "batch":
        return ctx.batch(s["jobs"])
    if kind == "lm":
        return ctx.lm_steps(s["J"], s["r"], s["b"], s["sig"], s["damping"], return_jtj=True)
    return ctx.invert_interface(s["mesh"], s["depth0"], s["rho"], s["st"], s["data"], lam=1e-2,
                                iterations=c["iterations"])


# ---------------------------------------------------------------------------
def work(case):
    """Arrays in and out once (doubles) and the operations of the direct sums:
    12 a point-mass pair, 20 a prism pair, 40 an interface pair and gradient,
    J^T J and an LU of each damped system."""
    c, kind = case, case["kind"]
    if kind in ("pointmass", "misfit"):
        n = ((c["di"] - 1) * c["fh"] + 1) * ((c["dj"] - 1) * c["fh"] + 1) * \
            ((c["dk"] - 1) * c["fv"] + 1)
        ns = max(0, c["di"] - 2 * c["bfr"]) * max(0, c["dj"] - 2 * c["bfr"])
        both = 2 if kind == "misfit" else 1
        return {"bytes": 8.0 * (both * n + 2 * both * c["di"] * c["dj"]),
                "flops": 12.0 * both * n * ns}
    if kind in ("prism", "adjoint", "step"):
        n, ns = c["nx"] * c["ny"] * c["nz"], c["nsx"] * c["nsy"]
        both = 2 if kind == "step" else 1
        return {"bytes": 8.0 * (both * n + 4 * ns), "flops": 20.0 * both * n * ns}
    if kind in ("interface", "invert"):
        n, ns = c["nx"] * c["ny"], c["nsx"] * c["nsy"]
        return {"bytes": 8.0 * (4 * n + 5 * ns), "flops": 80.0 * n * ns * c.get("iterations", 1)}
    if kind == "batch":
        jobs = [dict(c, trials=c["trials"])] + [dict(r, trials=1) for r in _regions(c)]
        b = f = 0.0
        for j in jobs:
            n, ns = j["nx"] * j["ny"] * j["nz"], j["nsx"] * j["nsy"]
            b += 8.0 * (j["trials"] * n + (3 + j["trials"]) * ns)
            f += (18.0 + 2.0 * j["trials"]) * n * ns
        return {"bytes": b, "flops": f}
    m, n, nd = c["rows"], c["cols"], c["pairs"]
    return {"bytes": 8.0 * (m * n + n * n + nd * n), "flops": 1.0 * m * n * n + nd * 2.0 / 3.0 * n ** 3}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
def _phi(x, y, z):
    """Corner function x ln(y+r) + y ln(x+r) - z atan(xy/(zr))."""
    r = torch.sqrt(x * x + y * y + z * z)

    def xlog(a, b):
        v = torch.where(b >= 0, b + r, (a * a + z * z) / (r - b))
        return torch.where(a == 0, torch.zeros_like(v), a * torch.log(torch.where(a == 0, torch.ones_like(v), v)))

    at = z * torch.atan(x * y / (z * r))
    return xlog(x, y) + xlog(y, x) - torch.where(z == 0, torch.zeros_like(at), at)


def _unit_mesh(c, st):
    """U[s, l, iy, ix]: the unit responses of the mesh's prisms."""
    ax = [torch.arange(n + 1, device="cuda", dtype=torch.float64) for n in (c["nx"], c["ny"], c["nz"])]
    x = ax[0][None, None, None, :] * c["dx"] - st[:, 0, None, None, None]
    y = ax[1][None, None, :, None] * c["dy"] - st[:, 1, None, None, None]
    z = -ax[2][None, :, None, None] * c["dz"] - st[:, 2, None, None, None]
    x, y, z = torch.broadcast_tensors(x, y, z)
    return -torch.diff(torch.diff(torch.diff(_phi(x, y, z), dim=1), dim=2), dim=3)


def _mesh_exact(c, rho, st, resid=None):
    """(gz, g_rho); resid: the residual, or a function of gz."""
    n = c["nx"] * c["ny"] * c["nz"]
    step = max(1, int(2.0e8 / n))
    gz = torch.cat([G5 * (_unit_mesh(c, st[a:a + step]).reshape(-1, n) @ rho)
                    for a in range(0, st.shape[0], step)])
    if resid is None:
        return gz, None
    r = resid(gz)
    g = torch.zeros_like(rho)
    for a in range(0, st.shape[0], step):
        g += G5 * (r[a:a + step] @ _unit_mesh(c, st[a:a + step]).reshape(-1, n))
    return gz, g


def _pm_kernel(c, surf, sel):
    """K[station, selected node] of the point-mass sum, by station ranges."""
    ii, jj = (c["di"] - 1) * c["fh"] + 1, (c["dj"] - 1) * c["fh"] + 1
    x = (sel % ii).double() / c["fh"]
    y = ((sel // ii) % jj).double() / c["fh"]
    z = (sel // (ii * jj)).double() / c["fv"]
    b = c["bfr"]
    j0, i0 = torch.meshgrid(torch.arange(b, c["dj"] - b, device="cuda"),
                            torch.arange(b, c["di"] - b, device="cuda"), indexing="ij")
    m = (i0 + j0 * c["di"]).reshape(-1)
    i0, j0, k0 = i0.reshape(-1).double(), j0.reshape(-1).double(), surf[m]
    f = 66.7 / (c["fh"] ** 2 * c["fv"])
    step = max(1, int(2.0e8 / max(1, sel.numel())))
    for a in range(0, m.numel(), step):
        t = slice(a, a + step)
        dz = k0[t, None] - z[None, :]
        r2 = (i0[t, None] - x[None, :]) ** 2 + (j0[t, None] - y[None, :]) ** 2 + dz * dz
        yield m[t], f * dz * r2 ** -1.5


def _interface_exact(c, s):
    x0 = torch.arange(c["nx"] + 1, device="cuda", dtype=torch.float64) * c["cell"]
    y0 = torch.arange(c["ny"] + 1, device="cuda", dtype=torch.float64) * c["cell"]
    top, n = -s["depth"].reshape(c["ny"], c["nx"]), c["nx"] * c["ny"]
    step = max(1, int(1.0e8 / n))

    def units(st):
        sx, sy, sz = (st[:, k, None, None] for k in range(3))
        x, y = x0[None, None, :] - sx, y0[None, :, None] - sy
        zb = (-45000.0 - sz).expand(-1, c["ny"] + 1, c["nx"] + 1)
        u = -torch.diff(torch.diff(_phi(x.expand_as(zb), y.expand_as(zb), zb), dim=1), dim=2)
        zt = top[None] - sz
        w, face = -zt, 0.0
        for a in (0, 1):
            for b in (0, 1):
                xx, yy = x[..., a:a + c["nx"]].expand_as(zt), y[:, b:b + c["ny"], :].expand_as(zt)
                sign = 1.0 if a == b else -1.0
                u += sign * _phi(xx, yy, zt)
                face = face + sign * torch.atan(xx * yy / (w * torch.sqrt(xx * xx + yy * yy + w * w)))
        return u.reshape(-1, n), face.reshape(-1, n)

    gz, rng = [], range(0, s["st"].shape[0], step)
    for a in rng:
        gz.append(G5 * (units(s["st"][a:a + step])[0] @ s["rho"]))
    gz = torch.cat(gz)
    r = gz - s["data"]
    g_rho, g_dep = torch.zeros_like(s["rho"]), torch.zeros_like(s["rho"])
    for a in rng:
        u, face = units(s["st"][a:a + step])
        g_rho += G5 * (r[a:a + step] @ u)
        g_dep -= G5 * s["rho"] * (r[a:a + step] @ face)
    return (0.5 * (r * r).sum()).reshape(1), gz, g_rho, g_dep


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "invert" or work(c)["flops"] > 4.0e11 and kind != "lm":
        return None  # a whole inversion has no closed value; the largest sums take minutes
    s = prepare(c, seed)
    if kind in ("pointmass", "misfit"):
        drho, surf, data = (torch.as_tensor(s[k], device="cuda") for k in ("drho", "surf", "data"))
        sel = torch.nonzero(torch.abs(drho) > 0.001).reshape(-1)
        w = drho[sel]
        G = torch.zeros_like(surf)
        for m, K in _pm_kernel(c, surf, sel):
            G[m] = K @ w
        if kind == "pointmass":
            return G
        b, di, dj = c["bfr"], c["di"], c["dj"]
        res = torch.zeros_like(surf)
        inner = torch.zeros(dj, di, device="cuda", dtype=torch.bool)
        inner[b:dj - b, b:di - b] = True
        inner = inner.reshape(-1)
        res[inner] = (data[inner] - (G[inner] + 1.5)) / 2.0
        g = torch.zeros_like(drho)
        part = torch.zeros_like(w)
        for m, K in _pm_kernel(c, surf, sel):
            part += (-res[m]) @ K
        g[sel] = part
        flat = res.reshape(dj, di)[b:dj - b, b:di - b].t().reshape(-1)
        # on device the misfit comes as one-element arrays, on the host as numbers
        ssq, g0 = (flat * flat).sum().reshape(1), (-flat.sum()).reshape(1)
        if c["arrays"] == "host":
            ssq, g0 = float(ssq), float(g0)
        return {"ssq": ssq, "res": flat, "G": G, "g_drho": g, "g_g0": g0}
    if kind in ("prism", "adjoint", "step"):
        how = {"prism": None, "adjoint": lambda gz: s["data"], "step": lambda gz: gz - s["data"]}
        gz, g = _mesh_exact(c, s["rho"], s["st"], how[kind])
        return gz if kind == "prism" else g if kind == "adjoint" else (gz, g)
    if kind == "interface":
        return _interface_exact(c, s)
    if kind == "batch":
        jobs = [dict(c, dx=1000.0, dy=1000.0, dz=500.0)] + _regions(c)
        return [torch.stack([_mesh_exact(d, m, st)[0] for m in rho])
                for d, (_, rho, st) in zip(jobs, s["jobs"])] if c["trials"] <= 4 else None
    JJ = s["J"].t() @ s["J"]
    rhs, diag = s["J"].t() @ s["r"], torch.diagonal(JJ)
    B = []
    for d0, d1 in s["damping"].tolist():
        B.append(s["b"] + torch.linalg.solve(JJ + torch.diag(d0 * diag + d1 / s["sig"] ** 2), rhs))
    return torch.stack(B), JJ
