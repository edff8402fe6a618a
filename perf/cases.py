"""Timing cases of the pressure-Poisson path and the steps around it.

Each case is one thing a flow solver has this framework do, through the
binding of the C ABI (``fg``): pressure solves on device and host fields,
batches and served requests, a moving body's time step, re-tagging, the
projection steps and the momentum line SOR.  ``listed()`` gives the named
cases, ``draw(rng)`` one more of the same ranges, ``prepare`` what a program
holds before the call, ``run`` one pass, ``work`` what a pass cannot do
without, ``exact`` the result in 64 bits where it can be stated without the
library.

Fields are device tensors of shape (nz+2, ny+2, nx+2) (node counts): the
memory layout of the Fortran arrays (0:nx+1, 0:ny+1, 0:nz+1).  Sizes in a
case are cell counts.
"""
import functools
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RTOL = 1e-11  # relative residual at which the pressure is within 1e-9 of the discrete solution


def _package():
    """The package's directory name is no identifier: it goes by feicar_b200."""
    if "feicar_b200" not in sys.modules:
        d = os.path.join(ROOT, "feicar3d_3.0_febio_b200")
        spec = importlib.util.spec_from_file_location("feicar_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["feicar_b200"] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module("feicar_b200.fg"), importlib.import_module("feicar_b200.synth")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest solve a program makes (a coarse trial grid): launch latency
        dict(name="solve_32x16x16_mixed", kind="solve", nx=32, ny=16, nz=16, stretch=0.0, body=True,
             precision="mixed", nu1=2, nu2=2),
        # the plain FP64 method on a small grid with a sphere
        dict(name="solve_128x64x64_fp64", kind="solve", nx=128, ny=64, nz=64, stretch=0.0, body=True,
             precision="fp64", nu1=2, nu2=2),
        # a channel without a body on a ragged, stretched grid
        dict(name="solve_201x97x75_mixed", kind="solve", nx=201, ny=97, nz=75, stretch=1.5, body=False,
             precision="mixed", nu1=2, nu2=2),
        # a host program's FP64 solve: page-locked host fields in and out
        dict(name="host_256x128x128_fp64", kind="host", nx=256, ny=128, nz=128, stretch=0.0, body=False,
             precision="fp64", nu1=2, nu2=2),
        # the headline solve, with the smoothing steps the autotuner settles on
        dict(name="solve_512x256x256_mixed", kind="solve", nx=512, ny=256, nz=256, stretch=2.0, body=True,
             precision="mixed", nu1=2, nu2=1),
        # independent problems of uneven size solved together (parameter study)
        dict(name="batch_16_cubes_mixed", kind="batch", problems=16, lo=32, hi=112, precision="mixed"),
        # a few requests through the serving engine: tagging, set-up and solves overlapping
        dict(name="serve_4_requests", kind="serve", problems=4, lo=32, hi=72, steps=2, precision="mixed"),
        # one time step of a pitching plate: move, re-tag, lists, hierarchy, solve
        dict(name="plate_step_256x128x128", kind="plate", nx=256, ny=128, nz=128, precision="mixed"),
        # geometry alone: a sphere tagged on a stretched grid, lists read back
        dict(name="tag_256x256x256", kind="tag", nx=256, ny=256, nz=256, stretch=2.0, subdiv=5),
        # the projection steps either side of the solve on the largest grid
        dict(name="project_512x256x256", kind="project", nx=512, ny=256, nz=256, stretch=2.0, body=True,
             outflow=True),
        # one line-SOR pass of a velocity component and its residual
        dict(name="momentum_192x96x96", kind="momentum", nx=192, ny=96, nz=96, stretch=0.0, body=False,
             crank_nicolson=True),
        # the momentum iteration of a time step: three components, ghost cells, boundaries, residuals
        dict(name="solve_ad_128x64x64", kind="solve_ad", nx=128, ny=64, nz=64, stretch=0.0, iterations=2),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi, most):
        """Three extents between lo and hi, x up to twice the edge, at most `most` cells."""
        while True:
            e = size(lo, hi)
            n = [e * rng.choice((1, 2)) + rng.randint(-1, 1), e + rng.randint(-3, 3), e + rng.randint(-3, 3)]
            if n[0] * n[1] * n[2] <= most:
                return dict(nx=n[0], ny=n[1], nz=n[2])

    kind = rng.choice(("solve", "solve", "solve", "solve", "host", "batch", "serve", "plate", "tag", "project",
                       "project", "momentum", "momentum", "solve_ad"))
    stretch = rng.choice((0.0, 0.0, round(rng.uniform(1.0, 2.0), 2)))
    body = rng.random() < 0.6
    precision = rng.choice(("mixed", "mixed", "fp64"))
    if kind in ("solve", "host"):
        most = 256 ** 3 if precision == "mixed" else 6_000_000
        return dict(kind=kind, **grid(18, 256, most), stretch=stretch, body=body, precision=precision, nu1=2,
                    nu2=rng.choice((1, 2)))
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(4, 16), lo=size(24, 40), hi=size(64, 112), precision=precision)
    if kind == "serve":
        return dict(kind=kind, problems=rng.randint(2, 5), lo=size(24, 40), hi=size(48, 80),
                    steps=rng.randint(1, 3), precision=precision)
    if kind == "plate":
        e = rng.choice((64, 96, 128))
        return dict(kind=kind, nx=2 * e, ny=e, nz=e, precision=precision)
    if kind == "tag":
        return dict(kind=kind, **grid(32, 256, 256 ** 3), stretch=stretch, subdiv=rng.choice((4, 5)))
    if kind == "project":
        return dict(kind=kind, **grid(24, 256, 512 * 256 * 256), stretch=stretch, body=body,
                    outflow=rng.random() < 0.5)
    if kind == "momentum":
        return dict(kind=kind, **grid(16, 112, 192 * 96 * 96), stretch=stretch, body=body,
                    crank_nicolson=rng.random() < 0.7)
    return dict(kind=kind, **grid(24, 64, 128 * 64 * 64), stretch=stretch, iterations=rng.randint(1, 3))


# ------------------------------------------------------------------ inputs
def _lengths(case):
    """The domain: unit aspect of the cells on average; 4 across the smaller
    of y and z, 2 on the coarsest grids and 8 on the finest."""
    n = min(case["ny"], case["nz"])
    h = (2.0 if n < 24 else 4.0 if n < 200 else 8.0) / n
    return case["nx"] * h, case["ny"] * h, case["nz"] * h


def _nodes(n, length, beta):
    """n + 1 nodes on [0, length], clustered toward the middle for beta > 0."""
    eta = np.arange(n + 1, dtype=np.float64) / n
    if beta <= 0.0:
        return length * eta
    y = 0.5 * length * (1.0 + np.arctanh((2.0 * eta - 1.0) * math.tanh(beta)) / beta)
    y[0], y[-1] = 0.0, length
    return y


def _axes(case):
    lx, ly, lz = _lengths(case)
    b = case.get("stretch", 0.0)
    return _nodes(case["nx"], lx, 0.0), _nodes(case["ny"], ly, b), _nodes(case["nz"], lz, b)


class _Axis:
    """Node positions with the mirrored outer nodes, cell centres, widths
    and centre distances of one axis (index 0..n+1, n nodes), 64 bits."""

    def __init__(self, xn, device):
        n = len(xn)
        x = np.zeros(n + 2)
        x[1:n + 1] = xn
        x[0] = 2.0 * x[1] - x[2]
        x[n + 1] = 2.0 * x[n] - x[n - 1]
        xc = np.zeros(n + 2)
        xc[:n + 1] = 0.5 * (x[1:] + x[:-1])
        xc[n + 1] = x[n + 1]
        self.n = n
        self.x, self.xc = (torch.from_numpy(a).to(device) for a in (x, xc))
        self.d = self.x[1:] - self.x[:-1]       # width of cell i (0..n)
        self.dc = self.xc[1:] - self.xc[:-1]    # distance of centres i and i + 1
        # share of cell i in the value at its lower node
        self.f = torch.zeros(n + 2, dtype=torch.float64, device=device)
        self.f[1:] = (self.x[1:] - self.xc[:-1]) / self.dc


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _smooth(shape, gen, passes=3):
    """Gaussian noise after `passes` [1, 2, 1] / 4 filters per axis."""
    a = torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")
    for ax in range(3):
        for _ in range(passes):
            n = a.shape[ax]
            p = torch.cat([a.narrow(ax, 0, 1), a, a.narrow(ax, n - 1, 1)], dim=ax)
            a = 0.25 * p.narrow(ax, 0, n) + 0.5 * p.narrow(ax, 1, n) + 0.25 * p.narrow(ax, 2, n)
    return a


def _mirror(f, outlet):
    """The outer layers copy their neighbours (homogeneous Neumann); at an
    outlet (the far x face) they reflect them about zero (Dirichlet)."""
    f[:, :, 0] = f[:, :, 1]
    f[:, :, -2] = -f[:, :, -3] if outlet else f[:, :, -3]
    f[:, 0] = f[:, 1]
    f[:, -2] = f[:, -3]
    f[0] = f[1]
    f[-2] = f[-3]


def _laplacian(axes, p):
    """The 7-point operator on the interior cells, 0 elsewhere."""
    X, Y, Z = axes
    out = torch.zeros_like(p)
    c = p[1:-2, 1:-2, 1:-2]
    acc = torch.zeros_like(c)
    for dim, A in ((2, X), (1, Y), (0, Z)):
        n = A.n - 1
        shape = [1, 1, 1]
        shape[dim] = n
        am = (1.0 / (A.dc[0:n] * A.d[1:n + 1])).view(shape)
        ap = (1.0 / (A.dc[1:n + 1] * A.d[1:n + 1])).view(shape)
        full = p[1:-2, 1:-2, :] if dim == 2 else p[1:-2, :, 1:-2] if dim == 1 else p[:, 1:-2, 1:-2]
        acc += am * (full.narrow(dim, 0, n) - c) + ap * (full.narrow(dim, 2, n) - c)
    out[1:-2, 1:-2, 1:-2] = acc
    return out


_CORNERS = ((0, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 0), (0, 0, 1), (0, 1, 1), (1, 1, 1), (1, 0, 1))


def _rows(grid, *lists):
    """Element indices and weights of interpolation rows (ijk, cell, 8 weights);
    a row's own corner carries no weight (homogeneous Neumann data)."""
    NX, NY = grid.nx + 2, grid.ny + 2
    tgt, src, w = [], [], []
    for r in lists:
        t, c = r["ijk"].astype(np.int64), r["cell"].astype(np.int64)
        e = c[:, None, :] + np.array(_CORNERS, dtype=np.int64)[None]
        tgt.append(t[:, 0] + NX * (t[:, 1] + NY * t[:, 2]))
        src.append(e[..., 0] + NX * (e[..., 1] + NY * e[..., 2]))
        ww = r["coefN"].copy()
        ww[src[-1] == tgt[-1][:, None]] = 0.0
        w.append(ww)
    return [torch.from_numpy(np.concatenate(a)).cuda() for a in (tgt, src, w)]


def _outlet(case):
    """Whether the far x face holds p = 0: in the cases whose result is the
    solver's own field.  With no such face the pressure is known up to a
    constant: the step then ends with update_pressure, as in the flow solver,
    which also clears the domain's edge lines (they would hold it)."""
    return case["kind"] in ("host", "batch", "serve")


def _potential(grid, gen, outlet):
    """Smoothed noise on the interior cells with its outer layers."""
    phi = torch.zeros(grid.shape[::-1], dtype=torch.float64, device="cuda")
    phi[1:-2, 1:-2, 1:-2] = _smooth((grid.nz - 1, grid.ny - 1, grid.nx - 1), gen)
    _mirror(phi, outlet)
    return phi


def _device_axes(axes):
    return [_Axis(a, "cuda") for a in axes]


def _rhs(case, case_handle, grid, axes, masks, gen):
    """A compatible right-hand side: the operator applied to smoothed noise
    whose ghost and dead values satisfy the body's interpolation rows."""
    phi = _potential(grid, gen, _outlet(case))
    if masks is not None:
        ib, gh, dd = (torch.from_numpy(np.ascontiguousarray(a.T)).cuda() for a in masks)
        phi[(ib == 1) & (dd != -1)] = 0.0
        tgt, src, w = _rows(grid, case_handle.dead_rows(), case_handle.ghost_rows())
        flat = phi.view(-1)
        for _ in range(500):
            new = (w * flat[src]).sum(dim=1)
            step = float((new - flat[tgt]).abs().max()) if len(tgt) else 0.0
            flat[tgt] = new
            if step <= 1e-15 * max(1.0, float(phi.abs().max())):
                break
    rhs = _laplacian(_device_axes(axes), phi)
    if masks is not None:
        rhs[(ib != 0) | (gh != 0)] = 0.0
    return rhs


@functools.lru_cache(maxsize=8)
def _icosphere(subdiv):
    return _package()[1].icosphere(subdiv)


def _ball(centre, semi_axes, rotation, subdiv):
    _, synth = _package()
    v, t = _icosphere(subdiv)
    m = rotation @ np.diag(np.asarray(semi_axes, dtype=np.float64))
    return synth.Body(verts=np.asarray(centre, dtype=np.float64)[None, :] + v @ m.T, tri=t)


def _sphere(case, subdiv):
    """A sphere of diameter 1 a quarter down the domain."""
    lx, ly, lz = _lengths(case)
    return _ball((0.25 * lx, 0.5 * ly, 0.5 * lz), (0.5, 0.5, 0.5), np.eye(3), subdiv)


def _ellipsoid(rng):
    _, synth = _package()
    return _ball((0.5, 0.5, 0.5), rng.uniform(0.15, 0.35, size=3), synth.random_rotation(rng), 4)


def _config(case):
    fg, _ = _package()
    pbc = [fg.FG_PBC_NEUMANN] * 6
    if _outlet(case):
        pbc[1] = fg.FG_PBC_DIRICHLET
    prec = fg.FG_PREC_MIXED if case.get("precision") == "mixed" else fg.FG_PREC_FP64
    return fg.default_config(precision=prec, rtol=RTOL, max_cycles=200, nu1=case.get("nu1", 2),
                             nu2=case.get("nu2", 2), pbc=pbc)


def _tagged(case, grid, body, stream):
    """A case with its geometry tagged and its hierarchy prepared, on `stream`."""
    fg, _ = _package()
    c = fg.Case(grid, _config(case))
    c.set_stream(stream.cuda_stream)
    if body is not None:
        c.add_body(body)
        c.set_iblank_body_fast()
        masks = c.gcm_set_internal_boundary()
    else:  # an open channel: every cell fluid, no interpolation rows
        masks, none = None, np.zeros((0, 3), dtype=np.int32)
        rows = dict(ijk=none, cell=none, coefN=np.zeros((0, 8)), probe=np.zeros(0), ip=np.zeros((0, 3)))
        c.set_geometry(*[np.zeros(grid.shape, dtype=np.int8, order="F") for _ in range(3)], rows, rows)
    c.mg_prepare()
    return c, masks


def _pinned(t):
    """A page-locked copy of a device field and its Fortran-ordered view."""
    p = t.cpu().pin_memory()
    return p, p.numpy().transpose(2, 1, 0)


def _edges(case):
    n, lo, hi = case["problems"], case["lo"], case["hi"]
    return [int(round(lo * (hi / lo) ** (q / max(1, n - 1)))) for q in range(n)]


def _cube(edge):
    _, synth = _package()
    axes = [np.arange(edge + 1) / float(edge)] * 3
    return synth.Grid(*axes), axes


def _flow(grid, gen):
    """A unit stream with smoothed noise: u, v, w over the whole arrays."""
    sh = grid.shape[::-1]
    u, v, w = (0.1 * _smooth(sh, gen) for _ in range(3))
    u += 1.0
    return u, v, w


def _step(case):
    """A time step at a Courant number of 0.3 on the unit stream."""
    lx, ly, lz = _lengths(case)
    return 0.3 * lx / case["nx"]


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    fg, synth = _package()
    kind, gen = case["kind"], _generator(seed)
    s = dict(kind=kind, fg=fg, case=case)
    s["stream"] = stream = torch.cuda.Stream()
    if kind in ("batch", "serve"):
        _prepare_many(s, case, seed, gen)
    else:
        axes = _axes(case)
        grid = synth.Grid(*axes)
        if kind in ("solve", "host"):
            subdiv = 4 if case["ny"] < 60 else 5 if case["ny"] < 200 else 6
            body = _sphere(case, subdiv) if case["body"] else None
            s["c"], masks = _tagged(case, grid, body, stream)
            f = _rhs(case, s["c"], grid, axes, masks, gen)
            if kind == "solve":
                s["f"], s["p"] = f, torch.zeros_like(f)
            else:
                s["keep"], s["f"], s["p"] = [], None, None
                for key, t in (("f", f), ("p", torch.zeros_like(f))):
                    keep, s[key] = _pinned(t)
                    s["keep"].append(keep)
        elif kind == "plate":
            lx, ly, lz = _lengths(case)
            base = synth.plate_body(n=64, size=1.0, tkns_factor=1.0, grid_h=lz / case["nz"])
            angle = math.radians(30.0) * math.sin(2.0 * math.pi * (int(seed) % 97) / 97.0)
            s["verts"] = synth.pitch_plate(base, (0.25 * lx, 0.5 * ly, 0.5 * lz), angle)
            body = synth.Body(verts=s["verts"], tri=base.tri, surface=2, membrane_tkns=base.membrane_tkns)
            s["c"], masks = _tagged(case, grid, body, stream)
            s["f"] = _rhs(case, s["c"], grid, axes, masks, gen)
            s["p"] = torch.zeros_like(s["f"])
        elif kind == "tag":
            lx, ly, lz = _lengths(case)
            shift = (int(seed) % 7) * lx / case["nx"]  # whole cells along x: the lists keep their lengths
            body = _ball((0.25 * lx + 0.0137 + shift, 0.5 * ly + 0.0071, 0.5 * lz + 0.0043), (0.5, 0.5, 0.5),
                         np.eye(3), case["subdiv"])
            s["c"] = fg.Case(grid, _config(case))
            s["c"].set_stream(stream.cuda_stream)
            s["c"].add_body(body)
        elif kind == "project":
            s["c"], _ = _tagged(case, grid, _sphere(case, 4) if case["body"] else None, stream)
            s["u"], s["v"], s["w"] = _flow(grid, gen)
            s["pp"] = 0.1 * _smooth(grid.shape[::-1], gen)
            s["bc"] = _face_arrays(s["u"], s["v"], s["w"])
            s["out"] = [torch.zeros_like(s["u"]) for _ in range(5)]  # face velocities, div, p
            s["dt"] = _step(case)
        else:
            s["c"], _ = _tagged(case, grid, _sphere(case, 4) if case.get("body", True) else None, stream)
            s["dt"] = _step(case)
            u, v, w = _flow(grid, gen)
            s["faces"] = _flow(grid, gen)
            s["vel"] = [u, v, w]
            s["rhs"] = [u + 0.01 * _smooth(grid.shape[::-1], gen), v.clone(), w.clone()]
            if kind == "momentum":
                s["prm"] = fg.AdParams(dt=s["dt"], reinv=0.01, omega_ad=1.0,
                                       crank_nicolson=int(case["crank_nicolson"]))
            else:
                _prepare_solve_ad(s, fg, grid)
    torch.cuda.synchronize()
    return s


def _face_arrays(u, v, w):
    """Boundary face velocities of a unit stream: bcxu, bcyv, bczw."""
    nz, ny, nx = u.shape
    z = dict(dtype=torch.float64, device="cuda")
    bx, by, bz = torch.ones((nz, ny, 2), **z), torch.zeros((nz, 2, nx), **z), torch.zeros((2, ny, nx), **z)
    bx[:, :, 1] = u[:, :, -3]
    return [bx, by, bz]


def _prepare_solve_ad(s, fg, grid):
    NX, NY, NZ = grid.shape
    z = dict(dtype=torch.float64, device="cuda")
    shapes = [(NZ, NY, 2)] * 3 + [(NZ, 2, NX)] * 3 + [(2, NY, NX)] * 3
    s["bc"] = [torch.zeros(sh, **z) for sh in shapes]
    vb = fg.VelocityBC()
    for f, t in enumerate((1, 2, 4, 4, 4, 4)):  # inflow, outflow, symmetry walls
        vb.type[f] = t
    vb.val[0][0] = 1.0
    s["vb"] = vb
    c, vel = s["c"], [t.data_ptr() for t in s["vel"]]
    bc = [t.data_ptr() for t in s["bc"]]
    faces = [torch.zeros_like(s["vel"][0]) for _ in range(3)]
    fg.set_outer_velocity_bc_device(c, *vel, bc, vb)
    fg.set_outer_ghost_velocity_device(c, *vel, bc)
    fg.face_vel_device(c, *vel, bc[0], bc[4], bc[8], *[t.data_ptr() for t in faces])
    s["faces"] = faces
    s["ubi"] = [torch.zeros(max(1, 3 * n), **z) for n in (c.nGhost, c.nDead)]
    s["prm"] = fg.AdParams(dt=s["dt"], reinv=0.01, omega_ad=1.0, crank_nicolson=1)


def _prepare_many(s, case, seed, gen):
    fg, synth = _package()
    rng = np.random.default_rng(seed)
    s["p"], s["f"], s["cases"], s["grids"], s["bodies"], s["keep"] = [], [], [], [], [], []
    s["result"] = []
    steps = case.get("steps", 1)
    for edge in _edges(case):
        grid, axes = _cube(edge)
        body = _ellipsoid(rng)
        c, masks = _tagged(case, grid, body, s["stream"])
        f = [_rhs(case, c, grid, axes, masks, gen) for _ in range(steps)]
        s["grids"].append(grid)
        s["bodies"].append(body)
        if case["kind"] == "batch":
            s["cases"].append(c)
            s["f"] += f
            s["p"].append(torch.zeros_like(f[0]))
        else:
            c.close()
            fp, pp = [_pinned(t) for t in f], [_pinned(torch.zeros_like(t)) for t in f]
            s["keep"] += [t for t, _ in fp]
            s["result"].append([t for t, _ in pp])
            s["f"].append([a for _, a in fp])
            s["p"].append([a for _, a in pp])
    if case["kind"] == "batch":
        s["batch"] = fg.Batch(_config(case))
        for c in s["cases"]:
            s["batch"].add(c)
    else:
        s["server"] = fg.Server(_config(case), max_active=8)


# ------------------------------------------------------------------ run
def run(s):
    fg, kind = s["fg"], s["kind"]
    with torch.cuda.stream(s["stream"]):
        if kind == "solve":
            s["p"].zero_()
            s["c"].solve_poisson_device(s["p"].data_ptr(), s["f"].data_ptr())
            fg.update_pressure_device(s["c"], s["p"].data_ptr())
            return s["p"]
        if kind == "host":
            s["p"].fill(0.0)
            s["c"].solve_poisson(s["p"], s["f"])
            return s["keep"][1]
        if kind == "batch":
            for p in s["p"]:
                p.zero_()
            s["batch"].solve_device([p.data_ptr() for p in s["p"]], [f.data_ptr() for f in s["f"]])
            return s["p"]
        if kind == "serve":
            for n, (g, b) in enumerate(zip(s["grids"], s["bodies"])):
                s["server"].submit(n, g, b, s["f"][n], s["p"][n])
            s["server"].wait_idle()
            status = sorted((r["id"], r["status"]) for r in s["server"].poll())
            return {"p": s["result"], "status": np.array(status)}
        if kind == "plate":
            c = s["c"]
            c.update_body(0, s["verts"])
            c.set_iblank_body_fast()
            masks = c.gcm_set_internal_boundary()
            c.mg_prepare()
            s["p"].zero_()
            c.solve_poisson_device(s["p"].data_ptr(), s["f"].data_ptr())
            fg.update_pressure_device(c, s["p"].data_ptr())
            return {"p": s["p"], "masks": list(masks)}
        if kind == "tag":
            c = s["c"]
            solid = c.set_iblank_body_fast()
            masks = c.gcm_set_internal_boundary()
            return {"solid": solid, "masks": list(masks), "ghost": c.ghost_rows(), "dead": c.dead_rows()}
        if kind == "project":
            return _run_project(s)
        if kind == "momentum":
            ptr = [t.data_ptr() for t in (s["vel"][0], s["rhs"][0], *s["faces"])]
            fg.itsolv_ad_device(s["c"], *ptr, s["prm"])
            res, at = fg.calc_residual_ad_device(s["c"], *ptr, s["prm"])
            return {"u": s["vel"][0], "res": res, "at": list(at)}
        it, res, at = fg.solve_ad_device(s["c"], *[t.data_ptr() for t in (*s["vel"], *s["rhs"], *s["faces"])],
                                         [t.data_ptr() for t in s["bc"]], s["ubi"][0].data_ptr(),
                                         s["ubi"][1].data_ptr(), s["prm"], s["vb"],
                                         itermax_ad=s["case"]["iterations"], restol_ad=0.0)
        return {"vel": s["vel"], "faces": s["faces"], "bc": s["bc"], "res": res, "iterations": it}


def _run_project(s):
    """Face velocities, the Poisson right-hand side, then the correction by
    p' and the pressure update (the solve between them is timed by itself)."""
    fg, c, dt = s["fg"], s["c"], s["dt"]
    u, v, w, pp = (s[k].data_ptr() for k in ("u", "v", "w", "pp"))
    fu, fv, fw, div, p = (t.data_ptr() for t in s["out"])
    bc = [t.data_ptr() for t in s["bc"]]
    fg.face_vel_device(c, u, v, w, *bc, fu, fv, fw)
    flux, most = fg.rhs_poisson_device(c, fu, fv, fw, *bc, [0, int(s["case"]["outflow"]), 0, 0, 0, 0], dt, div)
    fg.correct_vel_device(c, pp, dt, u, v, w)
    fg.update_pressure_device(c, pp, p)
    return {"vel": [s["u"], s["v"], s["w"]], "out": s["out"], "bc": s["bc"], "most": most}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes of inputs read once and outputs written once, and the
    operations of one application of the operators involved."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        n = sum(e ** 3 for e in _edges(case)) * case.get("steps", 1)
        return {"bytes": 16.0 * n, "flops": 13.0 * n}
    n = float(case["nx"]) * case["ny"] * case["nz"]
    if kind in ("solve", "host"):
        return {"bytes": 16.0 * n, "flops": 13.0 * n}
    if kind == "plate":
        return {"bytes": 19.0 * n, "flops": 13.0 * n}
    if kind == "tag":
        return {"bytes": 4.0 * n, "flops": 4.0 * n}
    if kind == "project":  # u, v, w read and written, p' read and written, faces, div and p written, masks
        return {"bytes": (6 + 2 + 5) * 8.0 * n + 3.0 * n, "flops": 55.0 * n}
    if kind == "momentum":  # u read and written, its right-hand side, three faces, masks
        return {"bytes": 6 * 8.0 * n + 2.0 * n, "flops": 150.0 * n}
    it = case["iterations"]
    return {"bytes": it * (12 * 8.0 * n + 2.0 * n), "flops": it * 450.0 * n}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """What run() returns in 64 bits, where it follows from the inputs alone:
    solves without a body (the potential the right-hand side was made from),
    the projection steps and a momentum pass without a body.  With a body the
    result also depends on the tagged geometry."""
    kind = case["kind"]
    if case.get("body", True) or kind not in ("solve", "host", "project", "momentum"):
        return None
    gen = _generator(seed)
    axes = _axes(case)
    shape = tuple(len(a) + 2 for a in axes)

    class grid:  # the array extents alone
        nx, ny, nz = (len(a) for a in axes)

    grid.shape = shape
    if kind in ("solve", "host"):
        return _exact_solve(grid, gen, _outlet(case))
    if kind == "project":
        return _exact_project(case, grid, _device_axes(axes), gen)
    if grid.nx * grid.ny * grid.nz > 3_000_000:
        return None
    return _exact_momentum(case, grid, [_Axis(a, "cpu") for a in axes], gen)


def _exact_solve(grid, gen, outlet):
    """The potential, less its value in the first cell where no face holds
    the pressure; the x edges of the domain are zero."""
    phi = _potential(grid, gen, outlet)
    if not outlet:
        phi[:-1, :-1, :-1] -= phi[1, 1, 1].clone()
    phi[-1], phi[:, -1], phi[:, :, -1] = 0.0, 0.0, 0.0
    lines = [(k, j) for k in (0, -2) for j in (0, -2)]
    for k, j in lines:
        phi[k, j] = 0.0
    if not outlet:
        _clear_edges(phi)
    return phi


def _clear_edges(p):
    """The domain's edge lines as update_pressure clears them."""
    for k in (0, -2, -1):
        for e in (0, -2):
            p[k, e, :-1] = 0.0
            p[k, :, e] = 0.0
    for j in (0, -2):
        for i in (0, -2):
            p[:, j, i] = 0.0


def _exact_project(case, grid, axes, gen):
    X, Y, Z = axes
    u, v, w = _flow(grid, gen)
    pp = 0.1 * _smooth(grid.shape[::-1], gen)
    bx, by, bz = _face_arrays(u, v, w)
    dt = _step(case)
    dims = (2, 1, 0)
    I = slice(1, -2)

    def along(a, dim, lo, hi):
        shape = [1, 1, 1]
        shape[dim] = hi - lo
        return a[lo:hi].view(shape)

    faces = []
    for f, A, dim, bc in ((u, X, 2, bx), (v, Y, 1, by), (w, Z, 0, bz)):
        n = A.n
        out = torch.zeros_like(f)
        t = along(A.f, dim, 2, n)
        cut = [I, I, I]
        src = f[tuple(I if d != dim else slice(None) for d in range(3))]
        cut[dim] = slice(2, n)
        out[tuple(cut)] = t * src.narrow(dim, 2, n - 2) + (1.0 - t) * src.narrow(dim, 1, n - 2)
        for side, at in ((0, 1), (1, n)):
            cut[dim] = at
            edge = bc.select(dim, side)
            out[tuple(cut)] = edge[I, I]
        faces.append(out)
    fu, fv, fw = faces
    if case["outflow"]:
        vol = [along(A.d, d, 1, A.n) for A, d in zip(axes, dims)]
        flux = (((fu[I, I, 2:-1] - fu[I, I, I]) * vol[1] * vol[2]).sum() +
                ((fv[I, 2:-1, I] - fv[I, I, I]) * vol[0] * vol[2]).sum() +
                ((fw[2:-1, I, I] - fw[I, I, I]) * vol[0] * vol[1]).sum())
        fix = -flux / (vol[1] * vol[2]).sum()
        bx[:-1, :-1, 1] += fix
        fu[I, I, -2] += fix
    div = torch.zeros_like(u)
    div[I, I, I] = ((fu[I, I, 2:-1] - fu[I, I, I]) / along(X.d, 2, 1, X.n) +
                    (fv[I, 2:-1, I] - fv[I, I, I]) / along(Y.d, 1, 1, Y.n) +
                    (fw[2:-1, I, I] - fw[I, I, I]) / along(Z.d, 0, 1, Z.n)) / dt
    most = float(div.abs().max()) * dt
    for f, A, dim in ((u, X, 2), (v, Y, 1), (w, Z, 0)):
        n = A.n
        src = pp[tuple(I if d != dim else slice(None) for d in range(3))]
        c = src.narrow(dim, 1, n - 1)
        hi, lo = along(A.f, dim, 2, n + 1), along(A.f, dim, 1, n)
        g = (hi * src.narrow(dim, 2, n - 1) + (1.0 - hi) * c - lo * c - (1.0 - lo) * src.narrow(dim, 0, n - 1))
        f[I, I, I] -= dt * g / along(A.d, dim, 1, n)
    _clear_edges(pp)
    return {"vel": [u, v, w], "out": [fu, fv, fw, div, pp], "bc": [bx, by, bz], "most": most}


def _exact_momentum(case, grid, axes, gen):
    """One pass of line Gauss-Seidel sweeps in x, y, z, lines in
    lexicographic order (all lines of an anti-diagonal at once: they do not
    read one another), and the largest residual with its first place."""
    u, v, w = _flow(grid, gen)
    fu, fv, fw = (a.cpu().numpy() for a in _flow(grid, gen))
    r = (u + 0.01 * _smooth(grid.shape[::-1], gen)).cpu().numpy()
    u = u.cpu().numpy()
    dt, nu = _step(case), 0.01
    half = 0.5 * dt if case["crank_nicolson"] else 0.0
    n = (grid.nx, grid.ny, grid.nz)
    sh = u.shape
    i = np.arange(1, n[0])
    central = ((i >= 25) & (i <= 375))[None, None, :]
    I = slice(1, -2)
    lo, hi, mid = [], [], []
    for q, (A, f) in enumerate(zip(axes, (fu, fv, fw))):
        dim = 2 - q
        shape = [1, 1, 1]
        shape[dim] = n[q] - 1
        d, dc, t = A.d.numpy(), A.dc.numpy(), A.f.numpy()
        m = n[q]
        am = -(0.5 * dt * nu) / (dc[0:m - 1] * d[1:m])
        ap = -(0.5 * dt * nu) / (dc[1:m] * d[1:m])
        am, ap, dd = (a.reshape(shape) for a in (am, ap, d[1:m]))
        t0, t1 = t[1:m].reshape(shape), t[2:m + 1].reshape(shape)
        f0 = f[I, I, I]
        cut = [I, I, I]
        cut[dim] = slice(2, -1)
        f1 = f[tuple(cut)]
        up0, up1 = np.copysign(1.0, f0) > 0, np.copysign(1.0, f1) > 0
        lo.append(am - half * f0 / dd * np.where(central, 1.0 - t0, up0))
        hi.append(ap + half * f1 / dd * np.where(central, t1, ~up1))
        mid.append(-(am + ap) + half / dd * np.where(central, f1 * (1.0 - t1) - f0 * t0, f1 * up1 - f0 * ~up0))
    diag = 1.0 + mid[0] + mid[1] + mid[2]
    step = (1, sh[2], sh[1] * sh[2])
    flat = u.reshape(-1)
    rhs = r.reshape(-1)
    full = []
    for a in (*lo, *hi, diag):
        b = np.zeros(sh)
        b[I, I, I] = a
        full.append(b.reshape(-1))
    L, H, D = full[0:3], full[3:6], full[6]
    for q in range(3):
        a_, b_ = [x for x in range(3) if x != q]
        m = n[q] - 1
        for diagonal in range(2, n[a_] + n[b_] - 1):
            a = np.arange(max(1, diagonal - (n[b_] - 1)), min(n[a_] - 1, diagonal - 1) + 1)
            base = a * step[a_] + (diagonal - a) * step[b_]
            at = base[None, :] + step[q] * np.arange(1, m + 1)[:, None]
            d = rhs[at].copy()
            for o in (a_, b_):
                d -= flat[at - step[o]] * L[o][at] + flat[at + step[o]] * H[o][at]
            l, h, c = L[q][at], H[q][at], D[at]
            d[0] -= l[0] * flat[base]
            d[-1] -= h[-1] * flat[base + step[q] * (m + 1)]
            g = np.zeros_like(d)
            g[0] = h[0] / c[0]
            d[0] /= c[0]
            for s in range(1, m):
                e = 1.0 / (c[s] - l[s] * g[s - 1])
                g[s] = h[s] * e
                d[s] = (d[s] - l[s] * d[s - 1]) * e
            for s in range(m - 2, -1, -1):
                d[s] -= g[s] * d[s + 1]
            flat[at] = d
    res = r[I, I, I] - diag * u[I, I, I]
    res -= lo[0] * u[I, I, :-3] + hi[0] * u[I, I, 2:-1] + lo[1] * u[I, :-3, I] + hi[1] * u[I, 2:-1, I]
    res -= lo[2] * u[:-3, I, I] + hi[2] * u[2:-1, I, I]
    res = np.abs(res)
    k, j, i = np.unravel_index(int(np.argmax(res)), res.shape)
    return {"u": torch.from_numpy(u), "res": float(res.max()), "at": [int(i) + 1, int(j) + 1, int(k) + 1]}
