"""Measured cases: the solver's work as a simulation program calls it.

Every case goes through ``uaamg_b200.solver`` (``Handle``, ``Server``) with default
kernels and schedules.  The families:

* ``solve``    ``Handle.solve_device``: one Poisson solve, right-hand side on the device.
* ``host``     ``Handle.solve``: the drop-in with host arrays.
* ``project``  ``Handle.project_device``: divergence, solve and face correction.
* ``static``   ``Handle.static_pressure_device`` (2D).
* ``step``     a moving obstacle: ``set_problem_device`` and ``project_device``, twice.
* ``batch``    ``Handle.solve_batch`` over uneven 2D and 3D problems (host arrays).
* ``serve``    ``Server.submit`` / ``drain`` / ``poll``: several simulations, two steps
               each, the second warm-started from the first.

Fluid domains are connected by construction: solids are disks or spheres in the cells
of a lattice, never touching each other or a wall.  Right-hand sides are smoothed noise
(sigma 4 cells) and velocity fields an inflow plus smoothed noise, as in the benchmark's
workloads.  The mixed form solves to a relative residual of 1e-6, which is single
precision in the pressure: its results are taken as float32, as a single-precision
simulation stores them.  The FP64 form solves to 1e-10 and its results stay float64.
"""
import math

import numpy as np
import torch

from uaamg_b200.solver import Handle, Server


# ---------------------------------------------------------------------------
# cases


def _case(op, nx, ny, nz=0, prec="mixed", solids=0, aniso=1.0, layered=False, count=0):
    return {"op": op, "nx": nx, "ny": ny, "nz": nz, "prec": prec, "solids": solids,
            "aniso": aniso, "layered": layered, "count": count}


def listed():
    named = [
        # the standalone 64 x 64 Dirichlet Poisson problem, FP64 to 1e-10, host arrays: the
        # smallest call, launches and latency
        ("host64_fp64", _case("host", 64, 64, prec="fp64")),
        # FP64 (reference-exact) 3D pressure solve, 1e-10
        ("solve96_fp64", _case("solve", 96, 96, 96, prec="fp64", solids=8)),
        # LFM static-pressure recovery on an odd, ragged 2D grid
        ("static777x333", _case("static", 777, 333, solids=3, aniso=1.5)),
        # the serving mix's median 2D simulation, one projection step
        ("project384", _case("project", 384, 384, solids=1)),
        # 2D obstacle flow, the largest 2D grid
        ("project2048x1024", _case("project", 2048, 1024, solids=1, aniso=1.5)),
        # 2D variable-coefficient operator (layered medium)
        ("layered1024x512", _case("solve", 1024, 512, solids=1, aniso=1.5, layered=True)),
        # the serving mix's median 3D simulation
        ("solve96", _case("solve", 96, 96, 96, solids=8)),
        # odd, uneven 3D box with a spacing per axis, one projection step
        ("project129x97x65", _case("project", 129, 97, 65, solids=4, aniso=1.5)),
        # moving obstacle: the mask changes before each of two projection steps
        ("step128", _case("step", 128, 128, 128, solids=1)),
        # 256^3 with 32 spheres: the benchmark's problem
        ("solve256", _case("solve", 256, 256, 256, solids=32)),
        # uneven 2D and 3D problems solved together
        ("batch24", _case("batch", 512, 512, 96, solids=4, count=24)),
        # requests of eight simulations, two steps each, on one server
        ("serve8", _case("serve", 384, 384, 96, solids=1, count=8)),
    ]
    return [dict(c, name=n) for n, c in named]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    r = rng.random()
    aniso = rng.choice([1.0, 1.25, 1.5])
    fp64 = rng.random() < 0.15
    if r < 0.35:  # 2D, one call
        hi = 512 if fp64 else 2048
        nx, ny = _log_size(rng, 64, hi), _log_size(rng, 64, hi // 2)
        op = rng.choice(["solve", "project", "static", "host"])
        return _case(op, nx, ny, prec="fp64" if fp64 else "mixed", solids=rng.choice([1, 2, 4]),
                     aniso=aniso, layered=op == "solve" and not fp64 and rng.random() < 0.5)
    if r < 0.75:  # 3D, one call
        hi = 96 if fp64 else 224
        n = [_log_size(rng, 32, hi) for _ in range(3)]
        return _case(rng.choice(["solve", "project", "host"]), *n, prec="fp64" if fp64 else "mixed",
                     solids=rng.choice([1, 4, 8]), aniso=aniso)
    if r < 0.87:  # moving obstacle, 2D or 3D
        if rng.random() < 0.5:
            return _case("step", _log_size(rng, 64, 1024), _log_size(rng, 64, 512), solids=1, aniso=aniso)
        return _case("step", *[_log_size(rng, 32, 160) for _ in range(3)], solids=1, aniso=aniso)
    if r < 0.94:
        return _case("batch", _log_size(rng, 128, 512), _log_size(rng, 128, 512), _log_size(rng, 32, 96),
                     solids=rng.choice([1, 4]), count=rng.randint(6, 24))
    return _case("serve", _log_size(rng, 128, 384), _log_size(rng, 128, 384), _log_size(rng, 32, 96),
                 solids=1, count=rng.randint(3, 8))


# ---------------------------------------------------------------------------
# problems (padded arrays, i fastest: shape (ny+2, nx+2) or (nz+2, ny+2, nx+2))


class _Gen:
    """Seeded fields on the GPU."""

    def __init__(self, seed):
        self.t = torch.Generator(device="cuda").manual_seed(int(seed))
        self.r = np.random.Generator(np.random.PCG64(int(seed)))

    def noise(self, shape, sigma=4.0):
        """N(0,1) noise blurred with a periodic Gaussian, unit variance."""
        a = torch.randn(shape, generator=self.t, device="cuda", dtype=torch.float64)
        f = torch.fft.rfftn(a)
        for ax, n in enumerate(shape):
            k = torch.fft.rfftfreq(n, device="cuda") if ax == len(shape) - 1 else torch.fft.fftfreq(n, device="cuda")
            w = torch.exp(-2.0 * (math.pi * sigma * k.double()) ** 2)
            f = f * w.reshape([-1 if q == ax else 1 for q in range(len(shape))])
        a = torch.fft.irfftn(f, s=shape)
        return a / a.std()

    def mask(self, dims, count, moved=0.0):
        """Padded byte mask of `count` disks or spheres in lattice cells, none touching
        another or a wall; dims = (nx, ny[, nz]); moved: shift along x in cells."""
        s = torch.zeros([n + 2 for n in reversed(dims)], dtype=torch.uint8, device="cuda")
        m = [1] * len(dims)
        while math.prod(m) < count:
            a = max(range(len(dims)), key=lambda q: dims[q] / m[q])
            m[a] += 1
        cell = [n / q for n, q in zip(dims, m)]
        for c in self.r.permutation(math.prod(m))[:count]:
            rad = float(self.r.uniform(0.12, 0.36)) * min(cell)
            at = []
            for n, q in zip(cell, m):
                play = max(0.0, n / 2 - rad - 3.0)
                at.append((c % q + 0.5) * n + float(self.r.uniform(-play, play)))
                c //= q
            at[0] += moved
            d2 = 0.0
            for ax, n in enumerate(dims):
                x = torch.arange(n + 2, device="cuda", dtype=torch.float64) - 0.5 - at[ax]
                d2 = d2 + (x * x).reshape([-1 if len(dims) - 1 - q == ax else 1 for q in range(len(dims))])
            s[d2 < rad * rad] = 1
        for ax in range(len(dims)):  # ghost cells stay fluid in the mask: walls are implied
            s.narrow(ax, 0, 1).zero_()
            s.narrow(ax, s.shape[ax] - 1, 1).zero_()
        return s.contiguous()

    def rhs(self, solid):
        """Smoothed noise, zero in solids, zero fluid mean, in padded layout."""
        b = torch.zeros(solid.shape, dtype=torch.float64, device="cuda")
        core = tuple(slice(1, -1) for _ in solid.shape)
        fluid = solid[core] == 0
        a = self.noise(fluid.shape) * fluid
        b[core] = (a - a.sum() / fluid.sum()) * fluid
        return b

    def faces(self, dims):
        """Face velocities u, v[, w]: an inflow of 1 along x plus smoothed noise."""
        out = []
        for ax in range(len(dims)):
            shape = [n + 1 if q == ax else n + 2 for q, n in enumerate(dims)][::-1]
            out.append((0.1 * self.noise(shape) + (1.0 if ax == 0 else 0.0)).contiguous())
        return out


def _dims(c):
    return (c["nx"], c["ny"], c["nz"]) if c["nz"] else (c["nx"], c["ny"])


def _spacing(c, dims):
    h = 1.0 / max(dims)
    return (h, h * c["aniso"], h if len(dims) == 2 else h / c["aniso"])


def _layered(solid, dx, dy):
    """Variable coefficients of a layered medium (x conductivity 1 + 0.5 sin(2 pi y), y
    conductivity 1 + 0.5 cos(2 pi x)): symmetric, zero row sums."""
    ny, nx = (n - 2 for n in solid.shape)
    y = (torch.arange(ny + 2, device="cuda", dtype=torch.float64) - 0.5) / ny
    x = (torch.arange(nx + 2, device="cuda", dtype=torch.float64) - 0.5) / nx
    ox = (-(1 + 0.5 * torch.sin(2 * math.pi * y))[:, None] / (dx * dx)).expand(solid.shape)
    oy = (-(1 + 0.5 * torch.cos(2 * math.pi * x))[None, :] / (dy * dy)).expand(solid.shape)
    return [a.contiguous() for a in (-2 * ox - 2 * oy, ox, oy)]


def _members(c):
    """(dims, ...) of the problems of a batch or the simulations of a server: two of three
    2D, sizes from an eighth (not under 48; 3D not under 24) to the whole of nx, ny, nz."""
    r = np.random.Generator(np.random.PCG64(c["count"] * 1000003 + c["nx"] * 1009 + c["nz"]))
    out = []
    for q in range(c["count"]):
        if q % 3 != 2:
            lo = max(48, min(c["nx"], c["ny"]) // 8)
            out.append(tuple(int(round(math.exp(r.uniform(math.log(lo), math.log(n))))) for n in (c["nx"], c["ny"])))
        else:
            lo = max(24, c["nz"] // 3)
            out.append(tuple(int(round(math.exp(r.uniform(math.log(lo), math.log(c["nz"]))))) for _ in range(3)))
    return out


def _options(c):
    if c["prec"] == "fp64":
        return Handle.options("fp64", 1e-10, 500, "rel")
    return Handle.options("mixed", 1e-6, 500, "rel")


def _problem(c, seed):
    """What a case's inputs are, on the GPU: masks, right-hand sides or velocities."""
    g = _Gen(seed)
    op, dims = c["op"], _dims(c)
    P = {"dims": dims, "h": _spacing(c, dims)}
    if op in ("batch", "serve"):
        P["members"] = []
        for d in _members(c):
            s = g.mask(d, c["solids"])
            b = [g.rhs(s)]
            if op == "serve":  # the next step's right-hand side
                b.append(b[0] + 0.05 * g.rhs(s))
            P["members"].append((d, (1.0 / max(d),) * 3, s, b))
        return P
    P["solid"] = [g.mask(dims, c["solids"])]
    if op == "step":  # the same obstacle, one cell further along x
        g2 = _Gen(seed)
        P["solid"].append(g2.mask(dims, c["solids"], moved=1.0))
    if op in ("solve", "host"):
        P["rhs"] = g.rhs(P["solid"][0])
    else:
        P["vel"] = g.faces(dims)
    P["lap"] = _layered(P["solid"][0], *P["h"][:2]) if c["layered"] else None
    return P


DT = 1e-3


def prepare(case, seed):
    c = dict(case)
    P = _problem(c, seed)
    op, dims, h = c["op"], P["dims"], P["h"]
    S = {"case": c, "dims": dims, "h": h, "opts": _options(c)}
    if op == "serve":
        S["srv"] = Server(0, "mixed", 1e-6, 500, max_active=8)
        S["sims"] = [(q, s.cpu().numpy(), [x.cpu().numpy() for x in b], hh, np.zeros(s.shape), np.zeros(s.shape))
                     for q, (_, hh, s, b) in enumerate(P["members"])]
        return S
    S["h_"] = hd = Handle(0)
    if op == "batch":
        S["probs"] = [(s.cpu().numpy(), b[0].cpu().numpy(), np.zeros(s.shape), *hh) for _, hh, s, b in P["members"]]
        return S
    solid = P["solid"][0]
    if op == "host":
        hd.set_dirichlet_walls(not c["solids"])
        hd.set_problem(solid.cpu().numpy(), *h)
        S["rhs"] = P["rhs"].cpu().numpy()
        S["p"] = np.zeros(solid.shape)
        return S
    S["solid"] = P["solid"]
    S["p"] = [torch.zeros(solid.shape, dtype=torch.float64, device="cuda") for _ in P["solid"]]
    S["shape"] = (len(dims), dims[0], dims[1], dims[2] if len(dims) == 3 else 0, *h)
    if op == "solve":
        S["rhs"] = P["rhs"]
    else:
        S["vel"] = P["vel"]
        S["work"] = [[torch.empty_like(a) for a in P["vel"]] for _ in P["solid"]]
    torch.cuda.synchronize()
    if op != "step":
        hd.set_problem_device(*S["shape"], solid.data_ptr())
        if P["lap"] is not None:
            hd.set_variable_laplacian(*[a.cpu().numpy() for a in P["lap"]])
    return S


def _result(c, a):
    """A simulation's own array of a result: single precision from the mixed form."""
    if c["prec"] == "fp64":
        return a
    return a.astype(np.float32) if isinstance(a, np.ndarray) else a.float()


def run(S):
    c = S["case"]
    op = c["op"]
    if op == "serve":
        srv, open_ = S["srv"], []
        for step in (0, 1):
            for q, s, b, h, *p in S["sims"]:
                open_.append(srv.submit(q, s, b[step], *h, p_out=p[step]))
        srv.drain()
        for t in open_:
            srv.poll(t)
        return [_result(c, p) for sim in S["sims"] for p in sim[4:]]
    hd, o = S["h_"], S["opts"]
    if op == "batch":
        for q in S["probs"]:
            q[2].fill(0.0)
        hd.solve_batch(S["probs"], o)
        return [_result(c, q[2]) for q in S["probs"]]
    if op == "host":
        S["p"].fill(0.0)
        hd.solve(S["rhs"], S["p"], o)
        return _result(c, S["p"])
    if op == "solve":
        p = S["p"][0]
        p.zero_()
        hd.solve_device(S["rhs"].data_ptr(), p.data_ptr(), o)
        return _result(c, p)
    if op == "static":
        u, v = S["vel"]
        hd.static_pressure_device(u.data_ptr(), v.data_ptr(), S["p"][0].data_ptr(), o)
        return _result(c, S["p"][0])
    out = []
    for solid, p, vel in zip(S["solid"], S["p"], S["work"]):
        for a, b in zip(vel, S["vel"]):  # the advected velocities of this step
            a.copy_(b)
        if op == "step":
            hd.set_problem_device(*S["shape"], solid.data_ptr())
        ptr = [a.data_ptr() for a in vel] + ([0] if len(vel) == 2 else [])
        hd.project_device(*ptr, p.data_ptr(), DT, o)
        out.append([_result(c, a) for a in (p, *vel)])
    return out


# ---------------------------------------------------------------------------
# the work a pass cannot do without, and its exact results


def work(case):
    """Each input read once and each output written once (right-hand side or velocities,
    mask, pressure); the operations of a multigrid-preconditioned solve counted as forty
    applications of the operator's order (12 a cell in 2D, 16 in 3D)."""
    c = dict(case)
    dims = [_dims(c)] if c["op"] not in ("batch", "serve") else _members(c)
    passes = 2 if c["op"] in ("serve", "step") else 1
    by = fl = 0.0
    for d in dims:
        n = float(math.prod(d))
        per = 8 + 1 + 8  # right-hand side, mask, pressure
        if c["op"] in ("project", "step"):
            per = 16 * len(d) + 1 + 8  # velocities in and out, mask, pressure
        elif c["op"] == "static":
            per = 8 * len(d) + 1 + 8
        if c["layered"]:
            per += 24
        by += passes * n * per
        fl += passes * n * 40 * (12 if len(d) == 2 else 16)
    return {"bytes": by, "flops": fl}


def _neighbours(solid, h, dirichlet):
    """Per axis (towards + of that array axis): coupling where both cells are fluid
    interior cells; the walls' diagonal with Dirichlet walls."""
    core = solid[tuple(slice(1, -1) for _ in solid.shape)] == 0
    nd = core.dim()
    coup, wall = [], torch.zeros(core.shape, dtype=torch.float64, device=core.device)
    for ax in range(nd):  # array axis ax is coordinate nd-1-ax
        w = 1.0 / h[nd - 1 - ax] ** 2
        both = core.narrow(ax, 0, core.shape[ax] - 1) & core.narrow(ax, 1, core.shape[ax] - 1)
        coup.append(both.double() * w)
        if dirichlet:
            wall.narrow(ax, 0, 1).add_(2 * w)
            wall.narrow(ax, core.shape[ax] - 1, 1).add_(2 * w)
    return core.double(), coup, wall


def _solve_exact(solid, b, h, dirichlet=False, lap=None):
    """lap(p) = b on the fluid cells in 64 bits: conjugate gradients in plain torch to a
    residual of 1e-13; with Neumann walls b loses its fluid mean and so does p."""
    fluid, coup, wall = _neighbours(solid, h, dirichlet)
    core = tuple(slice(1, -1) for _ in solid.shape)
    nd = fluid.dim()
    if lap is not None:  # A p = d p_C + ox (p_L + p_R) + oy (...), a missing neighbour reads p_C
        coup = []
        for ax, off in ((0, lap[2][core]), (1, lap[1][core])):
            n = fluid.shape[ax]
            coup.append(-off.narrow(ax, 0, n - 1) * fluid.narrow(ax, 0, n - 1) * fluid.narrow(ax, 1, n - 1))
    r = -b[core] * fluid
    if not dirichlet:
        r = (r - r.sum() / fluid.sum()) * fluid
    d = wall * fluid
    for ax, w in enumerate(coup):
        d.narrow(ax, 0, d.shape[ax] - 1).add_(w)
        d.narrow(ax, 1, d.shape[ax] - 1).add_(w)
    inv = torch.where(d > 0, 1.0 / torch.where(d > 0, d, 1.0), 0.0)

    def apply(p):
        a = d * p
        for ax, w in enumerate(coup):
            n = p.shape[ax]
            a.narrow(ax, 0, n - 1).sub_(w * p.narrow(ax, 1, n - 1))
            a.narrow(ax, 1, n - 1).sub_(w * p.narrow(ax, 0, n - 1))
        return a

    x, z = torch.zeros_like(r), inv * r
    p, rz, stop = z.clone(), (r * z).sum(), 1e-13 * float(r.norm())
    if stop == 0.0:
        return torch.zeros_like(b)
    for it in range(60000):
        a = apply(p)
        al = rz / (p * a).sum()
        x += al * p
        r -= al * a
        if it % 64 == 63 and float(r.norm()) < stop:
            break
        z = inv * r
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    if not dirichlet:
        x = (x - x.sum() / fluid.sum()) * fluid
    out = torch.zeros_like(b)
    out[core] = x
    return out


def _divergence(vel, solid, h):
    nd = solid.dim()
    inner = slice(1, -1)
    div = 0.0
    for ax, a in enumerate(vel):  # velocity ax lives on array axis nd-1-ax
        at = nd - 1 - ax
        hi = tuple(slice(1, None) if q == at else inner for q in range(nd))
        lo = tuple(slice(None, -1) if q == at else inner for q in range(nd))
        div = div + (a[hi] - a[lo]) / h[ax]
    return div


def _static_rhs(u, v, solid, h):
    """Right-hand side of the static-pressure recovery (pressure.cpp:35-66): cross
    derivatives from cell-centre velocities, clamped at the walls and dropped next to
    solids."""
    dx, dy = h[0], h[1]
    ui, vi = u[1:-1], v[:, 1:-1]
    dudx = (ui[:, 1:] - ui[:, :-1]) / dx
    dvdy = (vi[1:] - vi[:-1]) / dy
    uc, vc = 0.5 * (ui[:, 1:] + ui[:, :-1]), 0.5 * (vi[1:] + vi[:-1])
    up = torch.cat([uc[:1], uc, uc[-1:]], 0)
    vp = torch.cat([vc[:, :1], vc, vc[:, -1:]], 1)
    dudy = (up[2:] - up[:-2]) / (2 * dy) * ((solid[2:, 1:-1] == 0) & (solid[:-2, 1:-1] == 0))
    dvdx = (vp[:, 2:] - vp[:, :-2]) / (2 * dx) * ((solid[1:-1, 2:] == 0) & (solid[1:-1, :-2] == 0))
    b = torch.zeros(solid.shape, dtype=torch.float64, device="cuda")
    b[1:-1, 1:-1] = -(dudx * dudx + 2.0 * dudy * dvdx + dvdy * dvdy) * (solid[1:-1, 1:-1] == 0)
    return b


def exact(case, seed):
    c = dict(case)
    P = _problem(c, seed)
    if c["op"] == "static":
        return _solve_exact(P["solid"][0], _static_rhs(*P["vel"], P["solid"][0], P["h"]), P["h"])
    core = tuple(slice(1, -1) for _ in P["dims"])
    if c["op"] == "batch":
        return [_solve_exact(s, b[0], h) for _, h, s, b in P["members"]]
    if c["op"] == "serve":
        return [_solve_exact(s, x, h) for _, h, s, b in P["members"] for x in b]
    if c["op"] in ("solve", "host"):
        p = _solve_exact(P["solid"][0], P["rhs"], P["h"], c["op"] == "host" and not c["solids"], P["lap"])
        return p
    out = []
    for solid in P["solid"]:
        b = torch.zeros(solid.shape, dtype=torch.float64, device="cuda")
        b[core] = _divergence(P["vel"], solid, P["h"]) / DT * (solid[core] == 0)
        p = _solve_exact(solid, b, P["h"])
        vel = [a.clone() for a in P["vel"]]
        nd = solid.dim()
        for ax, a in enumerate(vel):  # faces between two fluid cells
            at = nd - 1 - ax
            lo = tuple(slice(1, -2) if q == at else slice(1, -1) for q in range(nd))
            hi = tuple(slice(2, -1) if q == at else slice(1, -1) for q in range(nd))
            f = tuple(slice(1, -1) for q in range(nd))
            ok = (solid[lo] == 0) & (solid[hi] == 0)
            a[f] -= DT * (p[hi] - p[lo]) / P["h"][ax] * ok
        out.append([p, *vel])
    return out
