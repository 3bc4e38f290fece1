"""The work that programs have this library do, as timed cases.

A program sets planets up (grid, fluid, particles, faces), gives them a state
and steps them: CFL time step, particle advection, fluid step, fade, deposit,
planet by planet or as a batch, and from time to time encodes the faces to
8-bit images.  The cases are that step at the sizes of the repository's
configurations (64 / 256 / 512 cells an edge) and at a ragged one, the start
from a velocity field, single stages that programs call by themselves, the
batched step, the output and the discrete operators.  Everything goes through
the public C entry points by the package's ctypes binding.

``exact`` evaluates the same formulas in FP64 with torch from the prepared
state (grid tables, fields and particles as the program holds them); the
Poisson solve there is a Jacobi-preconditioned CG run to a relative residual
of 1e-11.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gaseous-gusty-ball_b200"))

import ggb_api as G  # noqa: E402
import ggb_inputs  # noqa: E402

_api = None


def api():
    global _api
    if _api is None:
        _api = G.Api(G.PRODUCT_LIB)
    return _api


# ------------------------------------------------------------------ the cases

_STEP = dict(kind="step", tol=1e-4, forcing=0.0, rotation=0.0, bfecc=1, multigrid=1, mixed=0, radius=1.0)


def listed():
    return [
        # the smallest calls: the operators on a coarse grid, as a diagnostic run every step has them
        dict(name="operators-n32", kind="operators", N=32),
        # the repository's small workload: 100k particles, 256 x 256 faces, the default tolerance
        dict(_STEP, name="step-n64", N=64, particles=100_000, R=256),
        # a grid size and a face size as users round them (two coarsenings only, ragged tiles), with forcing
        dict(_STEP, name="step-n100", N=100, particles=150_000, R=500, forcing=0.5, rotation=3.0),
        # the repository's default workload: 1M particles, 1024 x 1024 faces
        dict(_STEP, name="step-n256", N=256, particles=1_000_000, R=1024, tol=1e-6),
        # the large workload with the mixed-precision solve
        dict(_STEP, name="step-n512-mixed", N=512, particles=4_000_000, R=2048, tol=1e-6, forcing=0.5, rotation=10.0,
             mixed=1),
        # the flow alone (no particles): rotating, forced, without BFECC
        dict(kind="fluid", name="fluid-n192", N=192, tol=1e-6, forcing=1.0, rotation=20.0, bfecc=0, multigrid=1,
             mixed=0),
        # a start from a velocity field: curl, mean removal, cold solve, velocity
        dict(kind="start", name="start-n128", N=128, tol=1e-6, multigrid=1, mixed=0),
        # tracer advection by itself
        dict(kind="advect", name="advect-1m", N=256, particles=1_000_000),
        # trails with a wide splat on ragged faces
        dict(kind="deposit", name="deposit-wide", particles=200_000, R=600, radius=2.5, arc=0.012),
        # uneven planets advanced together, mixed-precision solves
        dict(kind="batch", name="batch-10", planets=10, tol=1e-6, mixed=1),
        # an output step: faces, net and preview to host memory
        dict(kind="output", name="output-1024", R=1024, bg=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid_size(rng, most):
    """An edge that coarsens to between 5 and 27 cells (odd multiples of powers of two, odd sizes too)."""
    while True:
        n = rng.randint(5, 27) << rng.randint(0, 5)
        if 12 <= n <= most:
            return n


def draw(rng):
    kind = rng.choice(["step", "step", "step", "fluid", "start", "advect", "deposit", "batch", "output", "operators"])
    tol = rng.choice([1e-4, 1e-6])
    if kind == "step":
        n = _grid_size(rng, 400)
        return dict(_STEP, N=n, particles=_log(rng, 10_000, 2_000_000), R=_log(rng, 100, 1400), tol=tol,
                    forcing=rng.choice([0.0, 0.5]), rotation=rng.choice([0.0, 3.0, 10.0]), bfecc=rng.choice([1, 1, 0]),
                    mixed=rng.choice([0, 0, 1]), radius=rng.choice([1.0, 1.0, 1.5]))
    if kind == "fluid":
        return dict(kind=kind, N=_grid_size(rng, 512), tol=tol, forcing=rng.choice([0.0, 1.0]),
                    rotation=rng.choice([0.0, 20.0]), bfecc=rng.choice([0, 1]), multigrid=1,
                    mixed=rng.choice([0, 1]))
    if kind == "start":
        return dict(kind=kind, N=_grid_size(rng, 400), tol=tol, multigrid=1, mixed=rng.choice([0, 1]))
    if kind == "advect":
        return dict(kind=kind, N=_grid_size(rng, 512), particles=_log(rng, 20_000, 4_000_000))
    if kind == "deposit":
        return dict(kind=kind, particles=_log(rng, 10_000, 600_000), R=_log(rng, 100, 1500),
                    radius=rng.choice([0.75, 1.0, 1.5, 2.5, 3.0]), arc=rng.choice([0.002, 0.005, 0.012]))
    if kind == "batch":
        return dict(kind=kind, planets=rng.randint(2, 12), tol=tol, mixed=rng.choice([0, 1]))
    if kind == "output":
        return dict(kind=kind, R=_log(rng, 100, 2048), bg=rng.choice([0, 1]))
    return dict(kind=kind, N=_grid_size(rng, 512))


# ------------------------------------------------------------ objects and views


class Owner:
    """The library objects of a state, released with the last view of them."""

    def __init__(self):
        self.parts = []
        self.batch = None

    def add(self, part):
        self.parts.append(part)
        return part

    def __del__(self):
        try:
            if self.batch:
                api().lib.ggb_batch_free(self.batch)
            for p in reversed(self.parts):
                p.free()
        except Exception:  # the interpreter is ending
            pass


class _View:
    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=kind, data=(ptr, False), version=3)


def view(owner, ptr, shape, kind="<f4"):
    """A CUDA tensor over a public array (managed memory, updated by the library in place)."""
    return torch.as_tensor(_View(owner, C.cast(ptr, C.c_void_p).value, shape, kind), device="cuda")


def _ptr(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_float))


def _velocity(grid, seed):
    """The application driver's initial velocity: bands plus curl noise of this seed."""
    s = ggb_inputs.SMALL
    ip = G.InitParams(s["bands"], s["band_amp"], s["noise_amp"], s["noise_scale"], s["noise_lacunarity"],
                      s["noise_gain"], s["noise_octaves"], 1 + seed % 100_000)
    vel = torch.zeros(3 * grid.n, device="cuda")
    band = torch.zeros(3 * grid.n, device="cuda")
    torch.cuda.synchronize()
    api().lib.ggb_initial_velocity(C.byref(grid.cs), C.byref(ip), _ptr(vel), _ptr(band))
    return vel, band


def _fluid(own, c, seed, grid=None):
    grid = grid or own.add(api().grid(c["N"]))
    fs = own.add(G.FluidSim(api(), grid, forcing=c.get("forcing", 0.0), rotation=c.get("rotation", 0.0),
                            bfecc=c.get("bfecc", 1), cg_tol=c["tol"], multigrid=c["multigrid"],
                            mixed=bool(c["mixed"])))
    vel, band = _velocity(grid, seed)
    api().lib.fluid_set_state(C.byref(fs.F), _ptr(vel), _ptr(band))
    return grid, fs, vel, band


def _particles(own, n, seed):
    ps = own.add(G.ParticleSet(api(), n))
    ps.colour(ggb_inputs.strip(seed % 1000))
    return ps


def _fluid_views(own, grid, fs):
    n = grid.n
    return dict(omega=view(own, fs.F.omega, (n,)), psi=view(own, fs.F.psi, (n,)), vel=view(own, fs.F.vel, (n, 3)))


def _planet_views(own, grid, fs, ps, sp):
    R = sp.r.R
    return dict(_fluid_views(own, grid, fs), pos=view(own, ps.P.pos, (ps.P.n, 3)),
                faces=view(own, sp.r.buf, (6, R, R, 4)))


def _batch_planets(c):
    rng = np.random.default_rng(7)  # the planets' sizes are the case's, their states the seed's
    sizes = [64, 128, 256, 64, 128, 64, 128, 64, 256, 64, 128, 64][: c["planets"]]
    return [dict(_STEP, N=n, particles=int(rng.integers(100_000, 400_001)), R=512, tol=c["tol"], mixed=c["mixed"],
                 rotation=float(rng.choice([0.0, 5.0])), forcing=float(rng.choice([0.0, 0.5]))) for n in sizes]


CFL, FADE = 1.0, 0.02


def prepare(case, seed):
    c, own, kind = case, Owner(), case["kind"]
    st = dict(c=c, own=own, kind=kind, lib=api().lib)
    if kind in ("step", "fluid"):
        grid, fs, _, _ = _fluid(own, c, seed)
        st.update(grid=grid, fs=fs, h=grid.cs.h)
        if kind == "step":
            ps, sp = _particles(own, c["particles"], seed), own.add(G.Splat(api(), c["R"], c["radius"]))
            st.update(ps=ps, sp=sp, out=_planet_views(own, grid, fs, ps, sp))
        else:
            st["out"] = _fluid_views(own, grid, fs)
    elif kind == "start":
        grid, fs, vel, band = _fluid(own, c, seed)
        st.update(grid=grid, fs=fs, vel=vel, band=band, out=dict(_fluid_views(own, grid, fs),
                                                                 omega_band=view(own, fs.F.omega_band, (grid.n,))))
    elif kind == "advect":
        grid = own.add(api().grid(c["N"]))
        vel, _ = _velocity(grid, seed)
        ps = own.add(G.ParticleSet(api(), c["particles"]))
        dt = CFL * grid.cs.h / float(vel.view(-1, 3).norm(dim=1).max())
        st.update(grid=grid, ps=ps, vel=vel, dt=dt, out=dict(pos=view(own, ps.P.pos, (c["particles"], 3)),
                                                             prev=view(own, ps.P.prev, (c["particles"], 3))))
    elif kind == "deposit":
        ps, sp = _particles(own, c["particles"], seed), own.add(G.Splat(api(), c["R"], c["radius"]))
        g = torch.Generator("cuda").manual_seed(seed)
        a = torch.nn.functional.normalize(torch.randn(c["particles"], 3, generator=g, device="cuda"), dim=1)
        t = torch.randn(c["particles"], 3, generator=g, device="cuda")
        t = torch.nn.functional.normalize(t - a * (t * a).sum(1, keepdim=True), dim=1)
        th = c["arc"] * torch.rand(c["particles"], 1, generator=g, device="cuda")
        view(own, ps.P.prev, (c["particles"], 3)).copy_(a)
        view(own, ps.P.pos, (c["particles"], 3)).copy_(a * th.cos() + t * th.sin())
        st.update(ps=ps, sp=sp, out=dict(faces=view(own, sp.r.buf, (6, c["R"], c["R"], 4))))
    elif kind == "batch":
        grids, planets = {}, []
        for k, p in enumerate(_batch_planets(c)):
            if p["N"] not in grids:
                grids[p["N"]] = own.add(api().grid(p["N"]))
            grid, fs, _, _ = _fluid(own, p, seed + k, grids[p["N"]])
            planets.append((p, grid, fs, _particles(own, p["particles"], seed + k),
                            own.add(G.Splat(api(), p["R"], p["radius"]))))
        n, T = len(planets), api().T
        arrays = [(C.POINTER(T[t]) * n)(*[C.pointer(o) for o in objs]) for t, objs in (
            ("Fluid", [p[2].F for p in planets]), ("Particles", [p[3].P for p in planets]),
            ("Render", [p[4].r for p in planets]))]
        own.batch = api().lib.ggb_batch_create(n, *arrays, (C.c_double * n)(*[CFL] * n), (C.c_double * n)(*[FADE] * n))
        st.update(planets=planets, out=[_planet_views(own, *p[1:]) for p in planets])
    elif kind == "output":
        R = c["R"]
        sp = own.add(G.Splat(api(), R))
        g = torch.Generator("cuda").manual_seed(seed)
        a = torch.rand(6, R, R, 1, generator=g, device="cuda")
        view(own, sp.r.buf, (6, R, R, 4)).copy_(torch.cat([a * torch.rand(6, R, R, 3, generator=g, device="cuda"), a], 3))
        ch = 3 if c["bg"] else 4
        out = dict(faces=torch.empty(6, R, R, ch, dtype=torch.uint8, pin_memory=True),
                   net=torch.empty(3 * R, 4 * R, 4, dtype=torch.uint8, pin_memory=True),
                   preview=torch.empty(R, 2 * R, ch, dtype=torch.uint8, pin_memory=True))
        st.update(sp=sp, bg=(C.c_float * 3)(0.1, 0.2, 0.3) if c["bg"] else None, out=out,
                  to={k: C.cast(C.c_void_p(v.data_ptr()), C.POINTER(C.c_ubyte)) for k, v in out.items()})
    elif kind == "operators":
        grid = own.add(api().grid(c["N"]))
        vel, _ = _velocity(grid, seed)
        out = {k: torch.zeros(grid.n, device="cuda") for k in ("curl", "div", "lap")}
        st.update(grid=grid, vel=vel, out=out)
    torch.cuda.synchronize()
    return st


def run(st):
    kind, lib = st["kind"], st["lib"]
    if kind == "step":  # the application driver's loop body
        F, ps, sp = st["fs"].F, st["ps"].P, st["sp"].r
        dt = CFL * st["h"] / max(lib.fluid_max_speed(C.byref(F)), 1e-6)
        lib.particles_advect(C.byref(ps), C.byref(st["grid"].cs), F.vel, dt)
        lib.fluid_step(C.byref(F), dt)
        lib.render_fade(C.byref(sp), FADE)
        lib.render_deposit(C.byref(sp), C.byref(ps))
        return st["out"]
    if kind == "fluid":
        F = st["fs"].F
        lib.fluid_step(C.byref(F), CFL * st["h"] / max(lib.fluid_max_speed(C.byref(F)), 1e-6))
        return st["out"]
    if kind == "start":
        lib.fluid_set_state(C.byref(st["fs"].F), _ptr(st["vel"]), _ptr(st["band"]))
        return st["out"]
    if kind == "advect":
        lib.particles_advect(C.byref(st["ps"].P), C.byref(st["grid"].cs), _ptr(st["vel"]), st["dt"])
        return st["out"]
    if kind == "deposit":
        lib.render_fade(C.byref(st["sp"].r), FADE)
        lib.render_deposit(C.byref(st["sp"].r), C.byref(st["ps"].P))
        return st["out"]
    if kind == "batch":
        lib.ggb_batch_step(st["own"].batch, 1)
        return st["out"]
    if kind == "output":
        r, to = C.byref(st["sp"].r), st["to"]
        lib.ggb_encode_faces(r, st["bg"], None, to["faces"])
        lib.ggb_encode_net(r, st["bg"], to["net"])
        lib.ggb_encode_preview(r, st["bg"], to["preview"])
        return st["out"]
    cs, out = C.byref(st["grid"].cs), st["out"]  # operators
    lib.fluid_curl(cs, _ptr(st["vel"]), _ptr(out["curl"]))
    lib.fluid_divergence(cs, _ptr(st["vel"]), _ptr(out["div"]))
    lib.fluid_laplacian(cs, _ptr(out["curl"]), _ptr(out["lap"]))
    return out


# ------------------------------------------------------------------ the least work


def _fluid_work(N, tol, cold=False):
    """Bytes: tables of the operators, geometry and fields once.  Operations: the CG iterations (about 5 at a
    tolerance of 1e-4, 8 at 1e-6, twice that from a cold start), each three level-0 stencils and the V-cycle below."""
    n, its = 6 * N * N, (5 if tol > 1e-5 else 8) * (2 if cold else 1)
    return n * (16 + 128 + 17 + 52), n * (its * 4 / 3 * 3 * 30 + 800)


def _splat_work(n, R, arc, radius):
    samples = n * max(1.0, arc * R / 0.7)
    return n * (12 + 12 + 16) + 32 * min(6 * R * R, samples * 4), samples * (90 + 10 * (2 * radius) ** 2)


def work(case):
    c, kind = case, case["kind"]
    if kind == "operators":
        n = 6 * c["N"] ** 2
        return dict(bytes=n * (12 + 12 + 1 + 32 + 32 + 4 + 16 + 12), flops=n * 6 * 60)
    if kind in ("fluid", "start"):
        b, f = _fluid_work(c["N"], c["tol"], kind == "start")
        return dict(bytes=b, flops=f)
    if kind == "advect":
        return dict(bytes=c["particles"] * 36 + 72 * c["N"] ** 2, flops=c["particles"] * 400)
    if kind == "deposit":
        b, f = _splat_work(c["particles"], c["R"], 0.5 * c["arc"], c["radius"])
        return dict(bytes=b, flops=f)
    if kind == "output":
        return dict(bytes=c["R"] ** 2 * (6 * 16 + (6 + 2) * (3 if c["bg"] else 4) + 48), flops=c["R"] ** 2 * 600)
    total = [0.0, 0.0]
    for p in [c] if kind == "step" else _batch_planets(c):
        for b, f in (_fluid_work(p["N"], p["tol"]), (36 * p["particles"], 400 * p["particles"]),
                     _splat_work(p["particles"], p["R"], 0.4 * math.pi / 2 / p["N"], p["radius"])):
            total[0] += b
            total[1] += f
    return dict(bytes=total[0], flops=total[1])


# ------------------------------------------------- the same formulas in 64 bits


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _tangent(v, p):
    return v - p * _dot(v, p)


def _move(p, v, s):
    t = _tangent(v, p)
    sp = t.norm(dim=-1, keepdim=True)
    return torch.where(sp < 1e-300, p, _unit(p * torch.cos(sp * s) + t * (torch.sin(sp * s) / sp.clamp_min(1e-300))))


#: centre, right and up of the six faces
_AXES = torch.tensor([[[0, 0, 1], [1, 0, 0], [0, 1, 0]], [[1, 0, 0], [0, 0, -1], [0, 1, 0]],
                      [[0, 0, -1], [-1, 0, 0], [0, 1, 0]], [[-1, 0, 0], [0, 0, 1], [0, 1, 0]],
                      [[0, 1, 0], [1, 0, 0], [0, 0, -1]], [[0, -1, 0], [1, 0, 0], [0, 0, 1]]], dtype=torch.float64)


def _locate(d, N):
    a = d.abs()
    fx, fy, fz = (torch.where(d[:, k] > 0, pos, neg) for k, (pos, neg) in enumerate(((1, 3), (4, 5), (0, 2))))
    f = torch.where((a[:, 0] >= a[:, 1]) & (a[:, 0] >= a[:, 2]), fx, torch.where(a[:, 1] >= a[:, 2], fy, fz))
    ax = _AXES.to(d.device)[f]
    pr = (ax * d[:, None, :]).sum(-1)
    h = math.pi / 2 / N
    return f, (torch.atan(pr[:, 1] / pr[:, 0]) + math.pi / 4) / h - 0.5, \
        (torch.atan(pr[:, 2] / pr[:, 0]) + math.pi / 4) / h - 0.5


def _cell(f, i, j, N):
    """The cell of (i, j) on face f; off the face, the cell that holds that centre's direction.  A corner ghost's
    direction lies on the seam of two faces up to rounding: the centres' angles are rounded once, as by an FMA."""
    off = (i < 0) | (j < 0) | (i >= N) | (j >= N)
    c = (f * N + j) * N + i
    if bool(off.any()):
        fo, io, jo = f[off], i[off], j[off]
        ax = _AXES.to(f.device)[fo]
        k = np.arange(-1, N + 1).astype(np.longdouble) + 0.5
        tan = torch.from_numpy(np.tan((k * (math.pi / 2 / N) - math.pi / 4).astype(np.float64))).to(f.device)
        d = ax[:, 0] + ax[:, 1] * tan[io + 1][:, None] + ax[:, 2] * tan[jo + 1][:, None]
        d = d * (1.0 / torch.sqrt(_dot(d, d)))
        g, x, y = _locate(d, N)
        c[off] = (g * N + (y + 0.5).floor().long().clamp(0, N - 1)) * N + (x + 0.5).floor().long().clamp(0, N - 1)
    return c


def _taps(p, N):
    f, x, y = _locate(p, N)
    i, j = x.floor().long(), y.floor().long()
    fx, fy = x - i, y - j
    idx = torch.stack([_cell(f, i + a, j + b, N) for b in (0, 1) for a in (0, 1)], 1)
    return idx, torch.stack([(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy], 1)


def _sample(fld, p, N):
    idx, wt = _taps(p, N)
    if fld.dim() == 1:
        return (fld[idx] * wt).sum(1)
    return _tangent((fld[idx] * wt[..., None]).sum(1), p)


class _Grid64:
    """The public tables of a grid in FP64."""

    def __init__(self, own, grid):
        cs, n = grid.cs, grid.n
        self.N, self.n = cs.N, n
        self.pos = view(own, cs.pos, (n, 3)).double()
        self.area = view(own, cs.area, (n,)).double()
        nbr = view(own, cs.nbr, (n, 8), "<i4").long()
        nnb = view(own, cs.nnb, (n,), "|u1").long()
        on = torch.arange(8, device="cuda")[None] < nnb[:, None]
        self.nbr = torch.where(on, nbr, torch.arange(n, device="cuda")[:, None])
        self.w = view(own, cs.w, (n, 8)).double() * on
        self.elen = view(own, cs.elen, (n, 8)).double() * on
        self.gc = view(own, cs.gc, (n, 8, 3)).double() * on[..., None]
        self.on = on

    def stencil(self, x):
        return (self.w * (x[:, None] - x[self.nbr])).sum(1)

    def mean(self, f):
        return (self.area * f).sum() / self.area.sum()

    def normals(self):
        d = self.pos[self.nbr] - self.pos[:, None]
        return d / d.norm(dim=-1, keepdim=True).clamp_min(1e-300)

    def curl(self, vel):
        wi = torch.linalg.cross(vel, self.pos)
        return (self.elen * 0.5 * ((wi[:, None] + wi[self.nbr]) * self.normals()).sum(-1)).sum(1) / self.area

    def divergence(self, vel):
        return (self.elen * 0.5 * ((vel[:, None] + vel[self.nbr]) * self.normals()).sum(-1)).sum(1) / self.area

    def velocity(self, psi):
        return torch.linalg.cross(self.pos, (self.gc * (psi[self.nbr] - psi[:, None])[..., None]).sum(1))

    def solve(self, omega, psi):
        b = -self.area * (omega - self.mean(omega))
        dinv = 1.0 / self.w.sum(1)
        x = psi.clone()
        r = b - self.stencil(x)
        z = dinv * r
        p, rz, stop = z.clone(), (r * z).sum(), 1e-11 * float(b.norm())
        for it in range(30_000):
            ap = self.stencil(p)
            al = rz / (p * ap).sum()
            x += al * p
            r -= al * ap
            if it % 32 == 0 and float(r.norm()) <= stop:
                break
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x - self.mean(x)


def _fluid64(g, c, omega, psi, vel, band, dt):
    y2 = 2.0 * c.get("rotation", 0.0) * g.pos[:, 1]
    q0 = omega + y2

    def depart(s):
        return _move(g.pos, _tangent(_sample(vel, _move(g.pos, vel, 0.5 * s), g.N), g.pos), s)

    back = depart(-dt)
    q = _sample(q0, back, g.N)
    if c.get("bfecc", 1):
        src = q0 + 0.5 * (q0 - _sample(q, depart(dt), g.N))
        idx, wt = _taps(back, g.N)
        q = (src[idx] * wt).sum(1).clamp(min=q0[idx].amin(1), max=q0[idx].amax(1))
    w = q - y2
    w = w + (1.0 - math.exp(-c.get("forcing", 0.0) * dt)) * (band - w)
    w = w - g.mean(w)
    psi = g.solve(w, psi)
    return dict(omega=w, psi=psi, vel=g.velocity(psi))


def _advect64(pos, vel, N, dt):
    u = _sample(vel, pos, N)
    return _move(pos, _tangent(_sample(vel, _move(pos, u, 0.5 * dt), N), pos), dt)


def _splat64(prev, pos, col, faces, R, radius, alpha, g):
    """Every texel's samples blended "over" in the order of (particle, sample)."""
    dev = pos.device
    prev, pos = prev.float().double(), pos.float().double()  # the positions are stored as FP32
    ang = torch.atan2(torch.linalg.cross(prev, pos).norm(dim=1), (prev * pos).sum(1))
    ns = torch.ceil(ang / (0.7 / R)).long().clamp(1, 4096)
    who = torch.repeat_interleave(torch.arange(len(ns), device=dev), ns)
    k = torch.arange(len(who), device=dev) - (torch.cumsum(ns, 0) - ns)[who] + 1
    t = (k.double() / ns[who])[:, None]
    d = _unit(prev[who] * (1 - t) + pos[who] * t)
    order, texel, weight = [], [], []
    span = range(int(2 * radius) + 1)
    for f in range(6):
        ax = _AXES[f].to(dev)
        dc = d @ ax[0]
        at = torch.nonzero(dc >= 0.5)[:, 0]
        px = (d[at] @ ax[1] / dc[at] + 1) * 0.5 * R - 0.5
        py = (1 - d[at] @ ax[2] / dc[at]) * 0.5 * R - 0.5
        x0, y0 = torch.ceil(px - radius), torch.ceil(py - radius)
        for dy in span:
            for dx in span:
                x, y = x0 + dx, y0 + dy
                wx, wy = 1 - (x - px).abs() / radius, 1 - (y - py).abs() / radius
                ok = (wx > 0) & (wy > 0) & (x >= 0) & (y >= 0) & (x < R) & (y < R)
                order.append(at[ok])
                texel.append(((f * R + y.long()) * R + x.long())[ok])
                weight.append((wx * wy)[ok])
    order, texel, weight = torch.cat(order), torch.cat(texel), torch.cat(weight)
    by = torch.argsort(texel * len(who) + order)
    order, texel, weight = who[order[by]], texel[by], weight[by]
    del by, d
    tex, cnt = torch.unique_consecutive(texel, return_counts=True)
    first = torch.cumsum(cnt, 0) - cnt
    buf = faces.reshape(-1, 4).clone()
    for r in range(int(cnt.max()) if len(cnt) else 0):
        on = cnt > r
        e = first[on] + r
        cc = col[order[e]]
        w = (alpha * cc[:, 3] * weight[e])[:, None]
        add = w / g * torch.cat([cc[:, :3], torch.ones_like(w)], 1)
        buf[tex[on]] = buf[tex[on]] * (1 - w) + add
    return buf.reshape(faces.shape)


def _step64(own, c, grid, fs, ps, sp):
    g, n = _Grid64(own, grid), grid.n
    F = fs.F
    omega, psi, band = (view(own, p, (n,)).double() for p in (F.omega, F.psi, F.omega_band))
    vel = view(own, F.vel, (n, 3)).double()
    dt = CFL * grid.cs.h / max(float(vel.norm(dim=1).max()), 1e-6)
    out = _fluid64(g, c, omega, psi, vel, band, dt)
    if ps is not None:
        pos = view(own, ps.P.pos, (ps.P.n, 3)).double()
        out["pos"] = _advect64(pos, vel, g.N, dt)
        out["faces"] = _splat64(pos, out["pos"], view(own, ps.P.col, (ps.P.n, 4)).double(),
                                view(own, sp.r.buf, (6, sp.r.R, sp.r.R, 4)).double(), sp.r.R, sp.r.radius, sp.r.alpha,
                                (1 - FADE) * sp.r.g)
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "output":
        return None  # bytes
    st = prepare(c, seed)
    own = st["own"]
    if kind in ("step", "fluid"):
        return _step64(own, c, st["grid"], st["fs"], st.get("ps"), st.get("sp"))
    if kind == "batch":
        return [_step64(own, p[0], *p[1:]) for p in st["planets"]]
    if kind == "deposit":
        P, r = st["ps"].P, st["sp"].r
        return dict(faces=_splat64(view(own, P.prev, (P.n, 3)).double(), view(own, P.pos, (P.n, 3)).double(),
                                   view(own, P.col, (P.n, 4)).double(), st["out"]["faces"].double(), r.R, r.radius,
                                   r.alpha, (1 - FADE) * r.g))
    vel = st["vel"].double().view(-1, 3)
    if kind == "advect":
        pos = st["out"]["pos"].double()
        return dict(pos=_advect64(pos, vel, c["N"], st["dt"]), prev=pos)
    g = _Grid64(own, st["grid"])
    curl = g.curl(vel)
    if kind == "operators":
        return dict(curl=curl, div=g.divergence(vel), lap=-g.stencil(curl.float().double()) / g.area)
    omega = curl - g.mean(curl)
    band = g.curl(st["band"].double().view(-1, 3))
    psi = g.solve(omega, torch.zeros_like(omega))
    return dict(omega=omega, psi=psi, vel=g.velocity(psi), omega_band=band - g.mean(band))
