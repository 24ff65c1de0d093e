"""The work that users of this framework have it do, as cases to time.

Every case is the pressure-projection step of the flow solver (or, for the
allocation-free entry point, its divergence check) called the way a time loop
calls it: grids are set up once and stay resident with their operator and
multigrid hierarchy, each pass brings an intermediate velocity U* and takes
away the corrected fluxes and the pressure.  Sizes, wall stretching, skew,
bodies and tolerances are those of the repository's workloads (64^3 channel,
256x128x128 sphere, 512x256x256 terrain, the uneven batch, the served streams)
and of the sizes between them.

Kinds:
  resident   vfs_projection_step on the resident U*, then the fields read back
  flow       the reference-shaped calls (projection.py), one by one
  hosted     one served request: host U* in, host fluxes and pressure out
  batch      vfs_projection_step_batch over uneven grids
  serve      several streams in flight, each warm-started from its last phi
  moving     a body moved: new nvert, operator rebuilt, then a step
  divcheck   vfs_divergence_max_noalloc on the caller's device arrays
"""
import ctypes
import math
import random

import numpy as np
import torch

from vfs_v3p2_gb300 import capi, projection, synth

DT = 0.04
TOL = dict(rtol=1e-9, div_tol=1e-8)


def listed():
    base = dict(beta=2.0, skew=0.05, bodies=0, precision="mixed", flux="gauss")

    def c(name, kind, ni, nj, nk, levels, **kw):
        return dict(base, name=name, kind=kind, ni=ni, nj=nj, nk=nk, levels=levels, **kw)

    return [
        # the smallest grid of the batch and serving ranges, straight lines: launches and latency
        c("channel 32^3", "resident", 32, 32, 32, 4, skew=0.0),
        # the plain FP64 64^3 channel workload with its 3-level hierarchy
        c("channel 64^3 fp64", "resident", 64, 64, 64, 3, precision="fp64"),
        # extents that are no multiple of a warp, rows of odd pitch, two bodies
        c("ragged 104x40x72", "resident", 104, 40, 72, 4, bodies=2, beta=2.7, skew=0.08),
        # the headline workload: one large grid with an immersed sphere, mixed and plain FP64
        c("sphere 256x128x128", "resident", 256, 128, 128, 5, bodies=1, flux="profile"),
        c("sphere 256x128x128 fp64", "resident", 256, 128, 128, 5, bodies=1, flux="profile", precision="fp64"),
        # the largest workload: terrain-following lines, all cross terms
        c("terrain 512x256x256", "resident", 512, 256, 256, 5, beta=2.5, flux="profile", terrain=True),
        # a host time loop that keeps its fields in host memory
        c("hosted 192x96x96", "hosted", 192, 96, 96, 5, skew=0.0),
        # a caller that swaps the reference's functions one for one, re-orthogonalising
        c("flow 128x64x96", "flow", 128, 64, 96, 5, bodies=1, orth="cgs2"),
        # many uneven grids in one launch per iteration
        c("batch of 16", "batch", 192, 96, 96, 5, count=16, grids=4),
        # warm-started streams of different sizes in flight together
        c("serve 6 streams", "serve", 256, 128, 128, 5, count=6, grids=7),
        # a moving body: masks, operator and coarse inverse rebuilt every step
        c("moving 96x48x48", "moving", 96, 48, 48, 4, bodies=1),
        # the divergence check alone, on a caller's arrays of odd extents
        c("divcheck 151x67x93", "divcheck", 151, 67, 93, 1, bodies=1, skew=0.0),
    ]


def _extent(rng, lo, hi):
    return max(8, 8 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 8))


def draw(rng):
    kind = rng.choice(["resident"] * 8 + ["hosted", "hosted", "flow", "flow", "batch", "batch", "serve", "moving", "divcheck",
                                          "divcheck"])
    case = dict(kind=kind, beta=round(rng.uniform(1.5, 3.0), 3), skew=rng.choice([0.0, round(rng.uniform(0.0, 0.1), 4)]),
                bodies=rng.randrange(4), precision=rng.choice(["mixed", "mixed", "mixed", "fp64"]), flux="gauss")
    if kind == "divcheck":
        # any caller's grid: odd extents as they come
        e = [round(math.exp(rng.uniform(math.log(17), math.log(m)))) for m in (384, 192, 192)]
        case.update(ni=e[0], nj=e[1], nk=e[2], levels=1, skew=0.0)
        return case
    hi = {"moving": (128, 64, 64), "batch": (192, 96, 96)}.get(kind, (256, 128, 128))
    e = [_extent(rng, 32, m) for m in hi]
    case.update(ni=e[0], nj=e[1], nk=e[2], levels=synth.mg_levels(*e))
    if kind == "resident":
        case["flux"] = rng.choice(["gauss", "profile"])
        if rng.random() < 0.2:
            case.update(terrain=True, flux="profile", beta=round(rng.uniform(2.0, 3.0), 3), skew=0.0, bodies=0)
    if kind == "flow":
        case["orth"] = rng.choice(["cgs", "cgs2"])
    if kind in ("batch", "serve"):
        case.update(count=rng.randrange(3, 13) if kind == "batch" else rng.randrange(2, 7), grids=rng.randrange(1 << 20))
    if kind == "moving":
        case["bodies"] = max(1, case["bodies"])
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _lines(n, length):
    return length * torch.arange(n + 1, dtype=torch.float64, device=_dev()) / n


def _walls(nj, beta):
    eta = torch.arange(nj + 1, dtype=torch.float64, device=_dev()) / nj
    return torch.tanh(beta * (2.0 * eta - 1.0)) / math.tanh(beta)


def _hill(x, z):
    return 0.25 * torch.exp(-((x - math.pi) ** 2 + (z - math.pi / 2) ** 2) / 0.5)


def _coords(c):
    """Node coordinates [mz, my, mx, 3], nodes 0..n valid."""
    ni, nj, nk = c["ni"], c["nj"], c["nk"]
    coor = torch.zeros((nk + 2, nj + 2, ni + 2, 3), dtype=torch.float64, device=_dev())
    x, z = _lines(ni, 2 * math.pi), _lines(nk, math.pi)
    v = coor[: nk + 1, : nj + 1, : ni + 1]
    v[..., 2] = z[:, None, None]
    if c.get("terrain"):
        eta = torch.arange(nj + 1, dtype=torch.float64, device=_dev()) / nj
        s = 1.0 + torch.tanh(c["beta"] * (eta - 1.0)) / math.tanh(c["beta"])
        h = _hill(x[None, None, :], z[:, None, None])
        v[..., 0] = x
        v[..., 1] = h + (1.0 - h) * s[None, :, None]
    else:
        v[..., 0] = x[None, None, :] + c["skew"] * torch.sin(z)[:, None, None]
        v[..., 1] = _walls(nj, c["beta"])[None, :, None]
    return coor


def _spheres(c, rng):
    if c["bodies"] == 1 and c["kind"] != "moving":
        return [(math.pi, 0.0, math.pi / 2, 0.3)]
    return [(rng.uniform(1.0, 2 * math.pi - 1.0), rng.uniform(-0.5, 0.5), rng.uniform(0.6, math.pi - 0.6), rng.uniform(0.1, 0.3))
            for _ in range(c["bodies"])]


def _nvert(c, coor, spheres):
    """4 in a sphere, 1 on fluid cells beside one, 0 elsewhere."""
    nv = torch.zeros(coor.shape[:3], dtype=torch.float64, device=coor.device)
    if not spheres:
        return nv
    n = coor
    cent = 0.125 * sum(n[a : a - 1 or None, b : b - 1 or None, d : d - 1 or None] for a in (0, 1) for b in (0, 1) for d in (0, 1))
    cent = cent[: c["nk"], : c["nj"], : c["ni"]]
    solid = torch.zeros(coor.shape[:3], dtype=torch.bool, device=coor.device)
    for s in spheres:
        d = cent - torch.tensor(s[:3], dtype=torch.float64, device=coor.device)
        solid[1:-1, 1:-1, 1:-1] |= (d * d).sum(-1) < s[3] ** 2
    near = torch.zeros_like(solid)
    near[:, :, 1:] |= solid[:, :, :-1]
    near[:, :, :-1] |= solid[:, :, 1:]
    near[:, 1:] |= solid[:, :-1]
    near[:, :-1] |= solid[:, 1:]
    near[1:] |= solid[:-1]
    near[:-1] |= solid[1:]
    near[0] = near[-1] = near[:, 0] = near[:, -1] = near[:, :, 0] = near[:, :, -1] = False
    nv[near & ~solid] = 1.0
    nv[solid] = 4.0
    nv[:, :, 0], nv[:, :, -1] = nv[:, :, -2].clone(), nv[:, :, 1].clone()
    nv[0], nv[-1] = nv[-2].clone(), nv[1].clone()
    return nv


def _finish(u):
    """No flux through the walls, none outside the domain, periodic ghost faces equal to their partners."""
    out = torch.zeros_like(u)
    out[1:-1, 1:-1, :-1, 0] = u[1:-1, 1:-1, :-1, 0]
    out[1:-1, 1:-2, 1:-1, 1] = u[1:-1, 1:-2, 1:-1, 1]
    out[:-1, 1:-1, 1:-1, 2] = u[:-1, 1:-1, 1:-1, 2]
    out[:, :, 0, 0], out[:, :, -1, 0] = out[:, :, -2, 0], out[:, :, 1, 0]
    out[0, :, :, 2], out[-1, :, :, 2] = out[-2, :, :, 2], out[1, :, :, 2]
    return out


def _ustar(c, coor, seed):
    """U* on the faces: N(0, 1), or the workload's mean profile plus noise through the face areas."""
    gen = torch.Generator(device=_dev()).manual_seed(seed & 0x7FFFFFFF)
    u = torch.randn(coor.shape, generator=gen, dtype=torch.float64, device=_dev())
    if c["flux"] == "gauss":
        return _finish(u)
    u *= 0.05 if c.get("terrain") else 0.1
    n = coor
    y_i = 0.25 * (n[1:, 1:, :, 1] + n[:-1, 1:, :, 1] + n[1:, :-1, :, 1] + n[:-1, :-1, :, 1])
    out = torch.zeros_like(u)
    # the profile has an x component alone; the noise is N(0, sigma) times the face's largest area component
    for f, a, b in ((0, n[1:, 1:] - n[:-1, :-1], n[1:, :-1] - n[:-1, 1:]),
                    (1, n[1:, :, 1:] - n[:-1, :, :-1], n[:-1, :, 1:] - n[1:, :, :-1]),
                    (2, n[:, 1:, 1:] - n[:, :-1, :-1], n[:, 1:, :-1] - n[:, :-1, 1:])):
        area = 0.5 * torch.linalg.cross(b, a)
        to = (out[1:, 1:, :, 0], out[1:, :, 1:, 1], out[:, 1:, 1:, 2])[f]
        noise = (u[1:, 1:, :, 0], u[1:, :, 1:, 1], u[:, 1:, 1:, 2])[f]
        to += noise * area[..., f]
        if f == 0:
            if c.get("terrain"):
                h = _hill(n[1:, 1:, :, 0], n[1:, 1:, :, 2])
                to += area[..., 0] * torch.log1p(30.0 * torch.clamp(y_i - h, min=0.0)) / math.log(31.0)
            else:
                to += area[..., 0] * (1.0 - y_i**2)
        del area
    return _finish(out)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _to_host(t):
    h = _pinned(t.shape)
    h.copy_(t)
    return h


def _params(c, **kw):
    if c.get("orth"):
        kw["orth"] = c["orth"]
    return capi.default_params(precision=c["precision"], **TOL, **kw)


class State:
    pass


class _Loaded:
    """One grid of a context, set up, with its U* and its host buffers for the results."""

    def __init__(self, ctx, c, seed, spheres=None):
        self.case = c
        coor = _coords(c)
        nv = _nvert(c, coor, _spheres(c, random.Random("%(ni)d %(nj)d %(nk)d %(bodies)d" % c)) if spheres is None else spheres)
        self.ustar = _to_host(_ustar(c, coor, seed))
        self.coor, self.nvert = coor.cpu().numpy(), nv.cpu().numpy()
        self.shape = self.nvert.shape
        del coor, nv
        if torch.cuda.is_available():
            torch.cuda.empty_cache()
        self.ctx = ctx
        self.gid = ctx.grid_create(self.coor, self.nvert, c["levels"], 1 if c["bodies"] else 0)
        ctx.poisson_lhs(self.gid)
        self.u, self.p = _pinned(self.shape + (3,)), _pinned(self.shape)

    def put_ustar(self):
        self.ctx.set_field(self.gid, capi.FIELD_USTAR, self.ustar.numpy())

    def fetch(self):
        for field, to in ((capi.FIELD_UCONT, self.u), (capi.FIELD_P, self.p)):
            self.ctx.check(self.ctx.L.vfs_get_field(self.ctx.h, self.gid, field, capi.dptr(to.numpy())))
        return {"u": self.u, "p": self.p}


def _many(c):
    """The grids of a batch or of the served streams: extents log-uniform from 32^3 up to the case's."""
    rng = random.Random(c["grids"])
    out = []
    for _ in range(c["count"]):
        e = [_extent(rng, 32, m) for m in (c["ni"], c["nj"], c["nk"])]
        out.append(dict(c, ni=e[0], nj=e[1], nk=e[2], levels=synth.mg_levels(*e), beta=rng.uniform(1.5, 3.0),
                        skew=rng.uniform(0.0, 0.1), bodies=rng.randrange(4)))
    return out


def prepare(case, seed):
    s = State()
    s.case = case
    kind = case["kind"]
    if kind == "divcheck":
        coor = _coords(case)
        nv = _nvert(case, coor, _spheres(case, random.Random(seed)))
        u = _ustar(case, coor, seed)
        s.u = [u[..., q].contiguous() for q in range(3)]
        s.aj = torch.rand(nv.shape, generator=torch.Generator(device=_dev()).manual_seed(seed + 1), dtype=torch.float64,
                          device=_dev()) + 0.5
        s.nvert = nv
        s.out = torch.zeros(1, dtype=torch.float64, device=_dev())
        return s
    ctx = s.ctx = capi.Context(0)
    if kind in ("batch", "serve"):
        s.grids = [_Loaded(ctx, g, seed * 64 + q) for q, g in enumerate(_many(case))]
        s.params = _params(case, warm_start=1 if kind == "serve" else 0)
        if kind == "batch":
            for g in s.grids:
                g.put_ustar()
        else:
            for q, g in enumerate(s.grids):  # the stream's next velocity: a small change of the last
                gen = torch.Generator(device=_dev()).manual_seed((seed * 64 + q) & 0x7FFFFFFF ^ 0x5EED)
                d = 0.01 * torch.randn(g.ustar.shape, generator=gen, dtype=torch.float64, device=_dev())
                g.next = _to_host(_finish(g.ustar.to(_dev()) + d))
                g.u2, g.p2 = _pinned(g.shape + (3,)), _pinned(g.shape)
                g.p_in = torch.zeros_like(g.p).pin_memory() if torch.cuda.is_available() else torch.zeros_like(g.p)
        return s
    s.params = _params(case)
    if kind == "flow":
        coor = _coords(case)
        nv = _nvert(case, coor, _spheres(case, random.Random("%(ni)d %(nj)d %(nk)d %(bodies)d" % case)))
        s.ustar = _to_host(_ustar(case, coor, seed))
        s.user = projection.UserCtx(coor.cpu().numpy(), nv.cpu().numpy(), case["levels"], 1 if case["bodies"] else 0, dt=DT, ctx=ctx)
        projection.PoissonLHSNew(s.user)
        s.u, s.p = _pinned(coor.shape), _pinned(coor.shape[:3])
        return s
    if kind == "moving":
        rng = random.Random(seed)
        s.grid = _Loaded(ctx, case, seed, _spheres(case, rng))
        s.grid.put_ustar()
        # where the bodies are at the step to come
        s.nvert = _nvert(case, torch.from_numpy(s.grid.coor).to(_dev()), _spheres(case, rng)).cpu().numpy()
        return s
    s.grid = _Loaded(ctx, case, seed)
    if kind == "resident":
        s.grid.put_ustar()
    else:
        s.p_in = _pinned(s.grid.shape)
        s.p_in.zero_()
    return s


# ---------------------------------------------------------------------------
# Passes
# ---------------------------------------------------------------------------
def _finish_requests(ctx, n):
    for _ in range(n):
        done = None
        while done is None:
            done = ctx.poll(wait=True)
        if done[1]:
            raise capi.VfsError(done[1], "request failed")


def run(s):
    kind = s.case["kind"]
    if kind == "resident":
        s.ctx.projection_step(s.grid.gid, s.params, dt=DT)
        return s.grid.fetch()
    if kind == "hosted":
        g = s.grid
        s.ctx.submit(g.gid, s.params, g.ustar.data_ptr(), g.u.data_ptr(), s.p_in.data_ptr(), g.p.data_ptr(), dt=DT)
        _finish_requests(s.ctx, 1)
        return {"u": g.u, "p": g.p}
    if kind == "flow":
        user = s.user
        user.Ucont = s.ustar.numpy()
        projection.Flow_Solver_pressure(user, s.params)
        for field, to in ((capi.FIELD_UCONT, s.u), (capi.FIELD_P, s.p)):
            user.ctx.check(user.ctx.L.vfs_get_field(user.ctx.h, user.grid, field, capi.dptr(to.numpy())))
        return {"u": s.u, "p": s.p}
    if kind == "batch":
        s.ctx.projection_step_batch([g.gid for g in s.grids], s.params, dt=DT)
        return [g.fetch() for g in s.grids]
    if kind == "serve":
        for g in s.grids:
            s.ctx.submit(g.gid, s.params, g.ustar.data_ptr(), g.u.data_ptr(), g.p_in.data_ptr(), g.p.data_ptr(), dt=DT)
        _finish_requests(s.ctx, len(s.grids))
        for g in s.grids:
            s.ctx.submit(g.gid, s.params, g.next.data_ptr(), g.u2.data_ptr(), g.p_in.data_ptr(), g.p2.data_ptr(), dt=DT)
        _finish_requests(s.ctx, len(s.grids))
        return [{"u": g.u, "p": g.p, "u2": g.u2, "p2": g.p2} for g in s.grids]
    if kind == "moving":
        g = s.grid
        s.ctx.update_nvert(g.gid, s.nvert)
        s.ctx.poisson_lhs(g.gid)
        s.ctx.projection_step(g.gid, s.params, dt=DT)
        return g.fetch()
    mz, my, mx = s.nvert.shape
    err = ctypes.create_string_buffer(256)
    rc = capi.load().vfs_divergence_max_noalloc(0, mx, my, mz, 1, 0, 1, *(ctypes.c_void_p(t.data_ptr()) for t in s.u),
                                                ctypes.c_void_p(s.aj.data_ptr()), ctypes.c_void_p(s.nvert.data_ptr()),
                                                ctypes.c_void_p(s.out.data_ptr()),
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), err, 256)
    if rc:
        raise capi.VfsError(rc, err.value.decode())
    return s.out


def work(case):
    cells = lambda c: (c["ni"] + 2) * (c["nj"] + 2) * (c["nk"] + 2)  # noqa: E731
    if case["kind"] == "divcheck":
        return {"bytes": 40.0 * cells(case), "flops": 7.0 * cells(case)}
    n = sum(map(cells, _many(case))) * (2 if case["kind"] == "serve" else 1) if "count" in case else cells(case)
    # U*, the pressure, nvert and the node coordinates read, U, the pressure and the Cartesian velocity written;
    # one application of the 19-point operator and of the correction
    return {"bytes": 120.0 * n, "flops": 120.0 * n}


# ---------------------------------------------------------------------------
# What the passes return, in 64 bits, where there is a closed way to it
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "divcheck":
        coor = _coords(case)
        nv = _nvert(case, coor, _spheres(case, random.Random(seed)))
        u = _ustar(case, coor, seed)
        aj = torch.rand(nv.shape, generator=torch.Generator(device=_dev()).manual_seed(seed + 1), dtype=torch.float64,
                        device=_dev()) + 0.5
        i = slice(1, -1)
        div = (u[i, i, i, 0] - u[i, i, :-2, 0] + u[i, i, i, 1] - u[i, :-2, i, 1] + u[i, i, i, 2] - u[:-2, i, i, 2]) * aj[i, i, i]
        wet = nv + sum(torch.roll(nv, s, a) for a in range(3) for s in (1, -1))
        return torch.where(wet[i, i, i] > 0.1, 0.0, div.abs()).max().reshape(1)
    if case["kind"] not in ("resident", "hosted") or case["skew"] or case["bodies"] or case.get("terrain"):
        return None  # the solution of a general 19-point system
    # straight lines: in x and z the operator is diagonal under the Fourier transform, in y it is tridiagonal
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    u = _ustar(case, _coords(case), seed)
    dx, dz, y = 2 * math.pi / ni, math.pi / nk, _walls(nj, case["beta"])
    yc = 0.5 * (y[1:] + y[:-1])
    h = torch.empty_like(yc)  # the cell heights as the face metrics have them
    h[1:-1] = 0.5 * (yc[2:] - yc[:-2])
    h[0], h[-1] = yc[1] - yc[0], yc[-1] - yc[-2]
    gi, gk = h * dz / dx, h * dx / dz
    gj = dx * dz / (0.5 * (y[2:] - y[:-2]))
    div = u[1:-1, 1:-1, 1:-1, 0] - u[1:-1, 1:-1, :-2, 0]
    div = div + u[1:-1, 1:-1, 1:-1, 1] - u[1:-1, :-2, 1:-1, 1] + u[1:-1, 1:-1, 1:-1, 2] - u[:-2, 1:-1, 1:-1, 2]
    rhs = torch.fft.fft2(div / DT, dim=(0, 2))
    lx = 2 * torch.cos(2 * math.pi * torch.arange(ni, dtype=torch.float64, device=_dev()) / ni) - 2
    lz = 2 * torch.cos(2 * math.pi * torch.arange(nk, dtype=torch.float64, device=_dev()) / nk) - 2
    lx[0] = lz[0] = 0.0
    diag = gi[None, :, None] * lx[None, None, :] + gk[None, :, None] * lz[:, None, None]
    diag[:, :-1] -= gj[None, :, None]
    diag[:, 1:] -= gj[None, :, None]
    rhs[0, 0, 0], diag[0, 0, 0] = 0.0, diag[0, 0, 0] - gj[0]  # the constant: pinned here, its mean taken out below
    m = [diag[:, 0].clone()]
    f = [rhs[:, 0].clone()]
    for j in range(1, nj):
        r = gj[j - 1] / m[-1]
        m.append(diag[:, j] - r * gj[j - 1])
        f.append(rhs[:, j] - r * f[-1])
    x = [None] * nj
    x[-1] = f[-1] / torch.where(m[-1] == 0, torch.ones_like(m[-1]), m[-1])
    for j in range(nj - 2, -1, -1):
        x[j] = (f[j] - gj[j] * x[j + 1]) / m[j]
    phi = torch.fft.ifft2(torch.stack(x, 1), dim=(0, 2)).real
    phi = phi - phi.mean()
    u[1:-1, 1:-1, 1:-1, 0] -= DT * gi[None, :, None] * (torch.roll(phi, -1, 2) - phi)
    u[1:-1, 1:-2, 1:-1, 1] -= DT * gj[None, :, None] * (phi[:, 1:] - phi[:, :-1])
    u[1:-1, 1:-1, 1:-1, 2] -= DT * gk[None, :, None] * (torch.roll(phi, -1, 0) - phi)
    # ghosts of the periodic axes hold their partners' values
    ii = torch.tensor([ni] + list(range(1, ni + 1)) + [1], device=_dev())
    kk = torch.tensor([nk] + list(range(1, nk + 1)) + [1], device=_dev())
    ux, uz = u[..., 0][kk][:, :, ii], u[..., 2][kk][:, :, ii]
    u[:, :, 0, 0], u[:, :, -1, 0] = ux[:, :, 0], ux[:, :, -1]
    u[0, :, :, 2], u[-1, :, :, 2] = uz[0], uz[-1]
    p = torch.zeros(u.shape[:3], dtype=torch.float64, device=_dev())
    p[1:-1, 1:-1, 1:-1] = phi
    p = p[kk][:, :, ii]
    return {"u": u.cpu(), "p": p.cpu()}
