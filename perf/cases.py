"""Performance cases of flub_gb300: what a fluid simulation has it do.

A simulation step on a MAC grid advects the level set and the velocity,
projects the velocity (classification, divergence, MGPCG, gradient update),
extrapolates it into the air and redistances the level set; the learned warm
start adds the U-Net's convolutions, forward and backward.  Each case is one
of these calls through the package's public entry points.

``listed()`` are the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes inputs and handles on the GPU, ``run`` is one pass,
``work`` its unavoidable traffic, ``exact`` the same result in 64 bits with
plain torch.
"""
import math

import numpy as np
import torch

from flub_gb300 import Projection, learned, scenes
from flub_gb300 import kernels as K
from flub_gb300 import unet
from flub_gb300.fields import Field, IntField, MACGrid, MACGridInt, field_shape

# "project": one pressure projection (Projection.project), solved to relative
# residual 1e-6 as the reference's callers do.  layout: "box" and "dam" are
# partly filled tanks, "sphere" a full channel with a solid sphere.
_PROJECT = {"kind": "project", "precision": "fp32", "schedule": "reference", "warm": False}


def listed():
    return [
        # a preview-resolution tank: the smallest grid a scene is tried at; launches and latency
        dict(_PROJECT, name="project_box32", layout="box", nx=32, ny=32, nz=32, levels=3),
        # the 64^3 tank with the reference's V-cycle in FP32
        dict(_PROJECT, name="project_box64", layout="box", nx=64, ny=64, nz=64, levels=4),
        # a domain cut to a scene: extents that are no powers of two, rows of the coarser levels no multiple of 8
        dict(_PROJECT, name="project_ragged", layout="dam", nx=104, ny=72, nz=88, levels=3),
        # the reference's default grid (256 x 64 x 256), a wide shallow tank
        dict(_PROJECT, name="project_default_grid", layout="dam", nx=256, ny=64, nz=256, levels=4),
        # flow past a sphere, every cell fluid, FP16-stored V-cycle
        dict(_PROJECT, name="project_sphere128_mixed", layout="sphere", nx=128, ny=128, nz=128, levels=5,
             precision="mixed"),
        # the 256^3 dam break with the reference's V-cycle in FP32
        dict(_PROJECT, name="project_dam256", layout="dam", nx=256, ny=256, nz=256, levels=6),
        # the same dam break as the benchmark's headline runs it: learned start, FP16-stored light V-cycle
        dict(_PROJECT, name="project_dam256_learned", layout="dam", nx=256, ny=256, nz=256, levels=6,
             precision="mixed", schedule="v22", warm=True),
        # a production-resolution dam break, light V-cycle in FP32
        dict(_PROJECT, name="project_dam512_v22", layout="dam", nx=512, ny=512, nz=512, levels=7, schedule="v22"),
        # the step's advection on the default grid: level set, then the three face arrays (MacCormack)
        {"kind": "advect", "name": "advect_default_grid", "nx": 256, "ny": 64, "nz": 256},
        # extrapolation into the air after a 256^3 projection, 16 * res / 128 passes as the reference calls it
        {"kind": "extrapolate", "name": "extrapolate_256", "nx": 256, "ny": 256, "nz": 256, "passes": 32},
        # redistancing the level set of the default grid, boundary cells kept, as the particle level set calls it
        {"kind": "redistance", "name": "redistance_default_grid", "nx": 256, "ny": 64, "nz": 256, "boundary": 0},
        # training the warm start: one decoder layer of the U-Net (skip connection), forward and backward, batch 4
        {"kind": "conv", "name": "conv_dec0a_train", "c0": 32, "c1": 16, "cout": 16, "batch": 4, "nx": 64, "ny": 64,
         "nz": 64},
    ]


# ------------------------------------------------------------------ drawn cases

def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_project(rng):
    layout = rng.choice(("box", "dam", "dam", "sphere"))
    mode = rng.choice(("reference", "reference", "mixed", "v22", "learned"))
    if mode == "learned":  # the network wants power-of-two rows; it runs on the level whose rows are 64 long
        k = rng.choice((0, 1, 2) if layout != "sphere" else (0, 1))
        dims, levels = [rng.choice((24, 32, 40, 48, 56, 64)) << k, rng.choice((32, 64)) << k, 64 << k], 4 + k
    else:
        # the reference's schedule sweeps the coarse levels hundreds of times; a full channel holds 4 times a tank's water
        top = {"reference": 192, "mixed": 192, "v22": 288}[mode]
        n = _log_int(rng, 24, top if layout != "sphere" else min(top, 128))
        dims = [n] + [max(16, int(n * rng.choice((0.5, 0.75, 1.0, 1.0)))) for _ in range(2)]
        levels = max(2, 1 + int(math.log2(min(dims) / 8)))
        unit = 1 << (levels - 1)
        # rows of the coarsest level in pairs; the FP16-stored levels want whole groups of 8
        row = unit * (8 if mode == "mixed" else 2)
        dims = [max(1, round(d / u)) * u for d, u in zip(dims, (unit, unit, row))]
    return dict(_PROJECT, layout=layout, nx=dims[0], ny=dims[1], nz=dims[2], levels=levels,
                precision="mixed" if mode in ("mixed", "learned") else "fp32",
                schedule="v22" if mode in ("v22", "learned") else "reference", warm=mode == "learned")


def _draw_shape(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return {"nx": n, "ny": max(12, int(n * rng.uniform(0.25, 1.0))), "nz": max(12, int(n * rng.uniform(0.5, 1.1)))}


def draw(rng):
    kind = rng.choice(("project",) * 7 + ("advect", "extrapolate", "redistance", "conv"))
    if kind == "project":
        return _draw_project(rng)
    if kind == "advect":
        return dict(kind=kind, **_draw_shape(rng, 24, 224))
    if kind == "extrapolate":
        s = _draw_shape(rng, 24, 256)
        return dict(kind=kind, passes=max(1, 16 * s["nx"] // 128), **s)
    if kind == "redistance":
        return dict(kind=kind, boundary=rng.choice((0, 1)), **_draw_shape(rng, 24, 256))
    _, c0, c1, cout, level = rng.choice(unet.LAYERS)
    n = 1 << (6 - level)
    return dict(kind=kind, c0=c0, c1=c1, cout=cout, batch=rng.choice((1, 2, 3, 4)),
                nx=rng.randint(max(4, n // 4), n), ny=n, nz=n)


# ------------------------------------------------------------------ inputs

def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _axes(shape, device="cuda"):
    """Cell centres along each axis, in units of the x extent, broadcastable."""
    h = 1.0 / shape[0]
    c = [(torch.arange(n, dtype=torch.float64, device=device) + 0.5) * h for n in shape]
    return c[0][:, None, None], c[1][None, :, None], c[2][None, None, :]


def _layout(case, seed):
    """Level set (FP32, negative inside water) and solid primitives; the water line moves a little with the seed."""
    shape = _shape(case)
    h = 1.0 / shape[0]
    ey, ez = shape[1] * h, shape[2] * h
    small = min(1.0, ey, ez)
    rng = np.random.default_rng(seed)
    jx, jy = rng.uniform(0.97, 1.03, 2)
    x, y, z = _axes(shape)
    objs = []
    layout = case.get("layout", "dam")
    if layout == "box":
        phi = torch.maximum(x - 0.4 * jx, y - 0.6 * ey * jy).expand(shape)
    elif layout == "sphere":
        phi = (x - (1.0 - h)).expand(shape)  # outflow: one layer of air at the far end
        objs = [dict(geometry=scenes.GEOM_SPHERE, x=(0.5, 0.5 * ey, 0.5 * ez), radius=float(0.15 * small * jx)),
                # inflow: one solid layer whose rigid velocity is u = 1
                dict(geometry=scenes.GEOM_BOX, x=(0.0, 0.5 * ey, 0.5 * ez), radius=(h, 0.5 * ey + h, 0.5 * ez + h))]
    else:
        phi = torch.maximum(x - 0.35 * jx, y - 0.55 * ey * jy).expand(shape)
        ball = torch.sqrt((x - 0.7) ** 2 + (y - 0.3 * ey) ** 2 + (z - 0.5 * ez) ** 2) - 0.08 * small
        phi = torch.minimum(phi, ball)
        objs = [dict(geometry=scenes.GEOM_BOX, x=(0.6, 0.05 * ey, 0.45 * ez), radius=0.05 * small)]
    return phi.float().contiguous(), scenes.make_prims(objs)


def _grid(arrays, cls=MACGrid, field=Field):
    return cls(*(field(a, d=d + 1) for d, a in enumerate(arrays)))


def _velocity(case, seed):
    """Fourier modes with noise (scenes.fourier_faces_device), plus the inflow or a step of gravity."""
    u, v, w = scenes.fourier_faces_device(_shape(case), seed, "cuda")
    if case.get("layout") == "sphere":
        u += 1.0
    else:
        v -= 9.8 / 60.0
    return u, v, w


def _rigid(case):
    r = [torch.zeros(field_shape(_shape(case), d), dtype=torch.float32, device="cuda") for d in (1, 2, 3)]
    if case.get("layout") == "sphere":
        r[0][1] = 1.0
    return r


def _conv_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    rand = lambda *s: torch.randn(s, generator=gen, device="cuda")
    grid = (case["batch"],) + _shape(case)
    std = math.sqrt(2.0 / (27 * (case["c0"] + case["c1"])))
    s = {"x0": rand(*grid, case["c0"]).relu().to(torch.bfloat16),
         "w0": (rand(27, case["cout"], case["c0"]) * std).to(torch.bfloat16),
         "b": rand(case["cout"]) * 0.1, "dy": (rand(*grid, case["cout"]) * 1e-2).to(torch.bfloat16),
         "x1": None, "w1": None}
    if case["c1"]:
        s["x1"] = rand(*grid, case["c1"]).relu().to(torch.bfloat16)
        s["w1"] = (rand(27, case["cout"], case["c1"]) * std).to(torch.bfloat16)
    return s


def _advect_inputs(case, seed):
    vel = _velocity(case, seed)
    return vel, _layout(case, seed)[0]


def _redistance_input(case, seed):
    """A level set whose distances have drifted: the layout's, stretched and rippled away from the surface."""
    phi, _ = _layout(case, seed)
    x, y, z = _axes(_shape(case))
    k = 2 * math.pi * (2 + seed % 5)
    ripple = 1.0 + 0.4 * torch.sin(k * x) * torch.cos(1.3 * k * y) * torch.sin(0.7 * k * z + seed % 7)
    return (phi.double() * ripple).float().contiguous()


def prepare(case, seed):
    kind, shape = case["kind"], _shape(case)
    if kind == "project":
        phi, prims = _layout(case, seed)
        star = _velocity(case, seed)
        return {"kind": kind, "proj": Projection(shape, case["levels"], precision=case["precision"],
                                                 schedule=case["schedule"]),
                "warm": learned.WarmStart(unet.UNet3D.load(learned.WEIGHTS)) if case["warm"] else None,
                "phi": phi, "prims": prims, "star": star, "rigid": _grid(_rigid(case)),
                "vel": _grid([torch.empty_like(a) for a in star])}
    if kind == "advect":
        vel, phi = _advect_inputs(case, seed)
        return {"kind": kind, "vel": _grid(vel), "new": _grid([torch.empty_like(a) for a in vel]), "phi": Field(phi),
                "new_phi": Field(torch.empty_like(phi))}
    if kind == "extrapolate":
        phi, _ = _layout(case, seed)
        flags = [torch.zeros(field_shape(shape, d), dtype=torch.int32, device="cuda") for d in (1, 2, 3)]
        return {"kind": kind, "vel": _grid(_velocity(case, seed)), "flags": _grid(flags, MACGridInt, IntField),
                "phi": phi, "passes": case["passes"]}
    if kind == "redistance":
        phi = _redistance_input(case, seed)
        return {"kind": kind, "drifted": phi, "phi": Field(torch.empty_like(phi)), "boundary": case["boundary"]}
    s = _conv_inputs(case, seed)
    # the data gradient runs on the flipped, transposed weights that the optimiser keeps beside the weights
    turn = lambda w: w.flip(0).transpose(1, 2).contiguous() if w is not None else None
    zeros = lambda w: torch.zeros(w.shape, dtype=torch.float32, device="cuda") if w is not None else None
    s.update(kind=kind, w0t=turn(s["w0"]), w1t=turn(s["w1"]), dw0=zeros(s["w0"]), dw1=zeros(s["w1"]),
             db=zeros(s["b"]))
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    kind = s["kind"]
    if kind == "project":
        # the step's velocity, as the advection leaves it: the projection works in place
        vel = s["vel"]
        for f, a in zip((vel.u, vel.v, vel.w), s["star"]):
            f.f.copy_(a)
        proj = s["proj"]
        proj.project(vel, s["rigid"], s["phi"], s["prims"], warm_start=s["warm"], sync=False)
        return {"u": vel.u.f, "v": vel.v.f, "w": vel.w.f, "p": proj.p.f, "tag": proj.tag.f}
    if kind == "advect":
        K.advect_phi_field(s["vel"], s["phi"], s["new_phi"])
        K.advect_uv_mc(s["vel"], s["new"])
        return {"phi": s["new_phi"].f, "u": s["new"].u.f, "v": s["new"].v.f, "w": s["new"].w.f}
    if kind == "extrapolate":
        v, t = s["vel"], s["flags"]
        K.extrapolate(v, t, s["phi"], s["passes"])
        return {"u": v.u.f, "v": v.v.f, "w": v.w.f, "tu": t.u.f, "tv": t.v.f, "tw": t.w.f}
    if kind == "redistance":
        s["phi"].f.copy_(s["drifted"])
        K.redistance(s["phi"], set_boundary=s["boundary"])
        return s["phi"].f
    for k in ("dw0", "dw1", "db"):
        if s[k] is not None:
            s[k].zero_()
    out = {"y": unet.conv3d(s["x0"], s["w0"], s["x1"], s["w1"], s["b"], relu=True)}
    unet.conv3d_wgrad(s["x0"], s["dy"], s["dw0"], s["db"])
    out.update(dw0=s["dw0"], db=s["db"], dx0=unet.conv3d(s["dy"], s["w0t"], relu=False))
    if s["x1"] is not None:
        unet.conv3d_wgrad(s["x1"], s["dy"], s["dw1"], None)
        out.update(dw1=s["dw1"], dx1=unet.conv3d(s["dy"], s["w1t"], relu=False))
    return out


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "project":
        # read phi, three faces, three rigid faces; write three faces, pressure, tags; one Poisson residual's arithmetic
        return {"bytes": 48.0 * n, "flops": 30.0 * n}
    if kind == "advect":
        # velocity and level set in and out; three-stage traces and tricubic samples of four arrays
        return {"bytes": 32.0 * n, "flops": 4 * 900.0 * n}
    if kind == "extrapolate":
        return {"bytes": 40.0 * n, "flops": 27 * 3.0 * n}  # level set, faces in and out, flags out
    if kind == "redistance":
        return {"bytes": 8.0 * n, "flops": 33 * 15.0 * n}
    cin, co, vox = case["c0"] + case["c1"], case["cout"], n * case["batch"]
    return {"bytes": 2.0 * vox * (2 * cin + 2 * co) + 27 * co * cin * 8.0, "flops": 3 * 2.0 * 27 * cin * co * vox}


# ------------------------------------------------------------------ the same in 64 bits

def _prim_solid(prims, shape):
    """Cells whose centre lies inside a solid primitive (axis-aligned boxes and spheres)."""
    xs = _axes(shape)
    solid = torch.zeros(shape, dtype=torch.bool, device="cuda")
    for p in prims:
        c, r = [float(v) for v in p["x"]], [float(v) for v in p["radius"]]
        d = [a - b for a, b in zip(xs, c)]
        if int(p["geometry"]) == scenes.GEOM_SPHERE:
            solid |= (d[0] ** 2 + d[1] ** 2 + d[2] ** 2) < r[0] ** 2
        else:
            solid |= (d[0].abs() < r[0]) & (d[1].abs() < r[1]) & (d[2].abs() < r[2])
    return solid


def _side(t, axis, step, fill):
    """t of the neighbour one cell along +axis (step 1) or -axis (step -1); fill outside."""
    out = torch.full_like(t, fill)
    n = t.shape[axis]
    a, b = (out.narrow(axis, 0, n - 1), t.narrow(axis, 1, n - 1)) if step > 0 else (out.narrow(axis, 1, n - 1),
                                                                                    t.narrow(axis, 0, n - 1))
    a.copy_(b)
    return out


def _poisson_cg(fluid, air, rhs, tol=1e-11, limit=12000):
    """sum over open neighbours of (x_n - x_c) = rhs on the fluid cells (x = 0 in air), conjugate gradients in FP64."""
    shape = fluid.shape
    cells = fluid.reshape(-1).nonzero().squeeze(1)
    m = cells.numel()
    slot = torch.full((fluid.numel(),), m, dtype=torch.int32, device="cuda")  # m: a slot that stays 0
    slot[cells] = torch.arange(m, dtype=torch.int32, device="cuda")
    slot = slot.view(shape)
    nbr, diag = [], torch.zeros(m, dtype=torch.float64, device="cuda")
    for axis in range(3):
        for step in (1, -1):
            nbr.append(_side(slot, axis, step, m).reshape(-1)[cells])
            diag += _side((fluid | air).to(torch.uint8), axis, step, 0).reshape(-1)[cells]
    ext = torch.zeros(m + 1, dtype=torch.float64, device="cuda")

    def a_times(p):  # minus the operator: positive definite
        ext[:m] = p
        q = diag * p
        for s in nbr:
            q -= ext.index_select(0, s)
        return q

    b = -rhs.reshape(-1)[cells]
    x, r = torch.zeros_like(b), b.clone()
    p, rr = r.clone(), torch.dot(r, r)
    stop = float(rr) * tol * tol
    for it in range(limit):
        q = a_times(p)
        alpha = rr / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        new = torch.dot(r, r)
        p.mul_(new / rr).add_(r)
        rr = new
        if it % 32 == 31 and float(rr) <= stop:
            break
    out = torch.zeros(fluid.numel(), dtype=torch.float64, device="cuda")
    out[cells] = x
    return out.view(shape)


def _exact_project(case, seed):
    shape = _shape(case)
    phi, prims = _layout(case, seed)
    faces, rigid = [a.double() for a in _velocity(case, seed)], [a.double() for a in _rigid(case)]
    solid = _prim_solid(prims, shape)
    air = (phi > 0) & ~solid
    fluid = ~(solid | air)
    div = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for axis in range(3):
        f, r, n = faces[axis], rigid[axis], shape[axis]
        for step, sign in ((-1, -1.0), (1, 1.0)):
            at = 0 if step < 0 else 1
            flux = torch.where(_side(solid, axis, step, False), r.narrow(axis, at, n), f.narrow(axis, at, n)).clone()
            flux.select(axis, 0 if step < 0 else n - 1).zero_()  # the domain's own walls
            div += sign * flux
    x = _poisson_cg(fluid, air, torch.where(fluid, div, torch.zeros_like(div)))
    out = {"tag": None, "p": x / shape[0]}
    for axis, name in enumerate("uvw"):
        f, r, n = faces[axis], rigid[axis], shape[axis]
        lo = lambda t: t.narrow(axis, 0, n - 1)
        hi = lambda t: t.narrow(axis, 1, n - 1)
        inner = torch.where(lo(solid) | hi(solid), hi(r), torch.where(lo(fluid) | hi(fluid), hi(f) - (hi(x) - lo(x)),
                                                                      torch.zeros_like(lo(x))))
        new = torch.zeros_like(f)
        new.narrow(axis, 1, n - 1).copy_(inner)
        out[name] = new
    return out


def _at(q, a, b, c):
    nx, ny, nz = q.shape
    idx = (a.clamp(0, nx - 1) * ny + b.clamp(0, ny - 1)) * nz + c.clamp(0, nz - 1)
    return q.reshape(-1)[idx]


def _floor_fract(x):
    f = torch.floor(x)
    return f.long(), x - f


def _trilinear(q, p):
    (a, fa), (b, fb), (c, fc) = (_floor_fract(x) for x in p)
    lerp = lambda s, t, f: s * (1 - f) + t * f
    plane = lambda dc: lerp(lerp(_at(q, a, b, c + dc), _at(q, a + 1, b, c + dc), fa),
                            lerp(_at(q, a, b + 1, c + dc), _at(q, a + 1, b + 1, c + dc), fa), fb)
    return lerp(plane(0), plane(1), fc)


def _backtrace(faces, p, dt, h):
    off = ((0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0))
    vel = lambda x: [_trilinear(f, [c - o for c, o in zip(x, off[d])]) for d, f in enumerate(faces)]
    v1 = vel(p)
    v2 = vel([x - 0.5 * dt / h * v for x, v in zip(p, v1)])
    v3 = vel([x - 0.75 * dt / h * v for x, v in zip(p, v2)])
    return [x - dt / h * (2 / 9 * a + 1 / 3 * b + 4 / 9 * c) for x, a, b, c in zip(p, v1, v2, v3)]


def _cubic(v, s):
    return (v[0] * (-s / 3 + s * s / 2 - s ** 3 / 6) + v[1] * (1 - s * s + (s ** 3 - s) / 2)
            + v[2] * (s + (s * s - s ** 3) / 2) + v[3] * ((s ** 3 - s) / 6))


def _tricubic(q, p):
    (a, fa), (b, fb), (c, fc) = (_floor_fract(x) for x in p)
    return _cubic([_cubic([_cubic([_at(q, a + l, b + m, c + n) for l in (-1, 0, 1, 2)], fa) for m in (-1, 0, 1, 2)], fb)
                   for n in (-1, 0, 1, 2)], fc)


def _points(shape, st):
    c = [torch.arange(n, dtype=torch.float64, device="cuda") + o for n, o in zip(shape, st)]
    return [t.expand(shape).reshape(-1) for t in (c[0][:, None, None], c[1][None, :, None], c[2][None, None, :])]


def _advect_one(faces, q, st, dt, h):
    out = []
    for p in zip(*(t.split(1 << 22) for t in _points(q.shape, st))):
        i = sum(o.numel() for o in out)
        here = q.reshape(-1)[i:i + p[0].numel()]
        foot = _backtrace(faces, list(p), dt, h)
        ahead = _backtrace(faces, list(p), -dt, h)
        back = _tricubic(q, [x - o for x, o in zip(foot, st)])
        better = back + 0.5 * (here - _tricubic(q, [x - o for x, o in zip(ahead, st)]))
        a, b, c = (torch.floor(x / h - o).clamp(-2.0 ** 31, 2.0 ** 31).long() for x, o in zip(foot, st))
        near = torch.stack([_at(q, a + l, b + m, c + n) for l in (0, 1) for m in (0, 1) for n in (0, 1)])
        inside = (near.amin(0) < better) & (better < near.amax(0))
        out.append(torch.where(inside, better, back))
    return torch.cat(out).view(q.shape)


def _exact_advect(case, seed):
    shape = _shape(case)
    vel, phi = _advect_inputs(case, seed)
    faces, phi = [a.double() for a in vel], phi.double()
    h = float(np.float32(1.0 / shape[0]))
    dt = float(np.float32(K.DT))
    moved = []
    for p in zip(*(t.split(1 << 22) for t in _points(shape, (0.5, 0.5, 0.5)))):
        foot = _backtrace(faces, list(p), dt, h)
        inside = torch.stack([(0 <= x) & (x < n) for x, n in zip(foot, shape)]).all(0)
        moved.append(torch.where(inside, _tricubic(phi, [x - 0.5 for x in foot]), torch.full_like(foot[0], h)))
    stagger = ((0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0))
    out = {"phi": torch.cat(moved).view(shape)}
    for d, name in enumerate("uvw"):
        out[name] = _advect_one(faces, faces[d], stagger[d], dt, h)
    return out


def _exact_extrapolate(case, seed):
    shape = _shape(case)
    phi, _ = _layout(case, seed)
    out = {"tu": None, "tv": None, "tw": None}
    for d, q in enumerate(_velocity(case, seed)):
        unknown = torch.zeros(q.shape, dtype=torch.bool, device="cuda")
        unknown[:shape[0], :shape[1], :shape[2]] = phi >= 0
        known = (~unknown).double()
        pad = lambda t: torch.nn.functional.pad(t, (1, 1, 1, 1, 1, 1))
        vals, cnts = pad(q.double() * known), pad(known)
        total, count = torch.zeros_like(known), torch.zeros_like(known)
        for a in range(3):
            for b in range(3):
                for c in range(3):
                    at = (slice(a, a + q.shape[0]), slice(b, b + q.shape[1]), slice(c, c + q.shape[2]))
                    total += vals[at]
                    count += cnts[at]
        mean = torch.where(count > 0, total / count.clamp(min=1), torch.zeros_like(total))
        out["uvw"[d]] = torch.where(unknown, mean, q.double())
    return out


_SWEEPS = ((1, 1, -1), (-1, 1, -1), (-1, -1, -1), (1, -1, -1), (1, 1, 1), (-1, 1, 1), (-1, -1, 1), (1, -1, 1))


def _exact_redistance(case, seed):
    shape = _shape(case)
    phi = _redistance_input(case, seed).double()
    h = float(np.float32(1.0 / shape[0]))
    edge = torch.ones(shape, dtype=torch.bool, device="cuda")
    edge[1:-1, 1:-1, 1:-1] = False
    # the distance to the surface where a neighbour lies on its other side, else +-2
    around = [(axis, step) for axis in range(3) for step in (-1, 1)]
    near_pos, near_neg = torch.zeros_like(edge), torch.zeros_like(edge)
    m_pos, m_neg = torch.full_like(phi, math.inf), torch.full_like(phi, math.inf)
    for n, (axis, step) in enumerate(around):
        q = _side(phi, axis, step, 0.5 * h)
        part = 1 - torch.maximum(phi, q) / (phi - q).abs()
        part = torch.where((phi < 0) & (q < 0), torch.ones_like(phi), torch.where((phi >= 0) & (q >= 0),
                                                                                torch.zeros_like(phi), part))
        near_pos |= (q < 0) & ~edge if n == 0 else q < 0
        near_neg |= (q > 0) & ~edge if n == 0 else q > 0
        m_pos, m_neg = torch.minimum(m_pos, 1 - part), torch.minimum(m_neg, part)
    keep = edge if not case["boundary"] else torch.zeros_like(edge)
    two = torch.full_like(phi, 2.0)
    out = torch.where((phi > 0) & ~keep, torch.where(near_pos, h * m_pos, two), phi)
    phi = torch.where((phi < 0) & ~keep, torch.where(near_neg, -h * m_neg, -two), out)
    i, j, k = torch.meshgrid(*(torch.arange(n, device="cuda") for n in shape), indexing="ij")
    parity = (i + j + k) % 2
    del i, j, k
    for _ in range(2):
        for inc in _SWEEPS:
            turned = sum(n - 1 for n, s in zip(shape, inc) if s < 0)
            for odd in (0, 1):
                a = [[_side(phi, axis, s, 0.0) for s in (-1, 1)] for axis in range(3)]
                before = _side(phi, 0, -inc[0], 0.0)
                neg = before < 0
                sgn = torch.where(neg, -1.0, 1.0).double()
                m = [torch.where(neg, -torch.maximum(s, t), torch.minimum(s, t)) for s, t in a]
                lo = torch.minimum(torch.minimum(m[0], m[1]), m[2])
                hi = torch.maximum(torch.maximum(m[0], m[1]), m[2])
                mid = m[0] + m[1] + m[2] - lo - hi
                d = lo + h
                d2 = 0.5 * (lo + mid + torch.sqrt((2 * h * h - (lo - mid) ** 2).clamp(min=0)))
                t = (lo + mid + hi) ** 2 - 3 * (lo * lo + mid * mid + hi * hi - h * h)
                d3 = (lo + mid + hi + torch.sqrt(t.clamp(min=0))) / 3
                d = torch.where(d > mid, torch.where(d2 > hi, d3, d2), d)
                new = sgn * torch.minimum(d, phi.abs())
                phi = torch.where((parity == (odd + turned) % 2) & (phi.abs() > h) & ~edge, new, phi)
    return phi


def _exact_conv(case, seed):
    s = _conv_inputs(case, seed)
    co = case["cout"]
    dy = s["dy"].double()

    def taps(t):
        pad = torch.nn.functional.pad(t, (0, 0, 1, 1, 1, 1, 1, 1))
        n = t.shape
        for k in range(27):
            a, b, c = k // 9, k // 3 % 3, k % 3
            yield pad[:, a:a + n[1], b:b + n[2], c:c + n[3]].reshape(-1, n[4])

    out = {"db": dy.reshape(-1, co).sum(0)}
    y = s["b"].double().expand(dy.numel() // co, co).clone()
    for c in ("0", "1"):
        if s["x" + c] is None:
            continue
        x, w = s["x" + c].double(), s["w" + c].double()
        dw = torch.empty_like(w)
        for k, t in enumerate(taps(x)):
            y += t @ w[k].T
            dw[k] = dy.reshape(-1, co).T @ t
        dx = torch.zeros(x.numel() // x.shape[-1], x.shape[-1], dtype=torch.float64, device="cuda")
        for k, t in enumerate(taps(dy)):
            dx += t @ w[26 - k]
        out.update({"dw" + c: dw, "dx" + c: dx.view(x.shape)})
    out["y"] = y.relu().view(dy.shape)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        return _exact_project(case, seed)
    return {"advect": _exact_advect, "extrapolate": _exact_extrapolate, "redistance": _exact_redistance,
            "conv": _exact_conv}[kind](case, seed)
