"""The performance cases: what a program that simulates water with this package has it do.

A FLIP step hands its basin to ``redistance!``/``classify!``/``filltrapped!``, ``project!`` and
``extrapolate!``; a design loop adds the adjoint and rollouts; a data generator projects batches;
the sparse basin has a ``project!`` of its own. The cases call those entry points over the sizes
of the tests and benchmark configurations (32^3 to 384 x 384 x 256, ragged edges among them; 4 to
2948 fine blocks), in the precisions, loop forms and tolerances that they use.

Inputs are made on the GPU from the seed alone, with the distributions of ``mpp.scene`` and
``mpp.sparse_scene``: a cylindrical basin, a surface with gentle waves, uniform face velocities
with a Rankine vortex, walled faces zero. ``project!`` works in place, so a pass first puts the
velocities and the warm start back, as a program that replays a state does.

``exact`` gives the same outputs in 64 bits by plain torch: the operators assembled as CSR
matrices and solved by Jacobi-preconditioned conjugate gradients to 1e-12.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "maelstrom.jl_b200"))

import mpp  # noqa: E402
from mpp import adjoint, scene  # noqa: E402
from mpp import sparse as msp  # noqa: E402
from mpp.batch import Batch  # noqa: E402
from mpp.rollout import Rollout  # noqa: E402
from mpp.sparse_scene import SparseGrid  # noqa: E402

SOLID, LIQUID, AIR = scene.SOLID, scene.LIQUID, scene.AIR
DT = 1.0 / 48.0  # the reference's frame step
RECOVER = 0.5
LOSS = 1.0005  # volume0 over the volume: a basin that has lost a little water, so gamma is not zero
BCELLS, BFACES = 4096, 17 * 256

# What a program's handle keeps when it has autotuned the 16-bit form at the benchmark's 256^3
# (sweeps on the fine level, on the coarser ones, on the coarsest).
TUNED = (5, 6, 10)


# ---- the cases -------------------------------------------------------------------------------

def _project(name, n, precision="fp32", graph=False, tol=1e-4, tuned=False, fallback=False, warm=False, vortex=0.0,
             depression=False):
    c = dict(kind="project", n1=n[0], n2=n[1], n3=n[2], precision=precision, graph=graph, tol=tol, tuned=tuned,
             fallback=fallback, warm=warm, vortex=vortex, depression=depression)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest: a preview basin at every default (host-driven loop, tol 1e-4, cold start)
        _project("project_32_default", (32, 32, 32)),
        # the plain configuration: 64^3, Float32, 1e-6
        _project("project_64_fp32", (64, 64, 64), tol=1e-6),
        # a basin of odd proportions inside a running simulation: graph, warm start, default tol
        _project("project_ragged_bf16", (176, 144, 112), precision="bf16", graph=True, warm=True),
        # the headline: 256^3 with a vortex, mixed precision, one graph launch, autotuned sweeps
        _project("project_256_fp16", (256, 256, 256), precision="fp16", graph=True, tol=1e-6, tuned=True, vortex=225.0),
        # the largest: the 384 x 384 x 256 whirlpool, mixed precision with the FGMRES fallback armed
        _project("project_384_fp16", (384, 384, 256), precision="fp16", graph=True, tol=1e-6, fallback=True,
                 vortex=225.0, depression=True),
        # many basins at once: 48 of mixed sizes as one graph launch, Float32
        dict(name="batch_48_fp32", kind="batch", count=48, precision="fp32", tol=1e-6),
        # a design loop's step: project! and its pullback under autograd
        dict(name="adjoint_128_fp32", kind="adjoint", n1=128, n2=128, n3=128, precision="fp32", graph=True, tol=1e-6),
        # a rollout of advect + project, forward and reverse
        dict(name="rollout_96_fp32", kind="rollout", n1=96, n2=96, n3=96, precision="fp32", graph=True, tol=1e-6, steps=4),
        # the level-set phase of a step before the projection
        dict(name="levelset_256", kind="levelset", n1=256, n2=256, n3=256, sweeps=7),
        # the velocity extrapolation right after the projection, step!'s six layers
        dict(name="extrapolate_256", kind="extrapolate", n1=256, n2=256, n3=256, layers=6),
        # a small sparse basin at the defaults
        dict(name="sparse_small", kind="sparse", b1=6, b2=6, b3=4, tol=1e-4, graph=False, fallback=False, rings=0),
        # the sparse whirlpool: 32 x 32 x 16 blocks
        dict(name="sparse_whirlpool", kind="sparse", b1=32, b2=32, b3=16, tol=1e-4, graph=False, fallback=False, rings=1),
    ]


def _edges(rng, lo, hi, most):
    """Three edges between lo and hi (spread over their logarithm, unequal), as FlipGrid pads them."""
    while True:
        base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        n = [min(hi, max(lo, base * math.exp(rng.uniform(-0.35, 0.35)))) for _ in range(3)]
        if n[0] * n[1] * n[2] > most:
            continue
        m = 2
        while True:
            e = [max(2 * m, int(round(x / m)) * m) for x in n]
            if e[0] * e[1] * e[2] // m ** 3 <= 1024:
                break
            m *= 2
        if e[0] * e[1] * e[2] <= most:
            return e


def draw(rng):
    kind = rng.choice(["project"] * 5 + ["batch", "adjoint", "rollout", "levelset", "extrapolate", "sparse", "sparse"])
    tol = rng.choice([1e-4, 1e-6])
    precision = rng.choice(["fp32", "fp16", "bf16"])
    if kind == "project":
        n = _edges(rng, 24, 352, 384 * 384 * 256)
        return _project(None, n, precision=precision, graph=rng.random() < 0.6, tol=tol, tuned=precision != "fp32" and rng.random() < 0.5,
                        fallback=rng.random() < 0.25, warm=rng.random() < 0.3, vortex=rng.choice([0.0, 225.0]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 40), precision=precision, tol=tol)
    if kind == "sparse":
        base = math.exp(rng.uniform(math.log(3), math.log(28)))
        b = [max(3, int(base * rng.uniform(0.7, 1.14))) for _ in range(3)]
        return dict(kind="sparse", b1=b[0], b2=b[1], b3=max(3, min(16, b[2])), tol=rng.choice([1e-4, 1e-5]), graph=rng.random() < 0.5,
                    fallback=rng.random() < 0.2, rings=rng.choice([0, 1]))
    n = _edges(rng, 32, {"adjoint": 192, "rollout": 112}.get(kind, 288), {"adjoint": 160 ** 3, "rollout": 96 ** 3}.get(kind, 256 ** 3))
    c = dict(kind=kind, n1=n[0], n2=n[1], n3=n[2])
    if kind == "adjoint":
        c.update(precision=precision, graph=rng.random() < 0.7, tol=1e-6)
    elif kind == "rollout":
        c.update(precision="fp32", graph=True, tol=1e-6, steps=rng.randint(2, 4))
    elif kind == "levelset":
        c.update(sweeps=rng.choice([6, 7, 8]))
    else:
        c.update(layers=rng.choice([4, 6]))
    return c


# ---- inputs ----------------------------------------------------------------------------------

def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _uniform(g, shape, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float32) * (hi - lo) + lo


def _centres(lo, dx, count, offset=0.5):
    i = torch.arange(count, dtype=torch.float32, device="cuda")
    return torch.tensor(lo, dtype=torch.float32, device="cuda") + (i + offset) * torch.tensor(dx, dtype=torch.float32, device="cuda")


def _solid_cells(grid):
    x, y, z = (_centres(grid.lo[a], grid.dx, grid.n[a]) for a in range(3))
    r2 = (x * x)[None, :] + (y * y)[:, None]
    return (r2 > torch.tensor(grid.radius, dtype=torch.float32, device="cuda") ** 2)[None] | (z < grid.floor)[:, None, None]


def _walled(solid, axis):
    """The walled faces along axis (0: x): the box's edge, or a SOLID cell on either side."""
    d = 2 - axis
    shape = list(solid.shape)
    shape[d] += 1
    out = torch.ones(shape, dtype=torch.bool, device="cuda")
    n = solid.shape[d]
    out.narrow(d, 1, n - 1).copy_(solid.narrow(d, 0, n - 1) | solid.narrow(d, 1, n - 1))
    return out


def _dense(n, seed, salt=0, vortex=0.0, depression=False, wall=0.45, height=0.6, core=2.5):
    """A cylindrical basin's grid and its arrays shaped (nz, ny, nx): mpp.scene.box_basin's
    distributions, the surface raised and lowered by waves of a few centimetres."""
    g, dx = _gen(seed, salt), 0.05
    n = tuple(int(v) for v in n)
    f32 = lambda v: float(np.float32(v))
    grid = scene.Grid(lo=(f32(-n[0] * dx / 2), f32(-n[1] * dx / 2), 0.0), dx=f32(dx), n=n, radius=f32(wall * min(n[0], n[1]) * dx),
                      floor=0.0, levels=scene.levels_for(n))
    solid = _solid_cells(grid)
    x, y, z = (_centres(grid.lo[a], grid.dx, n[a]) for a in range(3))
    ph = _uniform(g, (4,), 0.0, 6.28)
    surf = height * n[2] * dx + 0.04 * torch.sin(2.1 * x + ph[0])[None, :] * torch.sin(1.7 * y + ph[1])[:, None]
    if depression:
        r2 = (x * x)[None, :] + (y * y)[:, None]
        k = vortex * vortex / (8.0 * math.pi ** 2 * 9.81)
        surf = surf + torch.where(r2 < core * core, -2 * k / core ** 2 + k * r2 / core ** 4, -k / r2.clamp(min=1e-9))
    phi = (z[:, None, None] - surf[None]).contiguous()
    types = torch.where(solid, SOLID, torch.where(phi < 0, LIQUID, AIR)).to(torch.uint8)
    faces = []
    for axis in range(3):
        shape = grid.face_shape(axis)
        f = _uniform(g, shape[::-1])
        if vortex and axis < 2:
            fx, fy = (_centres(grid.lo[a], grid.dx, shape[a], 0.0 if a == axis else 0.5) for a in range(2))
            r = torch.sqrt((fx * fx)[None, :] + (fy * fy)[:, None]).clamp(min=1e-6)
            ut = torch.where(r < core, vortex * r / (2 * math.pi * core ** 2), vortex / (2 * math.pi * r))
            f = f + (ut * (-fy[:, None] if axis == 0 else fx[None, :]) / r)[None]
        f[_walled(solid, axis)] = 0.0
        faces.append(f.contiguous())
    return dict(grid=grid, solid=solid, types=types, phi=phi, faces=faces, gen=g)


def _basin(d, warm=False, **kw):
    """The FlipBasin of _dense's arrays, its context, and the pass's starting values."""
    grid, flat = d["grid"], lambda t: t.reshape(-1)
    P0 = torch.zeros(grid.ncells, dtype=torch.float32, device="cuda")
    if warm:  # about the pressure of the step before: hydrostatic, off by a tenth
        P0 = flat(torch.where(d["types"] == LIQUID, -d["phi"] * (0.2 + 0.02 * _uniform(d["gen"], d["phi"].shape)), 0.0)).contiguous()
    faces = [flat(f) for f in d["faces"]]
    s = mpp.FlipBasin(grid=grid, u=faces[0].clone(), v=faces[1].clone(), w=faces[2].clone(),
                      fu=torch.zeros_like(faces[0], dtype=torch.uint8), fv=torch.zeros_like(faces[1], dtype=torch.uint8),
                      fw=torch.zeros_like(faces[2], dtype=torch.uint8), P=P0.clone(), types=flat(d["types"]), phi=flat(d["phi"]),
                      volume0=0.0, iterations=[], projector=mpp.Projector(grid, **kw))
    s.volume0 = s.projector.volume(s.phi) * LOSS
    return s, faces, P0


def _options(c):
    kw = dict(tol=c["tol"], maxiter=200, precision=c["precision"], graph=c["graph"])
    if c.get("fallback"):
        kw["fallback"] = True
    return kw


def _dense_of(c, seed):
    return _dense((c["n1"], c["n2"], c["n3"]), seed, vortex=c.get("vortex", 0.0), depression=c.get("depression", False),
                  height=0.7 if c.get("depression") else 0.6)


def _batch_members(c, seed):
    """The batched workload's members: edge, depth and wall drawn per basin, velocities uniform."""
    rng = np.random.default_rng(1002 + 7 * c["count"])  # the sizes are the case's, the water the seed's
    out = []
    for b in range(c["count"]):
        edge = int(rng.choice(scene.BATCH_EDGES))
        height, wall = 0.3 + 0.5 * rng.random(), 0.35 + 0.13 * rng.random()
        out.append(_dense((edge,) * 3, seed, salt=b + 1, wall=float(wall), height=float(height)))
    return out


def _levelset_inputs(c, seed):
    """The benchmark's level set: wavy, noisy, 2% of the water made sealed air pockets."""
    d = _dense((c["n1"], c["n2"], c["n3"]), seed)
    dx, g = d["grid"].dx, d["gen"]
    phi = d["phi"] + 0.3 * dx * torch.sin(0.2 * torch.arange(c["n1"], device="cuda"))[None, None, :]
    phi = phi + _uniform(g, phi.shape, -0.2 * dx, 0.2 * dx)
    pocket = (d["types"] == LIQUID) & (torch.rand(phi.shape, generator=g, device="cuda") < 0.02)
    d["phi"] = torch.where(pocket, phi.abs(), phi).contiguous()
    return d


def _flags(types, axis):
    """The valid-face flags project! leaves: a LIQUID side, no SOLID side, inside the box."""
    d = 2 - axis
    n = types.shape[d]
    a, b = types.narrow(d, 0, n - 1), types.narrow(d, 1, n - 1)
    ok = (a != SOLID) & (b != SOLID) & ((a == LIQUID) | (b == LIQUID))
    shape = list(types.shape)
    shape[d] += 1
    out = torch.zeros(shape, dtype=torch.uint8, device="cuda")
    out.narrow(d, 1, n - 1).copy_(ok)
    return out


def _up(a, r):
    for d in range(3):
        a = a.repeat_interleave(r, dim=d)
    return a


def _sparse_scene(c, seed):
    """A SparseBasin's arrays: mpp.sparse_scene.sparse_basin's whirlpool funnel with waves of a few
    centimetres; the blocks are the case's, the velocities and the warm start the seed's. Every fifth
    slot is free where the basin has no extra ring."""
    g = _gen(seed)
    nb = (c["b1"], c["b2"], c["b3"])
    nc, nf = tuple(4 * b for b in nb), tuple(16 * b for b in nb)
    f32 = lambda v: float(np.float32(v))
    dx, cdx = f32(0.05), f32(4 * np.float32(0.05))
    lo = (f32(-nf[0] * dx / 2), f32(-nf[1] * dx / 2), 0.0)
    floor_z, radius = cdx, f32(0.45 * min(nf[0], nf[1]) * dx)
    h0 = floor_z + 0.55 * (nf[2] * dx - floor_z)
    depth, width = (0.45 if c["rings"] else 0.25) * (h0 - floor_z), 0.3 * radius
    grid = SparseGrid(lo=lo, dx=dx, nb=nb, radius=radius, floor_z=floor_z)

    def fields(h, n):
        x, y, z = (_centres(lo[a], h, n[a]) for a in range(3))
        r2 = (x * x)[None, :] + (y * y)[:, None]
        surf = h0 - depth * torch.exp(-r2 / width ** 2) + 0.03 * torch.sin(1.3 * x + 0.4)[None, :] * torch.sin(1.1 * y + 1.9)[:, None]
        return (z[:, None, None] - surf[None]).contiguous(), (r2 > radius * radius)[None] | (z < floor_z)[:, None, None]

    phic, csolid = fields(cdx, nc)
    near, sign = (phic.abs() < 1.5 * cdx), phic < 0
    for d in range(3):
        n = sign.shape[d]
        flip = sign.narrow(d, 0, n - 1) != sign.narrow(d, 1, n - 1)
        near.narrow(d, 0, n - 1).logical_or_(flip)
        near.narrow(d, 1, n - 1).logical_or_(flip)
    near &= ~csolid
    marks = near.reshape(nb[2], 4, nb[1], 4, nb[0], 4).any(5).any(3).any(1)
    for _ in range(c["rings"]):
        m = marks.clone()
        for d in range(3):
            n = marks.shape[d]
            m.narrow(d, 0, n - 1).logical_or_(marks.narrow(d, 1, n - 1))
            m.narrow(d, 1, n - 1).logical_or_(marks.narrow(d, 0, n - 1))
        marks = m
    want = torch.nonzero(marks.reshape(-1)).reshape(-1)
    order = torch.arange(want.numel(), device="cuda")
    slots = order + (0 if c["rings"] else order // 4)  # a slot released by a refinement after every fourth
    nslots = int(slots[-1]) + 1
    block = torch.full((nslots,), -1, dtype=torch.int64, device="cuda")
    block[slots] = want
    slot = torch.zeros(nb[0] * nb[1] * nb[2], dtype=torch.int32, device="cuda")
    slot[want] = (slots + 1).to(torch.int32)
    used = block >= 0
    at = torch.stack([block % nb[0], (block // nb[0]) % nb[1], block // (nb[0] * nb[1])], 1)
    where = torch.where(used[:, None], at, -1).to(torch.int32).contiguous()
    t = dict(grid=grid, slot=slot, where=where, nslots=nslots, nb=nb, nc=nc, nf=nf, used=torch.nonzero(used).reshape(-1), gen=g)
    phif, fsolid = fields(dx, nf)
    typf = torch.where(fsolid, SOLID, torch.where(phif < 0, LIQUID, AIR)).to(torch.uint8)
    cells = _cell_index(t)
    for name, src in (("phif", phif), ("tf", typf)):
        pool = torch.zeros(nslots, BCELLS, dtype=src.dtype, device="cuda")
        pool[t["used"]] = src.reshape(-1)[cells]
        t[name] = pool.reshape(-1)
    # under fine blocks: AIR if any of a coarse cell's 64 is, else LIQUID if any is; the mean level set
    tc = torch.where(csolid, SOLID, torch.where(phic < 0, LIQUID, AIR)).to(torch.uint8)
    by4 = lambda a: a.reshape(nc[2], 4, nc[1], 4, nc[0], 4)
    air, liq = (by4(typf == v).any(5).any(3).any(1) for v in (AIR, LIQUID))
    cov = _up(marks, 4)
    t["tc"] = torch.where(cov, torch.where(air, AIR, torch.where(liq, LIQUID, SOLID)).to(torch.uint8), tc).reshape(-1)
    t["phic"] = torch.where(cov, by4(phif).mean((1, 3, 5)), phic).reshape(-1)
    del phif, fsolid, typf
    for axis in range(3):
        def flow(h, n, noise):
            shape = [n[a] + (a == axis) for a in range(3)]
            x, y = (_centres(lo[a], h, shape[a], 0.0 if a == axis else 0.5) for a in range(2))
            r2 = (x * x)[None, :] + (y * y)[:, None] + 1e-6
            s = 2.0 * width * torch.exp(-r2 / (2 * width ** 2)) / torch.sqrt(r2)
            base = (-s * y[:, None], s * x[None, :], 0 * s)[axis]
            return base[None] + _uniform(g, tuple(shape[::-1]), -noise, noise)

        fine, coarse = flow(dx, nf, 0.5), flow(cdx, nc, 0.5)
        pool = torch.zeros(nslots, BFACES, dtype=torch.float32, device="cuda")
        pool[t["used"]] = fine.reshape(-1)[_face_index(t, axis)]
        t["uvw"[axis] + "f"] = pool.reshape(-1)
        t["uvw"[axis] + "c"] = torch.where(_held(t, axis), _face_means(fine, axis), coarse).reshape(-1)
        t["f" + "uvw"[axis] + "f"] = torch.zeros(nslots * BFACES, dtype=torch.uint8, device="cuda")
        t["f" + "uvw"[axis] + "c"] = torch.zeros(coarse.numel(), dtype=torch.uint8, device="cuda")
    for f in ("f", "c"):  # a warm start on the water cells
        liquid = t["t" + f] == LIQUID
        t["P" + f] = torch.where(liquid, _uniform(g, liquid.shape, 0.0, 0.01), 0.0)
    return t


def _cell_index(t):
    """Each used slot's 4096 cells as indices of the box's fine cells."""
    c = torch.arange(BCELLS, device="cuda")
    w = t["where"][t["used"]].long()[:, :, None] * 16
    I, J, K = w[:, 0] + (c & 15), w[:, 1] + ((c >> 4) & 15), w[:, 2] + (c >> 8)
    return I + t["nf"][0] * (J + t["nf"][1] * K)


def _face_local(axis):
    f = torch.arange(BFACES, device="cuda")
    e = [16 + (a == axis) for a in range(3)]
    return f % e[0], (f // e[0]) % e[1], f // (e[0] * e[1])


def _face_index(t, axis, dims=None, back=0, pad=0):
    """Each used slot's faces along axis as indices of the box's fine faces (or of an array of
    other dims, from a face shifted back along the axis, with a border of pad)."""
    n = dims or [t["nf"][a] + (a == axis) for a in range(3)]
    w = t["where"][t["used"]].long()[:, :, None] * 16
    I, J, K = (w[:, a] + l + pad - back * (a == axis) for a, l in enumerate(_face_local(axis)))
    return I + n[0] * (J + n[1] * K)


def _covered(t):
    return _up((t["slot"] > 0).reshape(t["nb"][::-1]), 4)


def _held(t, axis):
    """Coarse faces along axis whose 16 fine faces a fine block holds."""
    cov, d = _covered(t), 2 - axis
    shape = list(cov.shape)
    shape[d] += 1
    out = torch.zeros(shape, dtype=torch.bool, device="cuda")
    n = cov.shape[d]
    out.narrow(d, 0, n).logical_or_(cov)
    out.narrow(d, 1, n).logical_or_(cov)
    return out


def _face_means(fine, axis):
    """The mean of the 4 x 4 fine faces of every coarse face along axis."""
    a = fine[:, :, ::4] if axis == 0 else (fine[:, ::4] if axis == 1 else fine[::4])
    for d in range(3):
        if d != 2 - axis:
            a = a.unflatten(d, (a.shape[d] // 4, 4)).mean(d + 1)
    return a


# ---- prepare and run -------------------------------------------------------------------------

SPARSE_STATE = ("uf", "uc", "vf", "vc", "wf", "wc", "Pf", "Pc")


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "project":
        s, faces, P0 = _basin(_dense_of(c, seed), warm=c["warm"], **_options(c))
        if c["tuned"]:
            s.projector.set(sweeps=TUNED[0], sweeps_coarse=TUNED[1], coarse=TUNED[2])
        return dict(kind=k, s=s, faces=faces, P0=P0)
    if k == "batch":
        basins = []
        for d in _batch_members(c, seed):
            h = lambda t: t.reshape(-1).cpu().numpy()
            basins.append(scene.Basin(grid=d["grid"], types=h(d["types"]), phi=h(d["phi"]), u=h(d["faces"][0]), v=h(d["faces"][1]),
                                      w=h(d["faces"][2]), seed=int(seed)))
        b = Batch(basins, tol=c["tol"], maxiter=200, precision=c["precision"])
        b.volume0 = [v * LOSS for v in b.volume0]
        return dict(kind=k, b=b, init=[[a[n].clone() for n in "uvw"] for a in b.arrays])
    if k in ("adjoint", "rollout"):
        s, faces, _ = _basin(_dense_of(c, seed), **_options(c))
        g = _gen(seed, 77)
        target = [_uniform(g, f.shape) for f in faces]
        st = dict(kind=k, s=s, faces=faces, target=target)
        if k == "rollout":
            st["ro"] = Rollout(s, c["steps"], DT, RECOVER)
        else:
            st["faces"] = [f.requires_grad_(True) for f in faces]
        return st
    if k == "levelset":
        d = _levelset_inputs(c, seed)
        s, _, _ = _basin(d)
        return dict(kind=k, s=s, phi=d["phi"].reshape(-1).clone(), sweeps=c["sweeps"])
    if k == "extrapolate":
        d = _dense((c["n1"], c["n2"], c["n3"]), seed, vortex=225.0)
        s, _, _ = _basin(d)
        return dict(kind=k, s=s, flags=[_flags(d["types"], a).reshape(-1) for a in range(3)], layers=c["layers"])
    t = _sparse_scene(c, seed)
    kw = dict(tol=c["tol"], maxiter=200, graph=c["graph"])
    if c["fallback"]:
        kw.update(fallback=True, maxiter=240)
    s = msp.SparseBasin(t["grid"], t["slot"], t["where"], t["nslots"], {f: t[f] for f in msp.SparseBasin.FIELDS}, opts=kw)
    s.volume0 = msp.volume(s) * LOSS
    return dict(kind=k, s=s, init={f: t[f].clone() for f in SPARSE_STATE})


def run(state):
    k = state["kind"]
    if k == "batch":
        b = state["b"]
        for a, init in zip(b.arrays, state["init"]):
            for n, x in zip("uvw", init):
                a[n].copy_(x)
            a["P"].zero_()
        b.project(DT, RECOVER)
        return [torch.cat([a[n] for a in b.arrays]) for n in ("u", "v", "w", "fu", "fv", "fw", "P")]
    s = state["s"]
    if k == "project":
        for a, x in zip((s.u, s.v, s.w, s.P), state["faces"] + [state["P0"]]):
            a.copy_(x)
        mpp.project(s, DT, RECOVER)
        return [s.u, s.v, s.w, s.P, s.fu, s.fv, s.fw]
    if k == "adjoint":
        s.P.zero_()
        if getattr(s, "mu", None) is not None:
            s.mu.zero_()
        out = adjoint.project(*state["faces"], s, DT, RECOVER)
        loss = sum(0.5 * ((o - x) ** 2).sum() for o, x in zip(out, state["target"]))
        return [o.detach() for o in out] + list(torch.autograd.grad(loss, state["faces"]))
    if k == "rollout":
        ro = state["ro"]
        s.P.zero_()
        ro.mu.zero_()
        out = ro.forward(*state["faces"])
        grad = ro.backward(*(o - x for o, x in zip(out, state["target"])))
        return list(out) + list(grad)
    if k == "levelset":
        s.phi.copy_(state["phi"])
        mpp.redistance(s, state["sweeps"])
        mpp.classify(s)
        mpp.filltrapped(s)
        return [s.phi, s.types]
    if k == "extrapolate":  # the flagged values stay, the rest is rewritten: the flags are the state
        for f, x in zip((s.fu, s.fv, s.fw), state["flags"]):
            f.copy_(x)
        mpp.extrapolate(s, state["layers"])
        return [s.u, s.v, s.w, s.fu, s.fv, s.fw]
    for f, x in state["init"].items():
        getattr(s, f).copy_(x)
    msp.project(s, DT, RECOVER)
    return [getattr(s, f) for f in SPARSE_STATE + ("fuf", "fuc", "fvf", "fvc", "fwf", "fwc")]


# ---- the work and the tolerances --------------------------------------------------------------

def work(case):
    c, k = case, case["kind"]
    if k == "batch":
        rng = np.random.default_rng(1002 + 7 * c["count"])
        cells = 0
        for _ in range(c["count"]):
            cells += int(rng.choice(scene.BATCH_EDGES)) ** 3
            rng.random(), rng.random()
    elif k == "sparse":
        # a fine cell of the band: about 2.4 (sparse: 1.2) block layers of the box's footprint; coarse cells dense
        cells = int(c["b1"] * c["b2"] * (2.9 if c["rings"] else 1.3)) * BCELLS + 64 * c["b1"] * c["b2"] * c["b3"]
    else:
        cells = c["n1"] * c["n2"] * c["n3"]
    # a projection: u, v, w read and written (24), P read and written (8), phi and classes read (5),
    # flags written (3); its sums, at the least one operator and one preconditioner pass (40)
    per = {"project": (40, 60), "batch": (40, 60), "sparse": (40, 60), "adjoint": (40 + 24 + 24 + 13, 130),
           "levelset": (4 + 4 + 1, 20 * c.get("sweeps", 7)), "extrapolate": (3 * (4 + 4 + 2), 6),
           "rollout": ((24 + 40) * 2 * c.get("steps", 1), 700 * c.get("steps", 1))}[k]
    return dict(bytes=float(cells * per[0]), flops=float(cells * per[1]))


def tolerance(case):
    """About four times the distance from ``exact`` measured on the package's own outputs."""
    c, k = case, case["kind"]
    if k in ("extrapolate", "levelset"):  # elementwise Float32, a few roundings a value (3e-8 measured)
        return {"rel": 1e-6, "max": 1e-4}
    if k == "rollout":  # a gradient through points that round to either side of a sample (3.3e-3)
        return {"rel": 1.3e-2, "max": 0.5}
    if k == "adjoint":  # the faces and their gradients, not the pressure (8e-6)
        return {"rel": 1e-4, "max": 1e-2}
    # a solve stops anywhere below its residual tolerance; the pressure is off by that residual times
    # the operator's conditioning (1.4e-4 at 1e-6, 2.5e-3 at 1e-4; sparse: 1.3e-2 at 1e-4)
    if k == "sparse":
        return {"rel": 3e-2 if c["tol"] > 2e-5 else 1e-2, "max": 0.5}
    return {"rel": 1e-2 if c["tol"] > 1e-5 else 6e-4, "max": 0.5 if c["tol"] > 1e-5 else 3e-2}


# ---- the same in 64 bits, by plain torch -------------------------------------------------------

def _cg(n, i, j, c, dirichlet, b, x0):
    """A x = b with A the symmetric couplings c between i and j and the extra diagonal."""
    diag = dirichlet.index_add(0, i, c).index_add(0, j, c)
    # a cell with no neighbour to flow to has no equation
    live = diag > 0
    diag = torch.where(live, diag, 1.0)
    idx = torch.arange(n, device="cuda")
    A = torch.sparse_coo_tensor(torch.stack([torch.cat([i, j, idx]), torch.cat([j, i, idx])]), torch.cat([-c, -c, diag]),
                                (n, n)).coalesce().to_sparse_csr()
    x = torch.where(live, x0, 0.0)
    r = torch.where(live, b, 0.0) - A @ x
    inv = 1.0 / diag
    z = inv * r
    p, rho, target = z.clone(), r @ z, 1e-12 * b.norm()
    for it in range(30000):
        if it % 50 == 0 and float(r.norm()) <= float(target):
            break
        q = A @ p
        a = rho / (p @ q)
        x.add_(a * p)
        r.sub_(a * q)
        z = inv * r
        new = r @ z
        p = z + (new / rho) * p
        rho = new
    return x


def _theta(a, b):
    return (a / (a - b)).clamp(float(np.float32(0.01)), 1.0)


def _pairs(types, axis):
    d = 2 - axis
    n = types.shape[d]
    return lambda a: (a.narrow(d, 0, n - 1), a.narrow(d, 1, n - 1))


class _Dense64:
    """project! of one basin in 64 bits."""

    def __init__(self, d):
        self.grid, self.types, self.phi = d["grid"], d["types"], d["phi"].double()
        self.dx = self.grid.dx
        self.liquid = self.types == LIQUID
        self.n = int(self.liquid.sum())
        self.ids = (torch.cumsum(self.liquid.reshape(-1).long(), 0) - 1).reshape(self.types.shape)
        self.air = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        ei, ej = [], []
        for axis in range(3):
            two = _pairs(self.types, axis)
            (ta, tb), (pa, pb), (ia, ib) = two(self.types), two(self.phi), two(self.ids)
            m = (ta == LIQUID) & (tb == LIQUID)
            ei.append(ia[m])
            ej.append(ib[m])
            for t0, t1, p0, p1, i0 in ((ta, tb, pa, pb, ia), (tb, ta, pb, pa, ib)):
                m = (t0 == LIQUID) & (t1 == AIR)
                self.air.index_add_(0, i0[m], 1.0 / _theta(p0[m], p1[m]))
        self.i, self.j = torch.cat(ei), torch.cat(ej)
        self.c = torch.ones(self.i.numel(), dtype=torch.float64, device="cuda")
        x = (0.5 - self.phi / self.dx).clamp(0.0, 1.0)
        self.loss = 0.0
        vol = float(torch.where(d["solid"], 0.0, x).sum())
        if vol > 0:
            self.loss = (LOSS * vol - vol) / (LOSS * vol)
        self.gamma = min(0.01 / DT, max(-0.01 / DT, self.loss / RECOVER))

    def solve(self, b):
        x = _cg(self.n, self.i, self.j, self.c, self.air, b[self.liquid], torch.zeros(self.n, dtype=torch.float64, device="cuda"))
        out = torch.zeros_like(self.phi)
        out[self.liquid] = x
        return out

    def div(self, f):
        u, v, w = f
        return u[:, :, 1:] - u[:, :, :-1] + v[:, 1:] - v[:, :-1] + w[1:] - w[:-1]

    def weights(self, axis):
        """Per inner face: whether it is open, and the two cells' weights in the gradient."""
        two = _pairs(self.types, axis)
        (ta, tb), (pa, pb) = two(self.types), two(self.phi)
        la, lb = ta == LIQUID, tb == LIQUID
        ok = (ta != SOLID) & (tb != SOLID) & (la | lb)
        both = la & lb
        wa = torch.where(both, 1.0, torch.where(la, 1.0 / _theta(pa, pb), 0.0))
        wb = torch.where(both, 1.0, torch.where(lb, 1.0 / _theta(pb, pa), 0.0))
        return ok, torch.where(ok & la, wa, 0.0), torch.where(ok & lb, wb, 0.0)

    def project(self, f):
        b = torch.where(self.liquid, -self.dx * self.div(f) + self.dx ** 2 * self.gamma, 0.0)
        P = self.solve(b)
        out = []
        for axis in range(3):
            _, wa, wb = self.weights(axis)
            pa, pb = _pairs(self.types, axis)(P)
            o = f[axis].clone()
            o.narrow(2 - axis, 1, pa.shape[2 - axis]).sub_((wb * pb - wa * pa) / self.dx)
            out.append(o)
        return out, P

    def vjp(self, g):
        """g + D^T mu with A mu = dx G^T g."""
        beta = torch.zeros_like(self.phi)
        for axis in range(3):
            d = 2 - axis
            _, wa, wb = self.weights(axis)
            inner = g[axis].narrow(d, 1, wa.shape[d])
            n = beta.shape[d]
            beta.narrow(d, 1, n - 1).add_(wb * inner)
            beta.narrow(d, 0, n - 1).sub_(wa * inner)
        mu = self.solve(torch.where(self.liquid, beta, 0.0))
        out = []
        for axis in range(3):
            d = 2 - axis
            o = g[axis].clone()
            n = mu.shape[d]
            o.narrow(d, 1, n).add_(mu)
            o.narrow(d, 0, n).sub_(mu)
            out.append(o)
        return out


class _Project64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, u, v, w, sys64):
        ctx.sys64 = sys64
        return tuple(sys64.project([u, v, w])[0])

    @staticmethod
    def backward(ctx, *g):
        return (*ctx.sys64.vjp(list(g)), None)


def _trilinear(A, p, lo, dx, off):
    """A (z, y, x) at the points p, its samples off cells from lo, clamped to the array. A point at
    rest sits on a sample, where the derivative has two sides: the cell, and whether the clamp holds
    the point, are what Float32 finds."""
    n = A.shape[::-1]
    i, f = [], []
    f32 = lambda v: torch.tensor(v, dtype=torch.float32, device="cuda")
    for a in range(3):
        x = (p[a] - lo[a]) / dx - off[a]
        q = (p[a].detach().float() - f32(lo[a])) / f32(dx) - f32(off[a])
        x = torch.where((q >= 0) & (q <= n[a] - 1), x, x.detach().clamp(0.0, n[a] - 1.0))
        k = q.clamp(0.0, n[a] - 1.0).long().clamp(max=n[a] - 2)
        i.append(k)
        f.append(x - k)
    flat, base = A.reshape(-1), i[0] + n[0] * (i[1] + n[1] * i[2])
    at = lambda x, y, z: flat.gather(0, base + x + n[0] * (y + n[1] * z))
    line = lambda y, z: at(0, y, z) * (1 - f[0]) + at(1, y, z) * f[0]
    plane = lambda z: line(0, z) * (1 - f[1]) + line(1, z) * f[1]
    return plane(0) * (1 - f[2]) + plane(1) * f[2]


def _advect64(grid, f):
    """advect! of the faces through themselves: RK2 sub-steps of at most a cell, then the sample."""
    dx, lo = grid.dx, grid.lo
    off = [[0.0 if a == c else 0.5 for a in range(3)] for c in range(3)]
    vel = lambda p: [_trilinear(f[c], p, lo, dx, off[c]) for c in range(3)]
    out = []
    for c in range(3):
        shape = f[c].shape
        # the nodes where Float32 places them, so that a point at rest is on its side of its sample
        zyx = torch.meshgrid(*(_centres(lo[2 - a], dx, shape[a], off[c][2 - a]).double() for a in range(3)), indexing="ij")
        p = [zyx[2 - a].reshape(-1) for a in range(3)]
        speed = torch.sqrt(sum(v * v for v in vel(p))).detach()
        m = torch.ceil(speed * DT / dx).clamp(1, 32)
        h = DT / m
        for s in range(int(m.max())):
            v1 = vel(p)
            v2 = vel([x - 0.5 * h * v for x, v in zip(p, v1)])
            on = s < m
            p = [torch.where(on, x - h * v, x) for x, v in zip(p, v2)]
        out.append(_trilinear(f[c], p, lo, dx, off[c]).reshape(shape))
    return out


def _redistance64(d, sweeps):
    grid, solid = d["grid"], d["solid"]
    h = grid.dx
    top = (sweeps + 1) * h
    phi = d["phi"].double()

    def around(a, fill):
        p = torch.full([s + 2 for s in a.shape], fill, dtype=a.dtype, device="cuda")
        p[1:-1, 1:-1, 1:-1] = a
        return [p[1:-1, 1:-1, 2:], p[1:-1, 1:-1, :-2], p[1:-1, 2:, 1:-1], p[1:-1, :-2, 1:-1], p[2:, 1:-1, 1:-1], p[:-2, 1:-1, 1:-1]]

    open_ = [~s for s in around(solid, True)]
    for _ in range(sweeps):
        near = around(phi, 0.0)
        inside = phi < 0
        frozen = torch.zeros_like(solid)
        ax = []
        lowest = torch.full_like(phi, math.inf)
        for m in range(6):
            frozen |= open_[m] & ((near[m] < 0) != inside)
            lowest = torch.where(open_[m], torch.minimum(lowest, near[m]), lowest)
            if m % 2 == 0:
                pair = [torch.where(open_[q], near[q].abs(), top).clamp(max=top) for q in (m, m + 1)]
                ax.append(torch.minimum(*pair))
        a, b, c = torch.stack(ax).sort(0).values
        s1 = a + h
        s2 = 0.5 * (a + b + torch.sqrt((2 * h * h - (a - b) ** 2).clamp(min=0)))
        t = a + b + c
        s3 = (t + torch.sqrt((t * t - 3 * (a * a + b * b + c * c - h * h)).clamp(min=0))) / 3
        e = torch.where(s1 > b, torch.where(s2 > c, s3, s2), s1).clamp(max=top)
        wet = torch.where(frozen, phi, torch.where(inside, -e, e))
        phi = torch.where(solid, torch.where(torch.isinf(lowest), phi.clamp(-top, top), lowest), wet)
    return phi


def _filltrapped64(grid, solid, phi):
    """Air that no path joins to the top layer becomes water, phi at most -2 dx (basins whose air
    is joined within the sweep rounds, as open water is)."""
    air = ~solid & ~(phi < 0)
    reach = torch.zeros_like(air)
    reach[-1] = air[-1]
    while True:
        new = reach.clone()
        for d in range(3):
            n = air.shape[d]
            new.narrow(d, 1, n - 1).logical_or_(reach.narrow(d, 0, n - 1))
            new.narrow(d, 0, n - 1).logical_or_(reach.narrow(d, 1, n - 1))
        new &= air
        if torch.equal(new, reach):
            break
        reach = new
    return torch.where(air & ~reach, phi.clamp(max=-2 * grid.dx), phi)


def _extrapolate64(f, flags, walled, layers):
    f, flags = f.double(), flags.bool()
    for _ in range(layers):
        s, m = torch.zeros_like(f), torch.zeros_like(f)
        val = torch.where(flags, f, 0.0)
        for d in range(3):
            n = f.shape[d]
            for a, b in ((0, 1), (1, 0)):
                s.narrow(d, a, n - 1).add_(val.narrow(d, b, n - 1))
                m.narrow(d, a, n - 1).add_(flags.narrow(d, b, n - 1))
        grow = ~flags & ~walled & (m > 0)
        f = torch.where(grow, s / m.clamp(min=1), f)
        flags = flags | grow
    return torch.where(flags & ~walled, f, 0.0)


def _sparse64(t):
    """project! of a sparse basin: its fine and coarse cells as one graph of couplings."""
    nb, nc, nf, used = t["nb"], t["nc"], t["nf"], t["used"]
    dx, cdx = t["grid"].dx, 4 * t["grid"].dx
    cells, pool = _cell_index(t), used[:, None] * BCELLS + torch.arange(BCELLS, device="cuda")
    cov = _covered(t)
    tc, phic = t["tc"].reshape(nc[::-1]), t["phic"].double().reshape(nc[::-1])

    def virtual(coarse, fine):
        a = _up(coarse, 4).contiguous()
        a.view(-1)[cells] = fine[pool]
        return a

    liq_f, liq_c = t["tf"] == LIQUID, (tc == LIQUID) & ~cov
    used_cells = torch.zeros(t["nslots"], BCELLS, dtype=torch.bool, device="cuda")
    used_cells[used] = True
    liq_f &= used_cells.reshape(-1)
    nfl, ncl = int(liq_f.sum()), int(liq_c.sum())
    id_f, id_c = torch.cumsum(liq_f.long(), 0) - 1, (torch.cumsum(liq_c.reshape(-1).long(), 0) - 1 + nfl).reshape(liq_c.shape)
    T, PHI, ID, F = virtual(tc, t["tf"]), virtual(phic, t["phif"].double()), virtual(id_c, id_f), _up(cov, 4)
    n = nfl + ncl
    air = torch.zeros(n, dtype=torch.float64, device="cuda")
    ei, ej, ec = [], [], []

    def couple(types, phi, ids, keep, weight, axis):
        two = _pairs(types, axis)
        (ta, tb), (pa, pb), (ia, ib) = two(types), two(phi), two(ids)
        m = keep & (ta == LIQUID) & (tb == LIQUID)
        ei.append(ia[m])
        ej.append(ib[m])
        ec.append(weight[m])
        for t0, t1, p0, p1, i0 in ((ta, tb, pa, pb, ia), (tb, ta, pb, pa, ib)):
            m = keep & (t0 == LIQUID) & (t1 == AIR)
            air.index_add_(0, i0[m], weight[m] / _theta(p0[m], p1[m]))

    for axis in range(3):
        fa, fb = _pairs(F, axis)(F)
        couple(T, PHI, ID, fa | fb, torch.where(fa & fb, 1.0, 0.4).double(), axis)
        ca, cb = _pairs(cov, axis)(cov)
        couple(tc, phic, id_c, ~ca & ~cb, torch.full_like(ca, 4.0, dtype=torch.float64), axis)
    del ID
    # the volume's loss and the right-hand sides
    x, y, z = (_centres(t["grid"].lo[a], cdx, nc[a]) for a in range(3))
    r2 = t["grid"].radius ** 2
    csolid = ((x * x)[None, :] + (y * y)[:, None] > r2)[None] | (z < t["grid"].floor_z)[:, None, None]
    x, y, z = (_centres(t["grid"].lo[a], dx, nf[a]) for a in range(3))
    fsolid = ((x * x)[None, :] + (y * y)[:, None] > r2)[None] | (z < t["grid"].floor_z)[:, None, None]
    vol = float(torch.where(F & ~fsolid, (0.5 - PHI / dx).clamp(0, 1), 0.0).sum())
    vol += 64 * float(torch.where(~cov & ~csolid, (0.5 - phic / cdx).clamp(0, 1), 0.0).sum())
    gamma = min(0.01 / DT, max(-0.01 / DT, (1 - 1 / LOSS) / RECOVER)) if vol > 0 else 0.0
    del fsolid
    div_f = torch.zeros(t["nslots"], 16, 16, 16, dtype=torch.float64, device="cuda")
    div_c = torch.zeros(nc[::-1], dtype=torch.float64, device="cuda")
    for axis in range(3):
        d = 2 - axis
        e = [16 + (a == axis) for a in range(3)]
        f = t["uvw"[axis] + "f"].double().reshape(t["nslots"], e[2], e[1], e[0])
        div_f += f.narrow(d + 1, 1, 16) - f.narrow(d + 1, 0, 16)
        e = [nc[a] + (a == axis) for a in range(3)]
        f = t["uvw"[axis] + "c"].double().reshape(e[::-1])
        div_c += f.narrow(d, 1, nc[axis]) - f.narrow(d, 0, nc[axis])
    b = torch.cat([(-dx * div_f.reshape(-1) + gamma * dx * dx)[liq_f], (-16 * dx * div_c + 64 * gamma * dx * dx)[liq_c]])
    x = _cg(n, torch.cat(ei), torch.cat(ej), torch.cat(ec), air, b, torch.zeros_like(b))
    Pf, Pc = t["Pf"].double().clone(), torch.zeros(nc[::-1], dtype=torch.float64, device="cuda")
    Pf[used_cells.reshape(-1)] = 0.0
    Pf[liq_f], Pc[liq_c] = x[:nfl], x[nfl:]
    out = {}
    # the gradient: fine faces from the box's cells with a border of SOLID, then the coarse faces
    pad = lambda a, v: torch.nn.functional.pad(a, (1,) * 6, value=v).reshape(-1)
    Tp, PHIp, Pp, Fp = pad(T, SOLID), pad(PHI, 0.0), pad(virtual(Pc, Pf), 0.0), pad(F, False)
    dims = [m + 2 for m in nf]

    def drop(ta, tb, pa, pb, qa, qb):
        ok = (ta != SOLID) & (tb != SOLID) & ((ta == LIQUID) | (tb == LIQUID))
        both = (ta == LIQUID) & (tb == LIQUID)
        one = torch.where(ta == LIQUID, -pa / _theta(qa, qb), pb / _theta(qb, qa))
        return torch.where(ok, torch.where(both, pb - pa, one), 0.0)

    for axis in range(3):
        name, d = "uvw"[axis], 2 - axis
        hi, lo = _face_index(t, axis, dims, 0, 1), _face_index(t, axis, dims, 1, 1)
        D = drop(Tp[lo], Tp[hi], Pp[lo], Pp[hi], PHIp[lo], PHIp[hi]) / (torch.where(Fp[lo] & Fp[hi], 1.0, 2.5) * dx)
        fine = t[name + "f"].double().reshape(t["nslots"], BFACES).clone()
        fine[used] -= D
        ca, cb = _pairs(cov, axis)(cov)
        two = _pairs(tc, axis)
        (ta, tb), (pa, pb), (qa, qb) = two(tc), two(Pc), two(phic)
        D = torch.where(~ca & ~cb, drop(ta, tb, pa, pb, qa, qb), 0.0) / cdx
        coarse = t[name + "c"].double().reshape([nc[a] + (a == axis) for a in range(3)][::-1]).clone()
        coarse.narrow(d, 1, nc[axis] - 1).sub_(D)
        box = torch.zeros([nf[a] + (a == axis) for a in range(3)][::-1], dtype=torch.float64, device="cuda")
        box.view(-1)[_face_index(t, axis)] = fine[used]
        coarse = torch.where(_held(t, axis), _face_means(box, axis), coarse)
        out[name + "f"], out[name + "c"] = fine.reshape(-1), coarse.reshape(-1)
        del box
    out["Pf"], out["Pc"] = Pf, Pc.reshape(-1)
    return [out[f] for f in SPARSE_STATE] + [None] * 6


def exact(case, seed):
    c, k = case, case["kind"]
    flat = lambda ts: [x.reshape(-1) for x in ts]
    if k == "project":
        d = _dense_of(c, seed)
        out, P = _Dense64(d).project([f.double() for f in d["faces"]])
        return flat(out + [P]) + [None] * 3
    if k == "batch":
        outs = []
        for d in _batch_members(c, seed):
            out, P = _Dense64(d).project([f.double() for f in d["faces"]])
            outs.append(flat(out + [P]))
        u, v, w, P = (torch.cat(x) for x in zip(*outs))
        return [u, v, w, None, None, None, P]
    if k in ("adjoint", "rollout"):
        d = _dense_of(c, seed)
        sys64 = _Dense64(d)
        g = _gen(seed, 77)
        start = [f.double().requires_grad_(True) for f in d["faces"]]
        target = [_uniform(g, f.numel()).double().reshape(f.shape) for f in d["faces"]]
        f = start
        for _ in range(c["steps"] if k == "rollout" else 1):
            if k == "rollout":
                f = _advect64(d["grid"], f)
            f = _Project64.apply(*f, sys64)
        loss = sum(0.5 * ((o - x) ** 2).sum() for o, x in zip(f, target))
        return flat([o.detach() for o in f] + list(torch.autograd.grad(loss, start)))
    if k == "levelset":
        d = _levelset_inputs(c, seed)
        return [_filltrapped64(d["grid"], d["solid"], _redistance64(d, c["sweeps"])).reshape(-1), None]
    if k == "extrapolate":
        d = _dense((c["n1"], c["n2"], c["n3"]), seed, vortex=225.0)
        return flat([_extrapolate64(f, _flags(d["types"], a), _walled(d["solid"], a), c["layers"]) for a, f in enumerate(d["faces"])]) + [None] * 3
    return _sparse64(_sparse_scene(c, seed))
