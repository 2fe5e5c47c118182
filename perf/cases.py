"""The work a user of this package has it do, as a list of measurable cases.

Every case goes through the package's public classes (``FluidSim.step``, ``Batch.step``,
``SplatField.bake``, ``SurfaceExtractor.extract``, ``ClaySolver.step``, ``SdfVolume.build``,
``TracedField.query_mip_device``) on inputs made from a seed. Sizes are those of the package's
workloads (``clay_engine_b200/scenes.py``) and the ranges around them:

- ``listed()``: the named cases; ``draw(rng)``: one more case of the same ranges.
- ``prepare(case, seed)`` -> state; ``run(state)``: one pass, its outputs as device tensors.
- ``work(case)``: the bytes and operations a pass cannot do without.
- ``exact(case, seed)``: what ``run`` returns for a new state, in 64-bit arithmetic written here.

A fluid scene is a snapshot of a running simulation: its particle records are put back before
each frame (one device copy), so that every pass advances the same state instead of a state that
settles as passes go by. Colliders are planes computed here and uploaded, as a saved level is.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import clay_engine_b200 as ce
from clay_engine_b200 import _native, scenes

ORIGIN, WORLD = scenes.WORLD_ORIGIN, scenes.WORLD_SIZE
FLOOR, TAP_POS, BODY_POS = -2.0, scenes.CONFIG2["tap"]["pos"], (7.5, -0.9, 7.5)
SPACING, RADIUS = 0.1, 0.05
SMOOTHING, SURFACE = SPACING * 2.2, SPACING * 1.1
BAND = 4.0
_ROOT = None


def listed():
    return [
        # the small game scene: one blob of 4,096 particles, every launch nearly empty
        {"name": "frame_4096", "kind": "frame", "n": 4096, "spray": 0.0, "tap": 0, "collider": 96, "bake": 64, "mips": 3,
         "substeps": 2},
        # a full tap ring: 262,144 particles as pool, thin spray and dense clumps, 4,096 emitted each frame
        {"name": "frame_tap_262144", "kind": "frame", "n": 262144, "spray": 0.6, "tap": 4096, "collider": 192, "bake": 128,
         "mips": 4, "substeps": 2},
        # the largest single scene
        {"name": "frame_1048576", "kind": "frame", "n": 1048576, "spray": 0.05, "tap": 0, "collider": 288, "bake": 128,
         "mips": 4, "substeps": 2},
        # many uneven scenes per launch, a third of them with a clay body
        {"name": "batch_96", "kind": "batch", "scenes": 96, "lo": 1024, "hi": 65536, "subset": 0, "body_every": 3},
        # one frame of the serving loop: the scenes with a request in progress, of a resident pool
        {"name": "serve_frame_24_of_40", "kind": "batch", "scenes": 40, "lo": 2048, "hi": 65536, "subset": 24, "body_every": 0},
        # a clay body's shell (oriented discs) into the small volume that follows it
        {"name": "bake_body_3800", "kind": "bake", "n": 3800, "discs": True, "resolution": 32, "mips": 2, "band": 4.0},
        # a free cloud in no particular order
        {"name": "bake_cloud_100003", "kind": "bake", "n": 100003, "discs": False, "resolution": 128, "mips": 4, "band": 2.0},
        # surface nets: a body at the game's lattice, and a fine one
        {"name": "extract_32", "kind": "extract", "resolution": 32},
        {"name": "extract_128", "kind": "extract", "resolution": 128},
        # shape-matched clay bodies over a collider
        {"name": "solver_86", "kind": "solver", "bodies": 86, "cell": 0.067, "substeps": 2},
        # a world volume from its brush list
        {"name": "build_192", "kind": "build", "resolution": 192, "mips": 4, "brushes": 64},
        # sampling a volume at scattered points
        {"name": "query_4194304", "kind": "query", "n": 1 << 22, "mip": 0, "resolution": 192, "mips": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "batch", "batch", "bake", "bake", "extract", "solver", "build", "query"])
    if kind == "frame":
        bake, mips = rng.choice([(32, 2), (64, 3), (128, 4)])
        n = _log(rng, 1000, 600000)
        tap = rng.choice([0, 0, 1])
        return {"kind": kind, "n": n, "spray": rng.choice([0.0, 0.1, 0.5]), "tap": min(4096, n // 8) if tap else 0,
                "collider": rng.choice([64, 96, 192]), "bake": bake, "mips": mips, "substeps": rng.choice([1, 2, 2, 3])}
    if kind == "batch":
        n = _log(rng, 2, 64)
        return {"kind": kind, "scenes": n, "lo": 1000, "hi": _log(rng, 4000, 65536), "subset": rng.choice([0, max(1, n // 2)]),
                "body_every": rng.choice([0, 2, 3])}
    if kind == "bake":
        discs = rng.random() < 0.5
        res, mips = rng.choice([(32, 2), (32, 1), (64, 3), (64, 1)] + ([] if discs else [(128, 4)]))
        return {"kind": kind, "n": _log(rng, 300, 20000) if discs else _log(rng, 300, 300000), "discs": discs,
                "resolution": res, "mips": mips, "band": rng.choice([2.0, 3.0, 4.0])}
    if kind == "extract":
        return {"kind": kind, "resolution": _log(rng, 12, 128)}
    if kind == "solver":
        return {"kind": kind, "bodies": _log(rng, 1, 80), "cell": rng.choice([0.067, 0.09, 0.12]), "substeps": rng.choice([1, 2, 2, 4])}
    if kind == "build":
        mips = rng.choice([1, 2, 3])
        return {"kind": kind, "resolution": 32 * rng.randint(1, 6), "mips": mips, "brushes": _log(rng, 1, 100)}
    mips = rng.choice([1, 3, 4])
    return {"kind": kind, "n": _log(rng, 1000, 4000000), "mip": rng.randint(0, mips), "resolution": rng.choice([64, 128, 192]),
            "mips": mips}


# ---- inputs -------------------------------------------------------------------------------

def _root():
    global _ROOT
    if _ROOT is None:
        _ROOT = ce.init(0)
    return _ROOT


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def _rand(g, *shape):
    return torch.rand(*shape, device="cuda", dtype=torch.float64, generator=g)


class _Memory:
    """Device memory of a library object as a tensor (zero copy); it keeps `owner` alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 2}


def _view(owner, ptr, shape, typestr):
    return torch.as_tensor(_Memory(owner, ptr, shape, typestr), device="cuda")


class _Owner:
    """Destroys library objects in order once nothing refers to them."""

    def __init__(self):
        self.objects = []

    def add(self, *objects):
        self.objects += objects
        return objects[-1]

    def __del__(self):
        for o in reversed(self.objects):
            if hasattr(o, "destroy"):
                o.destroy()


def _plane_view(owner, volume, which=0):
    import ctypes

    d, m = ctypes.c_void_p(), ctypes.c_void_p()
    _native.check(_native.lib().clay_volume_device_planes(volume.handle, ctypes.byref(d), ctypes.byref(m)))
    return _view(owner, (d, m)[which].value, (volume.totalVoxels,), "<f2")


def _bumps(seed, count=12):
    g = _gen(seed, 7)
    c = (_rand(g, count, 3) * 2 - 1) * 9.5
    c[:, 1] = FLOOR - 0.2
    return c, 0.5 + 0.7 * _rand(g, count)


def _terrain(p, bumps):
    """A floor with rounded bumps: distance at points p (n x 3, float64)."""
    d = p[:, 1] - FLOOR
    for c, r in zip(*bumps):
        d = torch.minimum(d, (p - c).norm(dim=1) - r)
    return d


def _grid(res, world, origin, device="cuda"):
    a = (torch.arange(res, device=device, dtype=torch.float64) + 0.5) * (world / res)
    z, y, x = torch.meshgrid(a + origin[2], a + origin[1], a + origin[0], indexing="ij")
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)


def _planes(res, mips, world, origin, band, distance):
    """All levels of a volume of `distance`: (band-normalised distances, material), float16."""
    out = []
    for m in range(mips):
        bw = band * (world / res) * 2 ** m
        out.append((distance(_grid(res >> m, world, origin)) / bw).clamp(-1, 1).to(torch.float16))
    d = torch.cat(out)
    return d, torch.where(d < 0, 1.0, 0.25).to(torch.float16)


def _volume(owner, res, mips, world, origin, distance, band=BAND):
    vol = owner.add(ce.SdfVolume(_root(), resolution=res, worldSize=world, origin=origin, mipLevels=mips, band=band))
    d, m = _planes(res, mips, world, origin, band, distance)
    vol.upload(d.cpu().numpy().view(np.uint16), m.cpu().numpy().view(np.uint16))
    return vol


def _block(n, spacing, center, bumps, g, keep):
    """`n` particles of a jittered lattice resting on the terrain around (x, z) = center."""
    side = max(2, int(math.ceil((n * 1.06) ** (1 / 3))))
    layers = int(math.ceil(n * 1.06 / side ** 2)) + 3
    a = (torch.arange(side, device="cuda", dtype=torch.float64) + 0.5 - side / 2) * spacing
    y = FLOOR + 0.06 + torch.arange(layers + 14, device="cuda", dtype=torch.float64) * spacing
    yy, zz, xx = torch.meshgrid(y, a + center[1], a + center[0], indexing="ij")
    p = torch.stack([xx.reshape(-1), yy.reshape(-1), zz.reshape(-1)], 1)
    p += (_rand(g, *p.shape) * 2 - 1) * 0.1 * spacing
    p = p[(_terrain(p, bumps) > 0.045) & keep(p)]
    return p[:n]


def _particles(n, spray, seed, body=False, tap=False):
    """Records (n x 12 float32) of a pool on the terrain, a share of thin spray above it, and,
    with spray of half or more, dense clumps."""
    bumps, g = _bumps(seed), _gen(seed, 1)

    def keep(p):
        ok = torch.ones(len(p), dtype=torch.bool, device="cuda")
        if body:
            ok &= (p - torch.tensor(BODY_POS, device="cuda")).norm(dim=1) > 1.1
        if tap:
            ok &= (p - torch.tensor(TAP_POS, device="cuda")).norm(dim=1) > 1.3
        return ok

    ns = int(n * spray)
    nc = int(n * 0.05) if spray >= 0.5 else 0
    parts = [_block(n - ns - nc, SPACING, (-1.0, -1.0), bumps, g, keep)]
    if nc:
        parts.append(_block(nc, 0.082, (8.0, -7.0), bumps, g, keep))
    if ns:
        p = _rand(g, 3 * ns + 4096, 3)
        p = torch.stack([(p[:, 0] * 2 - 1) * 10, FLOOR + 0.1 + 4.5 * p[:, 1] ** 2, (p[:, 2] * 2 - 1) * 10], 1)
        parts.append(p[(_terrain(p, bumps) > 0.08) & keep(p)][:ns])
    p = torch.cat(parts)
    v = 0.3 * torch.randn(len(p), 3, device="cuda", dtype=torch.float64, generator=g)
    v[:, 0] += 0.3 * (p[:, 1] - FLOOR)
    v[:, 1] -= 0.2
    if ns:
        v[-ns:] *= 3.0
        order = torch.randperm(len(p), device="cuda", generator=g)  # a ring mixes its slots
        p, v = p[order], v[order]
    assert len(p) == n
    rec = torch.zeros(n, 12, device="cuda", dtype=torch.float32)
    rec[:, 0:3], rec[:, 4:7], rec[:, 8:11] = p.float(), v.float(), v.float()
    return rec


def _fluid_opts(n, bake, mips, substeps):
    return dict(capacity=int(n), spacing=SPACING, radius=RADIUS, substeps=substeps, gravity=(0, -9.8, 0), bakeResolution=bake,
                bakeMipLevels=mips, bakeBand=BAND, worldSize=WORLD, origin=ORIGIN)


def _shell(cell, radius=0.95):
    return scenes.surface_net_sphere(radius, cell)


def _body_splat(owner, center):
    b = scenes.CONFIG3["body"]
    pos, nrm = _shell(b["cell"], b["radius"])
    parts, rec = scenes.body_records(pos + np.array(center, np.float32), nrm, center)
    dp, db = torch.from_numpy(parts.view(np.uint8)).cuda(), torch.from_numpy(rec.view(np.uint8)).cuda()
    owner.add(dp, db)
    s = owner.add(ce.SplatField(_root(), ce.bodyCloud(dp, db, 0), radius=b["bake_box"] / b["bake_res"] * 1.15,
                                resolution=b["bake_res"], band=b["band"], worldSize=b["bake_box"]))
    s.setCenter(center)
    return s


def _scene(owner, n, seed, collider, bake, mips, substeps, spray=0.0, tap=False, body=False):
    """(sim, its record view, the records to start from, the body's SplatField or None)."""
    bumps = _bumps(seed)
    vol = _volume(owner, collider, 1, WORLD, ORIGIN, lambda p: _terrain(p, bumps))
    world = owner.add(ce.volumeField(vol))
    shell = None
    if body:
        shell = _body_splat(owner, BODY_POS)
        world = owner.add(ce.unionField(world, shell.field))
    sim = owner.add(ce.FluidSim(_root(), world, _fluid_opts(n, bake, mips, substeps)))
    rec = _particles(n, spray, seed, body=body, tap=tap)
    sim.upload(rec.cpu().numpy().view(ce.PARTICLE_DTYPE).reshape(-1))
    return sim, _view(owner, sim.particles_ptr()[0], (n, 12), "<f4"), rec, shell


def _batch_sizes(case, seed):
    r = np.random.default_rng(4242)  # the sizes belong to the case, not to its inputs
    n = np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["scenes"])).astype(np.int64)
    bakes = [[(64, 3)], [(32, 2), (64, 3), (128, 4)]][bool(case["subset"])]
    picks = r.integers(0, len(bakes), case["scenes"])
    sub = sorted(r.choice(case["scenes"], case["subset"], replace=False).tolist())
    body = [bool(case["body_every"]) and i % case["body_every"] == 0 for i in range(case["scenes"])]
    return [int(x) for x in n], [bakes[int(i)] for i in picks], body, sub


def _blob_distance(seed, radius):
    g = _gen(seed, 3)
    c, r = (_rand(g, 4, 3) * 2 - 1) * 0.35 * radius, radius * (0.45 + 0.2 * _rand(g, 4))

    def distance(p):
        d = torch.stack([(p - ci).norm(dim=1) - ri for ci, ri in zip(c, r)])
        return -torch.logsumexp(-d * 12, 0) / 12

    return distance


def _bake_cloud(case, seed):
    """(positions, normals or None, quaternion, radius, world size, origin) of a bake, float32."""
    n, g = case["n"], _gen(seed, 5)
    if case["discs"]:
        world = 2.656
        v = torch.randn(n, 3, device="cuda", dtype=torch.float64, generator=g)
        nrm = (v / v.norm(dim=1, keepdim=True)).float()
        # a shell's slots follow its lattice: sorted by height, then depth
        nrm = nrm[torch.argsort(torch.floor(nrm[:, 2] * 14) * 64 + torch.floor(nrm[:, 1] * 14))]
        pos = nrm * (0.95 * (0.9 + 0.1 * float(_rand(g, 1)))) + torch.tensor(BODY_POS, device="cuda")
        q = torch.randn(4, device="cuda", dtype=torch.float64, generator=g)
        quat = (q / q.norm()).float()
        return pos.contiguous(), nrm.contiguous(), quat, world / case["resolution"] * 1.15, world, tuple(c - world / 2 for c in BODY_POS)
    pos = torch.tensor((0.0, 3.0, 0.0), device="cuda") + (torch.randn(n, 3, device="cuda", generator=g) * 2.5).clamp(-8, 8)
    return pos.contiguous(), None, None, SURFACE, WORLD, ORIGIN


def _bodies(case, seed):
    """Particle and Body records of the solver's bodies over the terrain."""
    pos, nrm = _shell(case["cell"])
    n, k = len(pos), case["bodies"]
    r = np.random.default_rng(seed)
    parts, bodies = np.zeros(n * k, scenes.PARTICLE_RECORD), np.zeros(k, scenes.BODY_RECORD)
    for b in range(k):
        c = np.array([r.uniform(-9, 9), FLOOR + r.uniform(1.6, 4.0), r.uniform(-9, 9)], np.float32)
        s = slice(b * n, (b + 1) * n)
        parts["pos"][s] = pos + c
        vel = r.normal(0, 1.0, 3).astype(np.float32)
        parts["prev"][s] = parts["pos"][s] - vel / 120 + r.normal(0, 1e-3, (n, 3)).astype(np.float32)
        parts["vel"][s] = parts["velPrev"][s] = vel
        parts["rest"][s], parts["restNormal"][s], parts["body"][s], parts["material"][s] = pos, nrm, b, 0.5
        bodies["com"][b], bodies["first"][b], bodies["count"][b], bodies["rot"][b] = c, b * n, n, (0, 0, 0, 1)
        bodies["stiffness"][b] = 0.8
    return parts, bodies


def _brushes(case, seed):
    return scenes.random_brushes(case["brushes"], seed=seed)


def _query_points(case, seed):
    g = _gen(seed, 9)
    return ((_rand(g, case["n"], 3) * 1.02 - 0.01) * WORLD + torch.tensor(ORIGIN, device="cuda", dtype=torch.float64)).float().contiguous()


# ---- prepare and run ----------------------------------------------------------------------

def prepare(case, seed):
    own, kind = _Owner(), case["kind"]
    s = {"case": case, "own": own}
    if kind == "frame":
        sim, view, rec, _ = _scene(own, case["n"], seed, case["collider"], case["bake"], case["mips"], case["substeps"],
                                   case["spray"], tap=bool(case["tap"]))
        s.update(sim=sim, view=view, start=rec, sdf=_plane_view(own, sim.surface.volume))
    elif kind == "batch":
        sizes, bakes, body, sub = _batch_sizes(case, seed)
        sc = [_scene(own, n, seed * 4099 + i, 64, *bakes[i], 2, body=body[i]) for i, n in enumerate(sizes)]
        shells = [x[3] for x in sc if x[3] is not None]
        picked = sub or list(range(len(sc)))
        s.update(batch=own.add(ce.Batch(_root(), [x[0] for x in sc], extra_splats=shells)), sub=sub,
                 views=[sc[i][1] for i in picked], starts=[sc[i][2] for i in picked],
                 sdfs=[_plane_view(own, sc[i][0].surface.volume) for i in picked],
                 shells=[] if sub else [_plane_view(own, x.volume) for x in shells])
    elif kind == "bake":
        pos, nrm, quat, radius, world, origin = _bake_cloud(case, seed)
        live = torch.tensor([case["n"]], dtype=torch.int32, device="cuda")
        own.add(pos, nrm, quat, live)
        cloud = ce.ParticleCloud(case["n"], pos, live=("count", live), normals=nrm, normal_stride=12 if nrm is not None else None,
                                 rotation=quat)
        f = own.add(ce.SplatField(_root(), cloud, radius=radius, resolution=case["resolution"], mipLevels=case["mips"],
                                  band=case["band"], worldSize=world, origin=origin))
        s.update(splat=f, sdf=_plane_view(own, f.volume))
    elif kind == "extract":
        box = 2.656
        lo = (-box / 2,) * 3
        field = own.add(ce.volumeField(_volume(own, 64, 1, box, lo, _blob_distance(seed, 0.95))))
        cap = max(1024, 4 * case["resolution"] ** 2)
        parts = torch.zeros(cap, 24, device="cuda")
        bodies = torch.zeros(1, 16, device="cuda")
        own.add(parts, bodies)
        x = own.add(ce.SurfaceExtractor(_root(), parts, cap, bodies, 1, field, 0, 0, cap, resolution=case["resolution"]))
        x.setRegion(lo, box)
        idx = _view(own, x.indices_ptr, (x.quadCapacity, 6), "<i4")
        idx.zero_()
        s.update(extractor=x, parts=parts, bodies=bodies, idx=idx, draw=_view(own, x.draw_args_ptr, (4,), "<i4"))
    elif kind == "solver":
        parts, bodies = _bodies(case, seed)
        bumps = _bumps(seed)
        world = own.add(ce.volumeField(_volume(own, 64, 1, WORLD, ORIGIN, lambda p: _terrain(p, bumps))))
        dp = torch.from_numpy(parts.view(np.float32).reshape(-1, 24).copy()).cuda()
        db = torch.from_numpy(bodies.view(np.float32).reshape(-1, 16).copy()).cuda()
        own.add(dp, db)
        s.update(solver=own.add(ce.ClaySolver(_root(), dp, len(parts), db, len(bodies), world, {"substeps": case["substeps"]})),
                 parts=dp, bodies=db)
    elif kind == "build":
        vol = own.add(ce.SdfVolume(_root(), resolution=case["resolution"], worldSize=WORLD, origin=ORIGIN, mipLevels=case["mips"],
                                   band=BAND))
        s.update(volume=vol, brushes=_brushes(case, seed), dist=_plane_view(own, vol, 0), mat=_plane_view(own, vol, 1))
    else:
        bumps = _bumps(seed)
        vol = _volume(own, case["resolution"], case["mips"], WORLD, ORIGIN, lambda p: _terrain(p, bumps))
        s.update(field=own.add(ce.volumeField(vol)), points=_query_points(case, seed),
                 sample=torch.empty(case["n"], 2, device="cuda"), value=torch.empty(case["n"], 2, device="cuda"))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        s["view"].copy_(s["start"])
        if case["tap"]:
            s["sim"].spawn(case["tap"], TAP_POS, (0.0, -2.0, 0.0))
        s["sim"].step()
        v = s["view"]
        return {"pos": v[:, 0:3], "density": v[:, 3], "vel": v[:, 4:7], "pressure": v[:, 7], "nvel": v[:, 8:11], "sdf": s["sdf"]}
    if kind == "batch":
        torch._foreach_copy_(s["views"], s["starts"])
        if s["sub"]:
            s["batch"].step_subset(s["sub"])
        else:
            s["batch"].step()
        out = {"records": torch.cat(s["views"]), "sdf": torch.cat(s["sdfs"])}
        if s["shells"]:
            out["shells"] = torch.cat(s["shells"])
        return out
    if kind == "bake":
        s["splat"].bake()
        return {"sdf": s["sdf"]}
    if kind == "extract":
        s["extractor"].extract()
        return {"particles": s["parts"], "bodies": s["bodies"], "indices": s["idx"], "draw": s["draw"]}
    if kind == "solver":
        s["solver"].step(case["bodies"])
        return {"particles": s["parts"], "bodies": s["bodies"]}
    if kind == "build":
        s["volume"].build(s["brushes"])
        return {"dist": s["dist"], "mat": s["mat"]}
    s["field"].query_mip_device(s["points"], s["sample"], s["value"], case["mip"])
    return {"sample": s["sample"], "value": s["value"]}


# ---- work ---------------------------------------------------------------------------------

def _voxels(res, mips):
    return sum((res >> m) ** 3 for m in range(mips))


def _frame_work(n, substeps, collider, bake, mips):
    near = 4 / 3 * math.pi * (SMOOTHING / SPACING) ** 3  # neighbours at rest density
    in_band = sum(min((bake >> m) ** 3, 4 / 3 * math.pi * (SURFACE / (WORLD / bake * 2 ** m) + BAND) ** 3) for m in range(mips))
    return {"bytes": 96.0 * n + min(2.0 * collider ** 3, 32.0 * n) + 2.0 * _voxels(bake, mips),
            "flops": n * (substeps * near * (13 + 30) + 9 * in_band)}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        return _frame_work(case["n"], case["substeps"], case["collider"], case["bake"], case["mips"])
    if kind == "batch":
        sizes, bakes, body, sub = _batch_sizes(case, 0)
        w = [_frame_work(sizes[i], 2, 64, *bakes[i]) for i in (sub or range(len(sizes)))]
        shells = 0 if sub else sum(body)
        return {"bytes": sum(x["bytes"] for x in w) + shells * (3800 * 24 + 2 * _voxels(32, 2)),
                "flops": sum(x["flops"] for x in w) + shells * 3800 * 12.0 * 800}
    if kind == "bake":
        vox = (2.656 if case["discs"] else WORLD) / case["resolution"]
        r = 1.15 * vox if case["discs"] else SURFACE
        hits = sum(min((case["resolution"] >> m) ** 3, 4 / 3 * math.pi * (r / (vox * 2 ** m) + case["band"]) ** 3) for m in range(case["mips"]))
        return {"bytes": case["n"] * (24.0 if case["discs"] else 12.0) + 2.0 * _voxels(case["resolution"], case["mips"]),
                "flops": case["n"] * hits * (12.0 if case["discs"] else 9.0)}
    if kind == "extract":
        r = case["resolution"]
        return {"bytes": 2.0 * 64 ** 3 + 2.5 * r * r * (96 + 24), "flops": 30.0 * r ** 3}
    if kind == "solver":
        n = len(_shell(case["cell"])[0]) * case["bodies"]
        return {"bytes": n * (96.0 + 96.0) + 128.0 * case["bodies"] + 2.0 * 64 ** 3, "flops": n * case["substeps"] * 250.0}
    if kind == "build":
        v = _voxels(case["resolution"], case["mips"])
        return {"bytes": 4.0 * v + 80.0 * case["brushes"], "flops": v * 60.0}
    return {"bytes": case["n"] * 28.0 + min(4.0 * _voxels(case["resolution"], case["mips"]), 64.0 * case["n"]),
            "flops": case["n"] * 60.0}


# ---- exact --------------------------------------------------------------------------------

def _sample(plane, res, world, origin, band, p):
    """Trilinear band-scaled distance of float64 points inside a volume's level 0."""
    t = (p - torch.tensor(origin, device=p.device, dtype=p.dtype)) / world * res - 0.5
    f = torch.floor(t)
    w, i0 = t - f, f.long()
    out = torch.zeros(len(p), device=p.device, dtype=p.dtype)
    for k in range(8):
        bit = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=p.device)
        i = (i0 + bit).clamp(0, res - 1)
        out += plane[(i[:, 2] * res + i[:, 1]) * res + i[:, 0]].to(p.dtype) * torch.where(bit.bool(), w, 1 - w).prod(1)
    return out * (band * world / res)


def _normal(plane, res, world, origin, band, p):
    g = []
    for k in range(3):
        e = torch.zeros(3, device=p.device, dtype=p.dtype)
        e[k] = world / res
        g.append(_sample(plane, res, world, origin, band, p + e) - _sample(plane, res, world, origin, band, p - e))
    g = torch.stack(g, 1)
    return g / g.norm(dim=1, keepdim=True).clamp_min(1e-30)


def _neighbours(pos, h):
    """(order, rows): particles sorted by cell, and per row of three cells (first, past-last)."""
    c = torch.floor((pos - pos.min(0).values) / h).long() + 1
    nx, ny = int(c[:, 0].max()) + 2, int(c[:, 1].max()) + 2
    key = c[:, 0] + nx * (c[:, 1] + ny * c[:, 2])
    order = torch.argsort(key, stable=True)
    key = key[order]
    rows = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            base = key + nx * (dy + ny * dz)
            rows.append((torch.searchsorted(key, base - 1), torch.searchsorted(key, base + 1, right=True)))
    return order, rows


def _substep(p, v, plane, res, dt, h):
    """One substep in float64: (pos, density, vel, pressure, nvel)."""
    mass, poly6, spiky = SPACING ** 3, 315 / (64 * math.pi * h ** 9), -45 / (math.pi * h ** 6)
    reach = int(math.ceil(h / SPACING))
    rest = sum(mass * poly6 * (h * h - r2) ** 3 for x in range(-reach, reach + 1) for y in range(-reach, reach + 1)
               for z in range(-reach, reach + 1) if (r2 := (x * x + y * y + z * z) * SPACING ** 2) < h * h)
    order, rows = _neighbours(p, h)
    p, v = p[order], v[order]

    def each(f):
        for s, e in rows:
            for j in range(int((e - s).max())):
                q = (s + j).clamp(max=len(p) - 1)
                d = p - p[q]
                f(q, d, (d * d).sum(1), s + j < e)

    rho = torch.zeros(len(p), device=p.device, dtype=p.dtype)

    def density(q, d, r2, ok):
        rho.add_(torch.where(ok, (h * h - r2).clamp_min(0) ** 3, 0.0))

    each(density)
    rho *= mass * poly6
    dens, pres = rho.clamp_min(rest * 0.1), (220 * (rho - rest)).clamp_min(0)
    force, vs, ws = torch.zeros_like(p), torch.zeros_like(p), torch.zeros_like(rho)

    def forces(q, d, r2, ok):
        w = torch.where(ok, (h * h - r2).clamp_min(0) ** 3, 0.0)
        vs.add_(v[q] * w[:, None])
        ws.add_(w)
        r = r2.sqrt()
        s = mass * (pres + pres[q]) * 0.5 / dens[q] * spiky * (h - r).clamp_min(0) ** 2
        s = torch.where(ok & (r > 1e-6), s / r.clamp_min(1e-6), 0.0)
        force.sub_(d * s[:, None])

    each(forces)
    a = force / dens[:, None] + torch.tensor((0.0, -9.8, 0.0), device=p.device, dtype=p.dtype)
    nv = (v * 0.6 + vs / ws[:, None] * 0.4 + a * dt) * 0.995
    speed = nv.norm(dim=1, keepdim=True)
    nv = torch.where(speed > 15, nv * (15 / speed.clamp_min(1e-30)), nv)
    q = p + nv * dt
    d = _sample(plane, res, WORLD, ORIGIN, BAND, q)
    hit, n = (d < RADIUS)[:, None], _normal(plane, res, WORLD, ORIGIN, BAND, q)
    q = torch.where(hit, q + n * (RADIUS - d)[:, None], q)
    w = torch.where(hit, nv - n * (nv * n).sum(1, keepdim=True).clamp_max(0), nv)
    lo = torch.tensor(ORIGIN, device=p.device, dtype=p.dtype)
    c = torch.minimum(torch.maximum(q, lo + RADIUS), lo + WORLD - RADIUS)
    w = torch.where(c == q, w, 0.0)
    back = torch.empty_like(order)
    back[order] = torch.arange(len(order), device=order.device)
    return tuple(x[back] for x in (c, dens, w, pres, nv))


def _emit(n, spread):
    """Positions of the first emission, relative to the tap: the package's integer hash in f64."""
    mask = 0xFFFFFFFF

    def hash1(x):
        x = x ^ (x >> 16)
        x = (x * 0x7FEB352D) & mask
        x = x ^ (x >> 15)
        x = (x * 0x846CA68B) & mask
        x = x ^ (x >> 16)
        return (x & 0xFFFFFF).double() / 16777216.0

    seed = (9781 + torch.arange(n, device="cuda", dtype=torch.int64)) & mask
    r = torch.stack([hash1((seed * 3 + k) & mask) for k in range(3)], 1)
    d = r * 2 - 1 + 1e-4
    return d / d.norm(dim=1, keepdim=True) * (spread * r[:, :1] ** (1 / 3))


def _exact_splat(pos, nrm, radius, res, mips, world, origin, band):
    """Band-normalised distance of the union of spheres (or oriented discs), every level."""
    lo = torch.tensor(origin, device=pos.device, dtype=torch.float64)
    out = []
    for m in range(mips):
        r, vox = res >> m, world / res * 2 ** m
        bw = band * vox
        t = (pos - lo) / vox
        base, k = torch.floor(t).long(), int(math.ceil(radius / vox + band)) + 1
        best = torch.full((r ** 3,), bw, device=pos.device, dtype=torch.float64)
        for o in np.ndindex(2 * k + 1, 2 * k + 1, 2 * k + 1):
            i = base + (torch.tensor(o, device=pos.device) - k)
            ok = ((i >= 0) & (i < r)).all(1)
            d = (i[ok].double() + 0.5) * vox - (pos[ok] - lo)
            sd = d.norm(dim=1) - radius
            if nrm is not None:
                sd = torch.maximum(sd, (d * nrm[ok]).sum(1))
            i = i[ok]
            best.scatter_reduce_(0, (i[:, 2] * r + i[:, 1]) * r + i[:, 0], sd, "amin")
        out.append((best / bw).clamp(-1, 1))
    return torch.cat(out)


def _rotate(q, v):
    t = 2 * torch.cross(q[..., :3].expand_as(v), v, dim=-1)
    return v + t * q[..., 3:] + torch.cross(q[..., :3].expand_as(v), t, dim=-1)


def _exact_solver(case, seed):
    parts, bodies = _bodies(case, seed)
    k, n = case["bodies"], len(parts) // case["bodies"]
    bumps = _bumps(seed)
    plane, _ = _planes(64, 1, WORLD, ORIGIN, BAND, lambda p: _terrain(p, bumps))
    get = lambda name: torch.from_numpy(parts[name].copy()).cuda().double().reshape(k * n, 3)  # noqa: E731
    pos, prev, vel, vprev, rest = (get(x) for x in ("pos", "prev", "vel", "velPrev", "rest"))
    h, radius, grav = 1 / 60 / case["substeps"], 0.1, torch.tensor((0, -9.81, 0), device="cuda", dtype=torch.float64)
    rot = torch.tensor((0.0, 0, 0, 1), device="cuda", dtype=torch.float64).repeat(k, 1)

    def contact(q):
        d = _sample(plane, 64, WORLD, ORIGIN, BAND, q)
        return (d < radius)[:, None], _normal(plane, 64, WORLD, ORIGIN, BAND, q), (radius - d)[:, None]

    for _ in range(case["substeps"]):
        q = (pos * 4 - prev) / 3 + ((vel * 4 - vprev) / 3 + grav * (2 * h / 3)) * (2 * h / 3)
        hit, nn, push = contact(q)
        qc, pc = q + nn * push, pos + nn * push
        d = qc - pos
        qc = qc - (d - nn * (d * nn).sum(1, keepdim=True)) * 0.35
        q, prev = torch.where(hit, qc, q), torch.where(hit, pc, pos)
        pb, rb = q.reshape(k, n, 3), rest.reshape(k, n, 3)
        com, rcom = pb.mean(1, keepdim=True), rb.mean(1, keepdim=True)
        a = torch.einsum("bni,bnj->bji", pb - com, rb - rcom)  # a[b, j]: column j
        for _ in range(2):
            x, y, z, w = rot.unbind(1)
            m = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w),
                             2 * (x * y - z * w), 1 - 2 * (x * x + z * z), 2 * (y * z + x * w),
                             2 * (x * z + y * w), 2 * (y * z - x * w), 1 - 2 * (x * x + y * y)], 1).reshape(k, 3, 3)
            om = torch.cross(m, a, dim=2).sum(1) / ((m * a).sum((1, 2)).abs() + 1e-9)[:, None]
            wl = om.norm(dim=1, keepdim=True)
            r = torch.cat([om / wl.clamp_min(1e-30) * torch.sin(wl / 2), torch.cos(wl / 2)], 1)
            rv, rw, qv, qw = r[:, :3], r[:, 3:], rot[:, :3], rot[:, 3:]
            new = torch.cat([rw * qv + qw * rv + torch.cross(rv, qv, dim=1), rw * qw - (rv * qv).sum(1, keepdim=True)], 1)
            rot = torch.where(wl < 1e-9, rot, new / new.norm(dim=1, keepdim=True))
        target = (com + _rotate(rot[:, None, :].expand(k, n, 4), rb - rcom)).reshape(-1, 3)
        q = q * 0.2 + target * 0.8
        hit, nn, push = contact(q)
        q, prev = torch.where(hit, q + nn * push, q), torch.where(hit, prev + nn * push, prev)
        pos, v = q, (q - prev) / h * 0.995
        speed = v.norm(dim=1, keepdim=True)
        vprev, vel = vel, torch.where(speed > 40, v * (40 / speed.clamp_min(1e-30)), v)
    p = torch.from_numpy(parts.view(np.float32).reshape(-1, 24).copy()).cuda().double()
    p[:, 0:3], p[:, 4:7], p[:, 8:11], p[:, 12:15] = pos, prev, vel, vprev
    b = torch.from_numpy(bodies.view(np.float32).reshape(-1, 16).copy()).cuda().double()
    b[:, 0:3], b[:, 4:8], b[:, 8:11] = com.reshape(k, 3), rot, rcom.reshape(k, 3)
    return {"particles": p, "bodies": b}


def _exact_build(case, seed):
    """The brush fold: each 8^3 tile folds the brushes whose reach meets it, in order."""
    rec = _brushes(case, seed)
    dist, mat = [], []
    for m in range(case["mips"]):
        r, vox = case["resolution"] >> m, WORLD / case["resolution"] * 2 ** m
        bw, p, t = BAND * vox, _grid(r, WORLD, ORIGIN), r // 8
        centre = _grid(t, WORLD, ORIGIN)
        i = torch.arange(r, device="cuda") // 8
        tile = ((i[:, None, None] * t + i[None, :, None]) * t + i[None, None, :]).reshape(-1)
        ax, ay = torch.full((len(p),), 4 * bw, device="cuda", dtype=torch.float64), torch.zeros(len(p), device="cuda", dtype=torch.float64)
        for b in rec:
            f = lambda name: torch.tensor(np.atleast_1d(b[name]).astype(np.float64), device="cuda")  # noqa: E731, B023
            gap = ((f("pos") - centre).abs() - 4 * vox).clamp_min(0).norm(dim=1)
            on = (gap < float(b["bound"]) + bw)[tile]
            q = _rotate(f("rot") * torch.tensor((-1.0, -1, -1, 1), device="cuda"), p - f("pos")) / float(b["scale"])
            size, radius = f("size"), float(b["radius"])
            kind = int(b["kind"])
            if kind == 0:
                d = q.norm(dim=1) - size[0]
            elif kind == 1:
                e = q.abs() - size
                d = e.clamp_min(0).norm(dim=1) + e.max(1).values.clamp_max(0)
            elif kind == 3:
                c = torch.stack([q[:, 0], q[:, 1] - q[:, 1].clamp(-size[1], size[1]), q[:, 2]], 1)
                d = c.norm(dim=1) - radius
            else:
                d = torch.hypot(torch.hypot(q[:, 0], q[:, 2]) - size[0], q[:, 1]) - radius
            d = d * float(b["scale"])
            k = max(float(b["blend"]), 1e-6)
            if int(b["op"]) == 0:
                hh = (0.5 + 0.5 * (ax - d) / k).clamp(0, 1)
                nx, ny = ax * (1 - hh) + d * hh - k * hh * (1 - hh), ay * (1 - hh) + float(b["material"]) * hh
            else:
                hh = (0.5 - 0.5 * (ax + d) / k).clamp(0, 1)
                nx, ny = ax * (1 - hh) - d * hh + k * hh * (1 - hh), ay * (1 - 0.85 * hh) + float(b["material"]) * 0.85 * hh
            ax, ay = torch.where(on, nx, ax), torch.where(on, ny, ay)
        dist.append((ax / bw).clamp(-1, 1))
        mat.append(ay)
    return {"dist": torch.cat(dist), "mat": torch.cat(mat)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "frame":
        rec = _particles(case["n"], case["spray"], seed, tap=bool(case["tap"])).double()
        bumps = _bumps(seed)
        plane, _ = _planes(case["collider"], 1, WORLD, ORIGIN, BAND, lambda p: _terrain(p, bumps))
        p, v = rec[:, 0:3].clone(), rec[:, 4:7].clone()
        if case["tap"]:
            k = case["tap"]
            p[:k] = torch.tensor(TAP_POS, device="cuda") + _emit(k, SPACING * k ** (1 / 3) * 0.62)
            v[:k] = torch.tensor((0.0, -2.0, 0.0), device="cuda", dtype=torch.float64)
        for _ in range(case["substeps"]):
            p, dens, v, pres, nv = _substep(p, v, plane, case["collider"], 1 / 60 / case["substeps"], SMOOTHING)
        # the bake of a scene above 300,000 particles takes too long in 64 bits
        sdf = None if case["n"] > 300000 else _exact_splat(p, None, SURFACE, case["bake"], case["mips"], WORLD, ORIGIN, BAND)
        return {"pos": p, "density": dens, "vel": v, "pressure": pres, "nvel": nv, "sdf": sdf}
    if kind == "bake":
        pos, nrm, quat, radius, world, origin = _bake_cloud(case, seed)
        if nrm is not None:
            nrm = _rotate(quat.double(), nrm.double())
        return {"sdf": _exact_splat(pos.double(), nrm, radius, case["resolution"], case["mips"], world, origin, case["band"])}
    if kind == "solver":
        return _exact_solver(case, seed)
    if kind == "build":
        return _exact_build(case, seed)
    if kind == "query":
        bumps, pts = _bumps(seed), _query_points(case, seed).double()
        d, m = _planes(case["resolution"], case["mips"], WORLD, ORIGIN, BAND, lambda p: _terrain(p, bumps))
        lv = min(case["mip"], case["mips"] - 1)
        r, off = case["resolution"] >> lv, _voxels(case["resolution"], lv)
        e = (pts - torch.tensor(ORIGIN, device="cuda") - WORLD / 2).abs() - WORLD / 2
        box = e.clamp_min(0).norm(dim=1) + e.max(1).values.clamp_max(0)
        raw, mat = (_sample(x[off:off + r ** 3], r, WORLD, ORIGIN, r / WORLD, pts) for x in (d, m))
        out, bw = box > 0, BAND * WORLD / case["resolution"] * 2 ** lv
        sx = torch.where(out, box, raw * bw)
        return {"sample": torch.stack([sx, torch.where(out, 1.0, raw)], 1), "value": torch.stack([sx, torch.where(out, 0.0, mat)], 1)}
    # a batch of scenes takes too long in 64 bits; a mesh's slots follow sign tests of samples, so
    # one test that falls the other way in 64 bits moves every later record
    return None
