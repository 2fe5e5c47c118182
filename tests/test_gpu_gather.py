"""The gather bake (box tree over the cell-ordered cloud, every voxel finds its nearest particle)
against the splat of the same scenes, bit for bit: a batch of 2^18 particles and more lets the
device choose per scene, a scene of its own below 2^17 particles is splatted (and the splat is held
to the oracle in test_gpu_bake.py and test_gpu_configs.py, as is the gather of a large single scene)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORIGIN = (-12.0, -4.0, -12.0)


def particles(kind, n, seed):
    from clay_engine_b200 import scenes
    from clay_engine_b200.core import PARTICLE_DTYPE

    rng = np.random.default_rng(seed)
    if kind == "pile":  # dense: two particles a cell and more
        p = scenes.lattice_block(n, 0.1, (0.3, 2.0, -0.7), seed)
    else:  # thin spray over the whole volume, some of it outside
        p = np.zeros(n, PARTICLE_DTYPE)
        p["pos"] = rng.uniform((-12.5, -4.5, -12.5), (12.5, 20.5, 12.5), (n, 3))
    p["vel"] = rng.normal(0, 1, (n, 3))
    return p


# (kind, live, capacity, bake resolution, levels): around a leaf of 32, a group of 1,024, the bound of
# the Morton order (8,192) and of a super-group (32,768), scenes that stay splatted among them
SCENES = [("pile", 130000, 131071, 64, 3), ("pile", 40000, 40000, 64, 2), ("pile", 32769, 65000, 128, 4), ("pile", 8193, 8193, 8, 1),
          ("pile", 8192, 8192, 32, 2), ("pile", 1025, 1100, 40, 1), ("pile", 65, 65, 24, 1), ("pile", 63, 63, 32, 1),
          ("spray", 4100, 20000, 32, 2), ("spray", 60000, 70000, 32, 1), ("spray", 3000, 3000, 64, 3), ("pile", 0, 5000, 32, 2)]


def make(root, mode, wanted=SCENES):
    import clay_engine_b200 as ce

    sims = []
    for i, (kind, live, cap, res, mips) in enumerate(wanted):
        s = ce.FluidSim(root, None, dict(capacity=cap, spacing=0.1, radius=0.05, substeps=2, bakeResolution=res,
                                         bakeMipLevels=mips, bakeBand=(2.0, 4.0, 3.0)[i % 3], worldSize=24.0, origin=ORIGIN))
        s.set_mode(mode)
        s.upload(particles(kind, live, 30 + i))
        sims.append(s)
    return sims


@pytest.mark.parametrize("lanes", [1, 2, 0])
def test_gathered_batch_equals_splatted_scenes(root, lanes):
    """lanes 0: the listed scenes of a batch frame (step_subset), else a whole frame in that many lanes."""
    import torch

    import clay_engine_b200 as ce

    assert sum(n for _, n, _, _, _ in SCENES) >= 1 << 18 and max(c for _, _, c, _, _ in SCENES) < 1 << 17
    together, alone = make(root, "reference"), make(root, "reference")
    b = ce.Batch(root, together)
    if lanes:
        b.set_lanes(lanes)
    keys = torch.zeros(together[0].surface.volume.totalVoxels, dtype=torch.int32, device="cuda")
    together[0].surface.capture_keys(keys)
    for _ in range(2):
        if lanes:
            b.step()
        else:
            b.step_subset(list(range(len(together))))
        for s in alone:
            s.step()
    torch.cuda.synchronize()
    assert (keys.cpu().numpy() < 65535).any()
    for i, (x, y) in enumerate(zip(together, alone)):
        gd, ad = x.surface.volume.download()[0], y.surface.volume.download()[0]
        assert np.array_equal(gd, ad), f"scene {i} {SCENES[i]}: {(gd != ad).sum()} voxels differ"
        assert (ad != 0x3C00).any() == (SCENES[i][1] > 0)
    for o in [b] + together + alone:
        o.destroy()


def mist(n, spacing, center, seed):
    """Particles at random places of a cube, `spacing` apart on average, in no order."""
    from clay_engine_b200.core import PARTICLE_DTYPE

    p, half = np.zeros(n, PARTICLE_DTYPE), 0.5 * spacing * n ** (1 / 3)
    p["pos"] = np.random.default_rng(seed).uniform(-half, half, (n, 3)) + center
    return p


def is_gathered(p, res):
    """The rule by which the device gathers a surface that its launches let it choose for."""
    c = np.floor((p["pos"].astype(np.float64) - ORIGIN) / 0.22).astype(np.int64)  # smoothing 2.2 x the spacing of 0.1
    box = c.max(0) - c.min(0) + 1
    at = np.unique(np.ravel_multi_index((c - c.min(0)).T[::-1], box[::-1]))
    n, cells, occupied = len(p), int(np.prod(box)), len(at)
    held = min(128 * len(np.unique(at // 128)), cells)
    return n >= (4096 if res >= 64 else 8192) and (n >= 2 * cells or (8 * n >= res ** 3 and (5 * n >= 6 * cells or 3 * occupied >= held)))


def surface_sim(root, p, res, mips, band=3.0, capacity=None):
    import clay_engine_b200 as ce

    s = ce.FluidSim(root, None, dict(capacity=capacity or len(p), spacing=0.1, radius=0.05, substeps=1, gravity=(0, 0, 0), bakeResolution=res,
                                     bakeMipLevels=mips, bakeBand=band, worldSize=24.0, origin=ORIGIN))
    s.upload(p)
    return s


# (spacing: dense pile or mist, live, resolution, levels): around a super-group (32,768), partly filled leaves and groups, one
# level and several, levels of 8^3
GATHERED = [("pile", 0.1, 4096, 64, 2), ("pile", 0.1, 8192, 32, 2), ("pile", 0.1, 8193, 8, 1), ("pile", 0.1, 32768, 64, 2), ("pile", 0.1, 32769, 128, 4),
            ("mist", 0.2, 33000, 64, 3), ("mist", 0.18, 9999, 40, 1), ("pile", 0.1, 250000, 96, 3), ("mist", 0.17, 130000, 64, 3)]


@pytest.mark.parametrize("lanes", [1, 3, 0])
def test_gathered_scenes_of_a_batch_equal_splatted(root, lanes):
    """Scenes that the device gathers in a batch, and the same ones splatted by themselves (a scene alone of fewer than 2^18
    particles is). lanes 0: step_subset."""
    import clay_engine_b200 as ce
    from clay_engine_b200 import scenes

    clouds = []
    for i, (kind, spacing, n, res, mips) in enumerate(GATHERED):
        p = scenes.lattice_block(n, spacing, (0.3, 2.0, -0.7), i) if kind == "pile" else mist(n, spacing, (0.0, 5.0, 0.0), i)
        assert is_gathered(p, res) and n < 1 << 18
        clouds.append(p)
    assert sum(len(p) for p in clouds) >= 3 << 17
    together, alone = ([surface_sim(root, p, g[3], g[4], (2.0, 4.0, 3.0)[i % 3], len(p) + 5 * i) for i, (p, g) in enumerate(zip(clouds, GATHERED))]
                       for _ in range(2))
    b = ce.Batch(root, together)
    b.set_lanes(max(lanes, 1))
    for _ in range(2):
        if lanes:
            b.step()
        else:
            b.step_subset(list(range(len(together))))
        for s in alone:
            s.step()
    for i, (x, y) in enumerate(zip(together, alone)):
        gd, ad = x.surface.volume.download()[0], y.surface.volume.download()[0]
        assert np.array_equal(gd, ad), f"scene {i} {GATHERED[i]}: {(gd != ad).sum()} voxels differ"
        assert (ad != 0x3C00).any()
    for o in [b] + together + alone:
        o.destroy()


@pytest.mark.parametrize("kind,spacing,n,res,mips,gathered", [("mist", 0.2, 1 << 18, 64, 3, True), ("mist", 0.2, 270001, 128, 2, True),
                                                              ("pile", 0.1, 300000, 64, 3, True), ("mist", 0.2, 300000, 192, 1, False),
                                                              ("pile", 0.09, 1 << 19, 32, 2, True), ("spray", 0.0, 300000, 64, 3, False),
                                                              ("stream", 0.22, 300000, 64, 3, True)])
def test_large_scene_alone_equals_splatted(root, kind, spacing, n, res, mips, gathered):
    """A scene by itself at the sizes from which the device may choose, on either side of its rule, against its cloud baked
    by a SplatField of its own."""
    import torch

    import clay_engine_b200 as ce
    from clay_engine_b200 import scenes

    p = scenes.lattice_block(n, spacing, (0.0, 4.0, 0.0), n) if kind == "pile" else mist(n, spacing, (0.0, 6.0, 0.0), n)
    if kind == "spray":  # a pile, and a tenth of it as a thin spray over the world
        p = scenes.lattice_block(n, 0.1, (0.0, 1.0, 0.0), n)
        p["pos"][::10] = np.random.default_rng(n).uniform((-11, -3, -11), (11, 19, 11), (len(p[::10]), 3))
    if kind == "stream":  # a thin one falls into the mist, from as high again
        p["pos"][:3000] = np.random.default_rng(n).normal((0.0, 14.0, 0.0), (0.1, 2.0, 0.1), (3000, 3))
    assert is_gathered(p, res) == gathered
    sim = surface_sim(root, p, res, mips)
    for _ in range(2):
        sim.step()
    now = torch.from_numpy(np.ascontiguousarray(sim.download()["pos"])).cuda()
    splat = ce.SplatField(root, ce.ParticleCloud(n, now), radius=0.1 * 1.1, resolution=res, mipLevels=mips, band=3.0, worldSize=24.0,
                          origin=ORIGIN)
    splat.bake()
    gd, ad = sim.surface.volume.download()[0], splat.volume.download()[0]
    assert np.array_equal(gd, ad), f"{(gd != ad).sum()} voxels differ"
    assert (ad != 0x3C00).any()
    for o in (sim, splat):
        o.destroy()


def test_gathered_surface_of_many_chunks_equals_splatted(root):
    """A dense scene with a surface of more than 131,072 chunks of 8^3 voxels: its super-groups are counted, and a chunk's
    number times their 32,768 particles (which passes 2^32 there) decides nothing."""
    import clay_engine_b200 as ce
    from clay_engine_b200 import scenes

    assert (416 // 8) ** 3 + (208 // 8) ** 3 > 1 << 17
    clouds = [scenes.lattice_block(n, 0.1, (0.3, 2.0, -0.7), n) for n in (9000, 400000)]
    assert is_gathered(clouds[0], 416)
    together = [surface_sim(root, p, r, 2) for p, r in zip(clouds, (416, 64))]
    alone = surface_sim(root, clouds[0], 416, 2)
    b = ce.Batch(root, together)
    b.step()
    alone.step()
    gd, ad = together[0].surface.volume.download()[0], alone.surface.volume.download()[0]
    assert np.array_equal(gd, ad), f"{(gd != ad).sum()} voxels differ"
    assert (ad != 0x3C00).any()
    for o in [b, alone] + together:
        o.destroy()


def test_choice_under_capture(root):
    """A frame that may choose, captured by the caller: the branch joins the captured stream, and replays equal plain frames
    where the device gathers and where it splats."""
    import torch

    import clay_engine_b200 as ce

    n = 1 << 18
    cloud = mist(n, 0.2, (0.0, 6.0, 0.0), 1)
    far = cloud.copy()
    far["pos"][::2] = np.random.default_rng(2).uniform((-11, -3, -11), (11, 19, 11), (n // 2, 3))
    assert is_gathered(cloud, 64) and not is_gathered(far, 64)
    captured, plain = surface_sim(root, cloud, 64, 2), surface_sim(root, cloud, 64, 2)
    stream = torch.cuda.Stream()
    captured.step(stream.cuda_stream)  # uploads what the frame reads
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        captured.step(torch.cuda.current_stream().cuda_stream)
    for p in (cloud, far):
        captured.upload(p)
        plain.upload(p)
        torch.cuda.synchronize()
        graph.replay()
        plain.step()
        torch.cuda.synchronize()
        assert np.array_equal(captured.download()["pos"], plain.download()["pos"])
        gd, ad = captured.surface.volume.download()[0], plain.surface.volume.download()[0]
        assert np.array_equal(gd, ad) and (ad != 0x3C00).any()
    del graph
    for o in (captured, plain):
        o.destroy()
