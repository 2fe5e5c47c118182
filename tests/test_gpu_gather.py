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


def test_gathered_surface_of_many_chunks_equals_splatted(root):
    """A small dense scene with a surface of more than 131,072 chunks of 8^3 voxels: its super-groups are counted, and a
    chunk's number times their 32,768 particles (which passes 2^32 there) decides nothing."""
    import clay_engine_b200 as ce

    wanted = [("pile", 8192, 8200, 416, 2), ("pile", 40000, 255000, 64, 2)]
    assert (416 // 8) ** 3 + (208 // 8) ** 3 > 1 << 17 and sum(c for _, _, c, _, _ in wanted) >= 1 << 18
    together, alone = make(root, "reference", wanted), make(root, "reference", wanted)
    b = ce.Batch(root, together)
    b.step()
    for i, (x, y) in enumerate(zip(together, alone)):
        y.step()
        gd, ad = x.surface.volume.download()[0], y.surface.volume.download()[0]
        assert np.array_equal(gd, ad), f"scene {i}: {(gd != ad).sum()} voxels differ"
        assert (ad != 0x3C00).any()
    for o in [b] + together + alone:
        o.destroy()
