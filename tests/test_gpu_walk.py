"""The rays' walk through the map (primary and lighting) at the sizes where its grid can go wrong: maps of one chunk, one
chunk thick, and with rows, planes and cell counts around the 16 cells of a grid word and the 32 of a warp -- opaque,
and with every third material see-through (chunks entered whose voxels the walk goes on through) -- and a map so long
that its rays' coordinates are integers (the kernels' FAR forms).  Against the oracle: hits and counters equal,
lighting bit for bit."""
import numpy as np
import pytest

import doonengine_gb300 as dn
from oracle import oracle as O
from parity_util import Pair

pytestmark = pytest.mark.gpu

COUNTERS = (("rays", "rays"), ("primaryRays", "primary"), ("outerSteps", "outerSteps"), ("chunksEntered", "chunksEntered"),
            ("innerSteps", "innerSteps"), ("hits", "hits"), ("litVoxels", "litVoxels"), ("degenerate", "degenerate"))


@pytest.mark.parametrize("glass", [False, True])
@pytest.mark.parametrize("size", [(1, 1, 1), (1, 3, 40), (31, 1, 2), (2, 15, 1), (15, 16, 17), (32, 5, 3)])
def test_walk_matches_oracle(gpu_ready, size, glass):
    pair = Pair("tiny", map=size, shapes=size[0] * size[2] // 4, res=(72, 40), K=5)
    try:
        if glass:
            for m in range(0, 14, 3):
                pair.vol.set_material(m, opacity=0.4, refract=1.3, specular=0.3, reflect_type=1, shininess=2)
        for _ in range(4):
            pair.draw()
            pair.sync()
            _, differ = pair.light(num_diffuse=2)
            assert differ == 0
        check_counters(pair)
    finally:
        pair.close()


def long_volume(length, glass):
    """1 x 2 chunks across, voxels near the far end: rays leave the map within the border's reach"""
    vol = dn.Volume((1, 2, length), 64)
    vol.palette(5, 16, 2, 0.1, 0.9, 0.5)
    rng = np.random.default_rng(5)
    z0 = length - 30
    for z in range(z0, z0 + 24):
        for _ in range(40):
            vol.set_voxel((0, 0, z), (int(rng.integers(8)), int(rng.integers(4)), int(rng.integers(8))),
                          int(rng.integers(16)), tuple(rng.normal(size=3)), tuple(int(x) for x in rng.integers(0, 256, 3)))
    if glass:
        for m in range(0, 14, 3):
            vol.set_material(m, opacity=0.4, refract=1.3, specular=0.3, reflect_type=1, shininess=2)
    vol.camera(0.3, 0.6, (z0 - 2.0) / length, 20.0, 8.0, 90.0)
    vol.s.numDirectRays = 3
    return vol


@pytest.mark.parametrize("glass", [False, True])
@pytest.mark.parametrize("length", [262141, 262143, 262200])
def test_long_map_matches_oracle(gpu_ready, length, glass):
    """262144 chunks along all axes together is the last map with coded coordinates"""
    dn.init()
    pair = Pair.__new__(Pair)
    pair.vol, pair.om = long_volume(length, glass), O.OracleMap((1, 2, length))
    pair.cfg, pair.W, pair.H, pair.frame = {}, 48, 24, 0
    pair.img = dn.Image(pair.W, pair.H)
    try:
        for _ in range(4):
            pair.draw()
            pair.sync()
            _, differ = pair.light()
            assert differ == 0
        assert pair.vol.stats()["litVoxels"] > 0
        check_counters(pair)
    finally:
        pair.close()


def test_batched_long_map_matches_plain(gpu_ready):
    """the batched FAR forms: a long map and a short one in one frame"""
    dn.init()
    plain, batched = ([long_volume(262200, True), long_volume(40, False)] for _ in range(2))
    images = [dn.Image(48, 24) for _ in range(4)]
    batch = dn.Batch(batched)
    try:
        for frame in range(4):
            for v, im in zip(plain, images):
                v.draw(im, *v.view_proj(0.5))
                v.sync()
                v.update_lighting(1, 1000, 1.0 + frame)
            batch.run([dn.Batch.item(v, im, *v.view_proj(0.5), sync=(2, 1), light=(1, 1000, 1.0 + frame))
                       for v, im in zip(batched, images[2:])])
            assert batch.finish()
            for k, (a, b) in enumerate(zip(plain, batched)):
                assert a.finish()
                for x, y in zip(a.export_lighting(), b.export_lighting()):
                    assert np.array_equal(x, y)
                for x, y in zip(images[k].numpy(), images[2 + k].numpy()):
                    assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
    finally:
        batch.close()
        for x in images + plain + batched:
            x.close()


def test_tall_image(gpu_ready):
    """more rows of blocks than a grid's y dimension holds (65535 of 8 pixels)"""
    pair = Pair("tiny", res=(2, 65535 * 8 + 9))
    try:
        for _ in range(2):
            pair.draw()
            pair.sync()
        pair.draw()
    finally:
        pair.close()


def check_counters(pair):
    st, oc = pair.vol.stats(), pair.om.counters()
    for k_gpu, k_or in COUNTERS:
        assert st[k_gpu] == oc[k_or], (k_gpu, st[k_gpu], oc[k_or])
