"""How the diffuse kernel gives voxels lanes: a lane per path in launches with few voxels (all paths up to 32, 16 lanes in
several passes for more), a lane per voxel in the others, and maps of different numbers of paths in one launch."""
import time

import numpy as np
import pytest
import torch

import doonengine_gb300 as dn
from doonengine_gb300 import configs
from parity_util import Pair
from test_gpu_walk import check_counters

pytestmark = pytest.mark.gpu


def see_through(vol):
    for m in range(0, 14, 3):
        vol.set_material(m, opacity=0.5, refract=1.2)


@pytest.mark.parametrize("glass", [False, True])
@pytest.mark.parametrize("paths", [16, 17, 34, 48, 49, 65])
def test_passes_match_oracle(gpu_ready, paths, glass):
    pair = Pair("tiny", K=3, map=(3, 2, 3), shapes=3)
    try:
        if glass:
            see_through(pair.vol)
        for _ in range(3):
            pair.draw()
            pair.sync()
            _, differ = pair.light(num_diffuse=paths)
            assert differ == 0
        check_counters(pair)
    finally:
        pair.close()


def same_lighting(a, b):
    for x, y in zip(a.export_lighting(), b.export_lighting()):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")     # (no paths: 0 / 0)


@pytest.mark.parametrize("glass", [False, True])
@pytest.mark.parametrize("counts", [(1, 1, 32, 1), (33, 1, 1, 2), (40, 17, 1, 64), (1, 5, 1, 33), (0, 3, 1, 2)])
def test_batched_mixes_match_plain(gpu_ready, counts, glass):
    dn.init()
    sizes = [(2, 2, 1), (5, 3, 4), (1, 2, 3), (4, 4, 4)]
    plain, batched = ([configs.build_volume("tiny", map=s, shapes=2, seed=80 + i)[0] for i, s in enumerate(sizes)] for _ in range(2))
    if glass:
        for v in plain + batched:
            see_through(v)
    images = [dn.Image(64, 48) for _ in plain]
    batch = dn.Batch(batched)
    try:
        for frame in range(5):
            for v, im, c in zip(plain, images, counts):
                v.draw(im, *v.view_proj(0.75))
                v.sync()
                v.update_lighting(c, 1000, 1.0 + frame)
            batch.run([dn.Batch.item(v, im, *v.view_proj(0.75), sync=(2, 1), light=(c, 1000, 1.0 + frame))
                       for v, im, c in zip(batched, images, counts)])
            assert batch.finish()
            for a, b in zip(plain, batched):
                assert a.finish()
                same_lighting(a, b)
    finally:
        batch.close()
        for x in images + plain + batched:
            x.close()


def wide_volume(limit):
    """a map with more than two voxels per lane of the diffuse launch; no voxel casts specular rays (reflect type 2), so the
    limit of their segments decides nothing but the kernels: packets and diffuse paths up to 8, ray streams above"""
    vol, _ = configs.build_volume("small", map=(32, 12, 32), seed=11, mean=0.26, amp=0.14, shapes=200, shape_max=18, K=1)
    vol.s.specBounceLimit, vol.s.diffuseBounceLimit = limit, 3
    for m in range(14):
        vol.set_material(m, specular=0.4, reflect_type=2, shininess=3)
    return vol


@pytest.mark.parametrize("glass", [False, True])
@pytest.mark.parametrize("paths", [2, 3, 33])
def test_wide_launches_match_the_streams(gpu_ready, paths, glass):
    dn.init()
    vols = [wide_volume(2), wide_volume(9), wide_volume(2)]
    if glass:
        for v in vols:
            see_through(v)
    images = [dn.Image(320, 180) for _ in vols]
    batch = dn.Batch(vols[2:])
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 7 * 128
    # views of the whole map, so that a frame lights most of its surface
    views = [(x, 0.8, z, 50.0, yaw) for x in (0.2, 0.5, 0.8) for z in (0.2, 0.5, 0.8) for yaw in (0.0, 90.0, 180.0, 270.0)]
    try:
        wide = 0
        for frame in range(6):
            for v, im in zip(vols, images):
                for view in views:
                    v.camera(*view, 90.0)
                    v.draw(im, *v.view_proj(180 / 320))
            for v in vols[:2]:
                v.sync()
                v.update_lighting(paths, 1000, 1.0 + frame)
                assert v.finish()
            batch.run([dn.Batch.item(vols[2], None, *vols[2].view_proj(180 / 320), sync=(2, 1), light=(paths, 1000, 1.0 + frame))])
            assert batch.finish()
            wide += vols[0].s.numLightingRequests * 32 > 2 * lanes
            same_lighting(vols[0], vols[1])
            same_lighting(vols[2], vols[1])
        assert wide >= 2, vols[0].s.numLightingRequests
    finally:
        batch.close()
        for x in images + vols:
            x.close()


def lighting_seconds(vol, paths):
    best = 1e9
    for _ in range(3):
        vol.finish()
        start = time.perf_counter()
        for i in range(4):
            vol.update_lighting(paths, 1000, 1.0 + i)
        vol.finish()
        best = min(best, time.perf_counter() - start)
    return best


@pytest.mark.parametrize("size,shapes", [((6, 5, 7), 6), ((16, 12, 16), 40)])
def test_one_path_more_than_a_warp(gpu_ready, size, shapes):
    """33 paths take two passes where 32 take one (or 33 after one another on a lane): far from 4 times as long"""
    dn.init()
    vol, _ = configs.build_volume("small", map=size, seed=11, mean=0.26, amp=0.14, shapes=shapes, shape_max=18, K=4)
    img = dn.Image(320, 180)
    try:
        for i in range(8):
            vol.draw(img, *vol.view_proj(180 / 320))
            vol.sync()
            vol.update_lighting(1, 1000, 0.5 + i)
        lighting_seconds(vol, 32)
        assert lighting_seconds(vol, 33) < 4.0 * lighting_seconds(vol, 32)
    finally:
        img.close()
        vol.close()


def test_small_map_of_many_paths_among_others(gpu_ready):
    """a small map's 64 paths run side by side with the others' one: the frame is far from 3 times as long as without"""
    dn.init()
    vols = [configs.build_volume("small", map=s, seed=20 + i, mean=0.26, amp=0.14, shapes=10, shape_max=18, K=4)[0]
            for i, s in enumerate([(14, 9, 14), (14, 9, 14), (3, 2, 3)])]
    images = [dn.Image(64, 48) for _ in vols]
    batch = dn.Batch(vols)
    try:
        def seconds(counts):
            items = [dn.Batch.item(v, im, *v.view_proj(0.75), sync=(2, 1), light=(c, 1000, 1.0)) for v, im, c in zip(vols, images, counts)]
            best = 1e9
            for _ in range(4):
                start = time.perf_counter()
                for _ in range(8):
                    batch.run(items)
                assert batch.finish()
                best = min(best, time.perf_counter() - start)
            return best
        seconds((1, 1, 1))
        assert seconds((1, 1, 64)) < 3.0 * seconds((1, 1, 1))
    finally:
        batch.close()
        for x in images + vols:
            x.close()
