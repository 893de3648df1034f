"""Lighting of maps whose chunks are too many along their axes for coded coordinates (the kernels' FAR forms): packets up to
the reference's limit of specular segments, ray streams above it, alone and in a batch with a small map."""
import numpy as np
import pytest

import doonengine_gb300 as dn
from oracle import oracle as O
from parity_util import Pair
from test_gpu_walk import check_counters, long_volume

pytestmark = pytest.mark.gpu

LENGTH = 262200


def long_pair(length, glass, K, limit):
    dn.init()
    pair = Pair.__new__(Pair)
    pair.vol, pair.om = long_volume(length, glass), O.OracleMap((1, 2, length))
    pair.vol.s.numDirectRays, pair.vol.s.specBounceLimit = K, limit
    for m in range(0, 14, 2):
        pair.vol.set_material(m, specular=0.5, reflect_type=1, shininess=3)
    pair.cfg, pair.W, pair.H, pair.frame = {}, 48, 24, 0
    pair.img = dn.Image(pair.W, pair.H)
    return pair


@pytest.mark.parametrize("glass", [False, True])
@pytest.mark.parametrize("limit,K,paths", [(0, 5, 1), (1, 64, 2), (2, 33, 3), (3, 7, 2), (9, 4, 1)])
def test_long_map_lighting_matches_oracle(gpu_ready, limit, K, paths, glass):
    pair = long_pair(LENGTH, glass, K, limit)
    try:
        for _ in range(4):
            pair.draw()
            pair.sync()
            _, differ = pair.light(num_diffuse=paths)
            assert differ == 0
        assert pair.vol.stats()["litVoxels"] > 0
        check_counters(pair)
    finally:
        pair.close()


@pytest.mark.parametrize("limit", [1, 2])
def test_long_maps_take_the_packets(gpu_ready, limit):
    """a lighting update of a long map runs the kernels that one of a short map runs"""
    counts = []
    for length in (40, LENGTH):
        vol = long_volume(length, False)
        vol.s.specBounceLimit = limit
        before = vol.lib.dn_cuda_launch_count()
        vol.update_lighting(1, 1000, 1.0)
        vol.finish()
        counts.append(vol.lib.dn_cuda_launch_count() - before)
        vol.close()
    assert counts[0] == counts[1] == 4      # preparation, packets, diffuse paths, commit


@pytest.mark.parametrize("limits", [(2, 2), (1, 4), (9, 2)])
def test_batched_long_map_lighting_matches_plain(gpu_ready, limits):
    dn.init()
    plain, batched = ([long_volume(LENGTH, True), long_volume(40, False)] for _ in range(2))
    for vols in (plain, batched):
        for v, limit in zip(vols, limits):
            v.s.specBounceLimit, v.s.numDirectRays = limit, 17
    images = [dn.Image(48, 24) for _ in range(2)]
    batch = dn.Batch(batched)
    try:
        for frame in range(5):
            for v, im in zip(plain, images):
                v.draw(im, *v.view_proj(0.5))
                v.sync()
                v.update_lighting(2, 1000, 1.0 + frame)
            batch.run([dn.Batch.item(v, im, *v.view_proj(0.5), sync=(2, 1), light=(2, 1000, 1.0 + frame))
                       for v, im in zip(batched, images)])
            assert batch.finish()
            if frame == 2:
                batch.autotune()
            for a, b in zip(plain, batched):
                assert a.finish()
                for x, y in zip(a.export_lighting(), b.export_lighting()):
                    assert np.array_equal(x, y)
    finally:
        batch.close()
        for x in images + plain + batched:
            x.close()
