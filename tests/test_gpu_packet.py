"""The packet kernel's builds: specular rays of more segments than two (4- and 8-segment slots; 9 runs the ray streams) at
the fan sizes where a pool holds many voxels, one and a fraction of one; and a batch whose maps need different builds
and whose limit changes while its frame is replayed as a graph."""
import numpy as np
import pytest

import doonengine_gb300 as dn
from doonengine_gb300 import configs
from parity_util import Pair
from test_gpu_walk import check_counters

pytestmark = pytest.mark.gpu


def mirrors(vol):
    for m in range(0, 14):
        vol.set_material(m, specular=0.4 + 0.04 * m, reflect_type=m % 2, shininess=2 + m % 5)


@pytest.mark.parametrize("limit,K", [(2, 64), (3, 1), (3, 33), (4, 5), (4, 64), (5, 16), (8, 7), (8, 64), (9, 16)])
def test_specular_segments_match_oracle(gpu_ready, limit, K):
    pair = Pair("tiny", K=K)
    try:
        pair.vol.s.specBounceLimit = limit
        mirrors(pair.vol)
        for _ in range(3):
            pair.draw()
            pair.sync()
            _, differ = pair.light()
            assert differ == 0
        check_counters(pair)
    finally:
        pair.close()


def test_batched_limits_match_plain(gpu_ready):
    def build():
        out = []
        for i, limit in enumerate((2, 3, 7)):
            v, cfg = configs.build_volume("tiny", seed=40 + i)
            mirrors(v)
            v.s.specBounceLimit = limit
            out.append(v)
        return out

    dn.init()
    plain, batched = build(), build()
    W, H = 96, 64
    images = [dn.Image(W, H) for _ in plain]
    batch = dn.Batch(batched)
    try:
        for frame in range(6):
            # the last three frames repeat the composition (a replayed graph) with other limits
            if frame == 3:
                for vs in (plain, batched):
                    vs[2].s.specBounceLimit = 2
            if frame == 5:
                for vs in (plain, batched):
                    vs[0].s.specBounceLimit = 9
            for v, im in zip(plain, images):
                v.draw(im, *v.view_proj(H / W))
                v.sync()
                v.update_lighting(1, 1000, 1.0 + frame)
            batch.run([dn.Batch.item(v, im, *v.view_proj(H / W), sync=(2, 1), light=(1, 1000, 1.0 + frame))
                       for v, im in zip(batched, images)])
            assert batch.finish()
            for a, b in zip(plain, batched):
                assert a.finish()
                for x, y in zip(a.export_lighting(), b.export_lighting()):
                    assert np.array_equal(x, y)
    finally:
        batch.close()
        for im in images:
            im.close()
        for v in plain + batched:
            v.close()


@pytest.mark.parametrize("paths,bounces", [(1, 1), (3, 6)])
@pytest.mark.parametrize("rng", [0, 1])
def test_path_directions_match_oracle(gpu_ready, rng, paths, bounces):
    """sphere points drawn by a warp for its lanes: both generators, first segments only and many bounces"""
    pair = Pair("tiny", K=5)
    try:
        pair.vol.s.rngMode, pair.vol.s.diffuseBounceLimit = rng, bounces
        mirrors(pair.vol)
        for _ in range(3):
            pair.draw()
            pair.sync()
            _, differ = pair.light(num_diffuse=paths)
            assert differ == 0
        check_counters(pair)
    finally:
        pair.close()


def test_batched_generators_match_plain(gpu_ready):
    """maps of both generators in one batch: a warp's voxels come from both"""
    def build():
        out = []
        for i in range(6):
            v, _ = configs.build_volume("tiny", map=(1 + i, 2, 2), shapes=1 + i, seed=60 + i)
            v.s.rngMode = i % 2
            out.append(v)
        return out

    dn.init()
    plain, batched = build(), build()
    images = [dn.Image(96, 64) for _ in plain]
    batch = dn.Batch(batched)
    try:
        for frame in range(4):
            for v, im in zip(plain, images):
                v.draw(im, *v.view_proj(64 / 96))
                v.sync()
                v.update_lighting(2, 1000, 1.0 + frame)
            batch.run([dn.Batch.item(v, im, *v.view_proj(64 / 96), sync=(2, 1), light=(2, 1000, 1.0 + frame))
                       for v, im in zip(batched, images)])
            assert batch.finish()
            for a, b in zip(plain, batched):
                assert a.finish()
                for x, y in zip(a.export_lighting(), b.export_lighting()):
                    assert np.array_equal(x, y)
    finally:
        batch.close()
        for x in images + plain + batched:
            x.close()


@pytest.mark.parametrize("paths", [2, 3, 31, 32, 33])
@pytest.mark.parametrize("bounces", [0, 4])
def test_paths_side_by_side_match_oracle(gpu_ready, paths, bounces):
    """small launches give each of a voxel's paths a lane (up to 32 paths, at least one bounce)"""
    pair = Pair("tiny", K=3, map=(3, 2, 3), shapes=3)
    try:
        pair.vol.s.diffuseBounceLimit = bounces
        for m in range(0, 14, 3):
            pair.vol.set_material(m, opacity=0.5, refract=1.2)
        mirrors(pair.vol)
        for _ in range(3):
            pair.draw()
            pair.sync()
            _, differ = pair.light(num_diffuse=paths)
            assert differ == 0
        check_counters(pair)
    finally:
        pair.close()


def test_batched_path_counts_match_plain(gpu_ready):
    """maps with different numbers of paths in one batch, and a repeated composition whose count changes"""
    dn.init()
    plain, batched = ([configs.build_volume("tiny", map=(2, 2, 1 + i), shapes=2, seed=80 + i)[0] for i in range(4)] for _ in range(2))
    images = [dn.Image(64, 48) for _ in plain]
    batch = dn.Batch(batched)
    try:
        for frame in range(6):
            counts = (1, 1, 1, 1) if frame in (2, 5) else (1, 3, 40, 2)
            for v, im, c in zip(plain, images, counts):
                v.draw(im, *v.view_proj(0.75))
                v.sync()
                v.update_lighting(c, 1000, 1.0 + frame)
            batch.run([dn.Batch.item(v, im, *v.view_proj(0.75), sync=(2, 1), light=(c, 1000, 1.0 + frame))
                       for v, im, c in zip(batched, images, counts)])
            assert batch.finish()
            for a, b in zip(plain, batched):
                assert a.finish()
                for x, y in zip(a.export_lighting(), b.export_lighting()):
                    assert np.array_equal(x, y)
    finally:
        batch.close()
        for x in images + plain + batched:
            x.close()
