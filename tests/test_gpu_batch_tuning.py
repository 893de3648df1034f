"""The tuning of a batch (dn_cuda_batch_set_tuning, dn_cuda_batch_autotune) across frames of different kinds."""
import pytest

import doonengine_gb300 as dn
from doonengine_gb300 import configs

pytestmark = pytest.mark.gpu


class Maps:
    """a batch of small maps, each with an image"""

    def __init__(self, n=3, **settings):
        dn.init()
        self.vols = [configs.build_volume("tiny", map=(3 + i, 3, 4), shapes=3, seed=30 + i)[0] for i in range(n)]
        for v in self.vols:
            for k, x in settings.items():
                setattr(v.s, k, x)
        self.images = [dn.Image(64, 48) for _ in self.vols]
        self.batch = dn.Batch(self.vols)
        self.time = 0.5

    def frame(self, light=True, paths=1):
        self.time += 0.25
        self.batch.run([dn.Batch.item(v, im, *v.view_proj(0.75), sync=(2, 1) if light else None,
                                      light=(paths, 1000, self.time) if light else None)
                        for v, im in zip(self.vols, self.images)])
        assert self.batch.finish(), dn.load().dn_cuda_last_error().decode()

    def close(self):
        self.batch.close()
        for x in self.images + self.vols:
            x.close()


def test_autotune_needs_a_lit_last_frame(gpu_ready):
    """the launch that autotuning runs again reads the frame's table, which a frame without lighting has replaced"""
    maps = Maps()
    try:
        for k in range(3):          # the first two frames are issued, the third is a replayed graph
            for _ in range(k + 1):
                maps.frame()
            maps.batch.autotune()
            for _ in range(k + 1):
                maps.frame(light=False)
            with pytest.raises(RuntimeError):
                maps.batch.autotune()
        maps.frame()
        maps.batch.autotune()
    finally:
        maps.close()


def test_overflowed_list_counts_alike(gpu_ready):
    """more requests than a member's list holds: the batch and the map alone report what the list holds"""
    dn.init()
    vol, _ = configs.build_volume("small", map=(16, 12, 16), seed=11, mean=0.26, amp=0.14, shapes=40, shape_max=18, K=1)
    vol.s.lightingRequestCap = 1 << 30      # the host takes the device's list for long enough and never grows it
    img = dn.Image(320, 180)
    batch = dn.Batch([vol])
    try:
        for i in range(10):
            vol.draw(img, *vol.view_proj(180 / 320))
            vol.sync()
            vol.update_lighting(1, 1000, 1.0 + i)
        vol.draw(img, *vol.view_proj(180 / 320))
        vol.sync()
        assert not batch.finish()           # the overflow is reported
        assert vol.s.numLightingRequests == 1024
        vol.finish()                        # (an error is reported once)
        assert vol.s.numLightingRequests == 1024
    finally:
        batch.close()
        img.close()
        vol.close()


@pytest.mark.parametrize("change", [dict(poolRays=64), dict(diffuseBatch=7), dict(streamBatch=9), dict(blocksPerSM=1)])
def test_tuning_change_renews_the_graph(gpu_ready, change):
    """a repeated frame is replayed as a graph; a setting that the launches in it hold needs another"""
    maps = Maps()
    captures = lambda: maps.batch.lib.dn_cuda_batch_captures(maps.batch._gpu())
    try:
        maps.batch.set_tuning(poolRays=128, diffuseBatch=20, streamBatch=16, blocksPerSM=2, useGraph=1)
        for _ in range(4):
            maps.frame()
        assert captures() == 1
        maps.batch.set_tuning(**change)
        for _ in range(4):
            maps.frame()
        assert captures() == 2
    finally:
        maps.close()


@pytest.mark.parametrize("settings", [{}, {"specBounceLimit": 9}])     # packets and diffuse paths, ray streams
@pytest.mark.parametrize("light", [True, False])
def test_replayed_frame_counts_its_launches(gpu_ready, light, settings):
    """a frame counts the same kernels whether it is issued or replayed as a graph"""
    maps = Maps(**settings)
    count = maps.batch.lib.dn_cuda_launch_count
    try:
        for _ in range(6):      # the maps load
            maps.frame(light)
        counts = []
        for graph in (1, 0):
            maps.batch.set_tuning(useGraph=graph)
            before = count()
            maps.frame(light)
            counts.append(count() - before)
        assert counts[0] == counts[1] > 0, counts
    finally:
        maps.close()


@pytest.mark.parametrize("limit", [4, 8])
def test_autotune_keeps_a_pool_size_that_has_no_effect(gpu_ready, limit):
    """only the packet build of two segments has two pool sizes; for the others a trial of the second times the same
    kernel again, and would be chosen by chance"""
    maps = Maps(specBounceLimit=limit)
    try:
        for pool in (128, 64):
            for _ in range(6):
                maps.batch.set_tuning(poolRays=pool, kernel=2, streamBatch=16, blocksPerSM=2)
                maps.frame()
                assert maps.batch.autotune()["poolRays"] == pool
    finally:
        maps.close()
