"""The lighting rays' walk at the sizes where its grid can go wrong: maps of one chunk, one chunk thick, and with
rows, planes and cell counts around the 16 cells of a grid word and the 32 of a warp -- opaque, and with every third
material see-through (chunks entered whose voxels the walk goes on through).  Against the oracle: hits and counters
equal, lighting bit for bit."""
import pytest

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
        st, oc = pair.vol.stats(), pair.om.counters()
        for k_gpu, k_or in COUNTERS:
            assert st[k_gpu] == oc[k_or], (k_gpu, st[k_gpu], oc[k_or])
    finally:
        pair.close()
