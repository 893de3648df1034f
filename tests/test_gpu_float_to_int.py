"""Conversions of floats outside int32 (f2i saturates, the oracle's defines it so): the sine generator's quadrant at times
whose quadrants are numbered beyond 2^31."""
import pytest

from parity_util import Pair
from test_gpu_walk import check_counters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("time", [3.0e9, -3.5e9, 2.0e10])
def test_sine_generator_at_large_times(gpu_ready, time):
    pair = Pair("tiny", K=5)
    try:
        pair.vol.s.rngMode = 1
        for m in range(14):
            pair.vol.set_material(m, specular=0.5, reflect_type=m % 2, shininess=3)
        for _ in range(3):
            pair.draw()
            pair.sync()
            _, differ = pair.light(num_diffuse=2, time=time)
            assert differ == 0
        check_counters(pair)
    finally:
        pair.close()
