"""Medium tracking of scenes with an atmosphere: large waves track with refilled lanes, small ones
with one path per lane.  The same paths, bit for bit."""
import numpy as np
import pytest

from naivetrace_b200 import scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import make_params

pytestmark = pytest.mark.gpu

SIDE = 512  # 262,144 pixels: more than two paths per resident lane in one wave


def _accumulators(wave_paths, **range_):
    g = GpuContext(scenes.planet_atmosphere(SIDE, SIDE), make_params(max_ray_depth=5, wave_paths=wave_paths))
    g.render(1, seed=11, **range_)
    assert g.stats()["error_flags"] == 0
    return g.accumulators()[0]


# Waves of one sample per pixel, so that a pixel has one summand however the waves are cut: one
# wave (refilled), three, and one with a ragged rest of few paths.
@pytest.mark.parametrize("wave_paths", [100_000, SIDE * SIDE - 1, 151_553])
def test_refilled_tracking_equals_one_path_per_lane(wave_paths):
    assert np.array_equal(_accumulators(0), _accumulators(wave_paths))


def test_refilled_tracking_in_a_range():
    a = _accumulators(0, pixel_begin=7, pixel_end=SIDE * SIDE - 5)
    assert np.array_equal(a, _accumulators(50_001, pixel_begin=7, pixel_end=SIDE * SIDE - 5))
    assert np.any(a != 0)
