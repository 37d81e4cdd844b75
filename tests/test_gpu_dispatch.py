"""Which of a pass's bounces run as their own launches and which as whole paths in one launch, by the
launch counts in the stats (closest-hit launches count bounces that run as their own)."""
import pytest

from naivetrace_b200 import scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import make_params

pytestmark = pytest.mark.gpu


def _bounces(scene, spp, depth, **kw):
    """Bounces that ran as their own launches in one pass."""
    g = GpuContext(scene, make_params(max_ray_depth=depth, **kw))
    g.render(spp, seed=3)
    s = g.stats()
    assert s["error_flags"] == 0
    assert s["shadow_launches"] in (s["extend_launches"], s["extend_launches"] + 1)
    return s["extend_launches"]


# Few bounces through an atmosphere are faster as their own launches than as whole paths: waves of
# more than 8,192 paths below depth 4, and the last two bounces of larger waves.
@pytest.mark.parametrize("side,spp,depth,bounces", [(128, 1, 3, 3), (64, 2, 3, 0), (128, 1, 4, 0), (128, 2, 4, 4)])
def test_few_bounces_through_an_atmosphere(side, spp, depth, bounces):
    assert _bounces(scenes.planet_atmosphere(side, side), spp, depth) == bounces
