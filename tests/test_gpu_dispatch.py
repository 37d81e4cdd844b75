"""Which of a pass's bounces run as their own launches and which as whole paths in one launch, by the
launch counts in the stats (closest-hit launches count bounces that run as their own)."""
import pytest

from naivetrace_b200 import abi, scenes
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


# Waves of at most 16,384 paths run as whole paths from their camera samples, in scenes without media,
# sorted shading or byte boxes of at most 65,536.
@pytest.mark.parametrize("name,limit", [("cornell_box", 1 << 16), ("guiding_room", 1 << 16),
                                        ("cornell_box_materials", 1 << 14), ("spheres_box", 1 << 14),
                                        ("cornell_box_media_mix", 1 << 14), ("planet_atmosphere", 1 << 14)])
def test_limit_of_whole_waves(name, limit):
    spp = limit // (64 * 64)
    assert _bounces(getattr(scenes, name)(64, 64), spp, 9) == 0
    assert _bounces(getattr(scenes, name)(64, 64), spp + 1, 9) >= 2
    assert _bounces(getattr(scenes, name)(64, 64), spp, 9, algo=abi.ALGO_PT2) == 9


# Few bounces through an atmosphere are faster as their own launches than as whole paths: waves of
# more than 8,192 paths below depth 4, and the last two bounces of larger waves.
@pytest.mark.parametrize("side,spp,depth,bounces", [(128, 1, 3, 3), (64, 2, 3, 0), (128, 1, 4, 0), (128, 2, 4, 4)])
def test_few_bounces_through_an_atmosphere(side, spp, depth, bounces):
    assert _bounces(scenes.planet_atmosphere(side, side), spp, depth) == bounces


@pytest.mark.parametrize("side,spp,bounces", [(64, 1, 0), (320, 2, None)])
def test_launch_counts_of_a_pass(side, spp, bounces):
    """Cornell box (no media, one shader kind): every launch of the pass is counted once."""
    depth = 12
    plain = GpuContext(scenes.cornell_box(side, side), make_params(max_ray_depth=depth))
    plain.render(spp, seed=3)
    s = plain.stats()
    own = s["extend_launches"]
    if bounces is None:
        assert 2 <= own < depth  # ended as whole paths
        # generate; shadow, extend, shade per bounce; shadow, whole paths; gather, tally, accumulate.
        assert s["kernel_launches"] == 1 + 3 * own + 2 + 3
        assert s["shadow_launches"] == own + 1
    else:
        assert own == bounces and s["shadow_launches"] == 0
        assert s["kernel_launches"] == 1 + 3  # whole paths; gather, tally, accumulate
    profiled = GpuContext(scenes.cornell_box(side, side), make_params(max_ray_depth=depth))
    profiled.set_profiling(1)
    profiled.render(spp, seed=3)
    s = profiled.stats()
    assert (s["extend_launches"], s["shadow_launches"]) == (depth, depth + 1)
    assert s["kernel_launches"] == 1 + 3 * depth + 1 + 3


def test_launch_counts_of_view_batches():
    """The first wave of a batch may end as whole paths, the later (captured) ones launch every bounce;
    with profiling on all waves do.  The rays are the same."""
    depth = 12
    views = [(scenes.CameraSpec(pos=(0.5, 0.5, -1.4 - 0.1 * k), dir=(0, 0, 1), xres=150, yres=100), 5) for k in range(2)]
    rays = []
    for wave_paths, profiling, waves in ((0, 0, 1), (70_000, 0, 3), (70_000, 1, 3)):
        g = GpuContext(scenes.cornell_box(16, 16), make_params(max_ray_depth=depth, wave_paths=wave_paths))
        g.set_profiling(profiling)
        g.render_views(views, seed=3)
        s = g.stats()
        first = s["extend_launches"] - (waves - 1) * depth
        assert first == depth if profiling else 2 <= first < depth
        assert s["shadow_launches"] == first + 1 + (waves - 1) * (depth + 1)
        rays.append([s[k] for k in ("paths", "extension_rays", "shadow_rays")])
    assert rays[0] == rays[1] == rays[2]


# Paths at which the last bounces of a wave are handed over: 65,536 in scenes without media that do not
# sort their hits or have byte boxes (16,384 primitives on), else 16,384.
@pytest.mark.parametrize("name,limit", [("terrain", 1 << 16), ("cornell", 1 << 16), ("materials", 1 << 14),
                                        ("media", 1 << 14)])
def test_limit_of_the_last_paths(name, limit):
    depth = 14
    scene = {"terrain": lambda x, y: scenes.terrain_spheres(x, y, terrain_n=128, sphere_level=2, num_spheres=32,
                                                            env_w=64, env_h=32),
             "cornell": scenes.cornell_box, "materials": scenes.cornell_box_materials,
             "media": scenes.cornell_box_media_mix}[name](500, 300)
    g = GpuContext(scene, make_params(max_ray_depth=depth))
    assert (g.stats()["bvh_node_bytes"] == 64) == (name == "terrain")
    g.render(1, seed=3)
    lengths = [int(q) for q in g.queue_lengths(depth)[:, 0]]
    # From the third bounce on, by the length of the bounce before.
    first = next((b for b in range(2, depth) if lengths[b - 1] <= limit), depth)
    assert g.stats()["extend_launches"] == first
    assert lengths[0] > (1 << 16)
