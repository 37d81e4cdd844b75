"""Whole paths in one launch (small waves, and the last paths of larger ones) against the wavefront
kernels, which run when launches are timed: the same paths, bit for bit."""
import numpy as np
import pytest

from naivetrace_b200 import scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import make_params

pytestmark = pytest.mark.gpu

# Paths up to which a wave runs as whole paths from its camera samples: in any scene, and in a small
# uniform one (also the limits of the last bounces' paths).
WHOLE, WHOLE_UNIFORM = 1 << 14, 1 << 16


def _render(scene, params, spp, wavefront, rng=None, guide=False):
    g = GpuContext(scene, params)
    if guide:
        g.set_guiding(True, train=0, max_depth=2)
        w = np.random.default_rng(3).normal(scale=0.2, size=g.lib.tt_guide_num_params())
        g.guide_set_params(w.astype(np.float32))
    g.set_profiling(1 if wavefront else 0)
    g.render(spp, seed=5, **({} if rng is None else {"pixel_begin": rng[0], "pixel_end": rng[1]}))
    acc, light, _, _ = g.accumulators()
    return acc, light, g.stats(), g.queue_lengths(params.max_ray_depth + 1)


def _same(scene, params, spp, **kw):
    a, la, sa, qa = _render(scene, params, spp, True, **kw)
    b, lb, sb, qb = _render(scene, params, spp, False, **kw)
    assert np.array_equal(a, b)
    # Camera splats are added by float atomics in any order.
    assert np.allclose(la, lb, rtol=1e-5, atol=1e-6 * max(1e-30, np.abs(la).max()))
    for k in ("extension_rays", "shadow_rays", "paths"):
        assert sa[k] == sb[k]
    assert np.array_equal(qa, qb)
    assert sb["error_flags"] == 0


SCENES = {
    "materials": scenes.cornell_box_materials,
    "media": scenes.cornell_box_media_mix,
    "spheres": scenes.spheres_box,
    "planet": scenes.planet_atmosphere,
    "terrain": lambda x, y: scenes.terrain_spheres(x, y, terrain_n=128, sphere_level=2, num_spheres=8, env_w=64,
                                                   env_h=32),
}


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("xres,yres,spp", [(1, 1, 1), (31, 1, 1), (33, 3, 5), (64, 64, 3)])
def test_whole_paths(name, xres, yres, spp):
    _same(SCENES[name](xres, yres), make_params(max_ray_depth=9), spp)


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("spp", [3, 4, 5, 31, 32, 33])  # 64 x 64 x 4 = WHOLE
def test_around_the_limit(name, spp):
    assert 64 * 64 * 4 == WHOLE
    _same(SCENES[name](64, 64), make_params(max_ray_depth=12), spp)


@pytest.mark.parametrize("spp", [15, 16, 17])  # 64 x 64 x 16 = WHOLE_UNIFORM
def test_around_the_uniform_limit(spp):
    assert 64 * 64 * 16 == WHOLE_UNIFORM
    _same(scenes.cornell_box(64, 64), make_params(max_ray_depth=12), spp)


@pytest.mark.parametrize("depth", [1, 2, 3, 1000])
def test_depths(depth):
    _same(scenes.cornell_box(40, 30), make_params(max_ray_depth=depth), 2)
    _same(scenes.cornell_box(400, 330), make_params(max_ray_depth=depth), 2)


def test_waves_and_ranges():
    s = scenes.cornell_box_materials(50, 40)
    _same(s, make_params(max_ray_depth=8, wave_paths=777), 3)
    _same(s, make_params(max_ray_depth=8), 7, rng=(13, 1801))


@pytest.mark.parametrize("xres", [48, 480])
def test_after_guided_bounces(xres):
    _same(scenes.cornell_box(xres, 360), make_params(max_ray_depth=10), 1, guide=True)


def test_views():
    s = SCENES["terrain"](16, 16)
    views = [(scenes.CameraSpec(pos=(0.3 * k, 1.2, -3.0), dir=(0, -0.3, 1), xres=20 + k, yres=17), 1 + k) for k in range(5)]
    a = GpuContext(s, make_params(max_ray_depth=10)).render_views(views, seed=3)
    b = GpuContext(s, make_params(max_ray_depth=10, wave_paths=1500)).render_views(views, seed=3)  # captured waves
    for k, (cam, spp) in enumerate(views):
        t = GpuContext(s, make_params(max_ray_depth=10))
        t.scene.camera = cam
        one = GpuContext(t.scene, make_params(max_ray_depth=10))
        one.render(spp, seed=3 + k)
        ref = one.framebuffer().reshape(a[k].shape)
        assert np.allclose(a[k], ref, rtol=1e-5, atol=1e-6)
        assert np.allclose(b[k], ref, rtol=1e-5, atol=1e-6)
