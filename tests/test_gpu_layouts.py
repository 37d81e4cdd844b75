"""Hits on the 4-wide layout with byte boxes and refilled lanes equal those of the binary layout
with float boxes, bit for bit, around the primitive count where the format changes."""
import numpy as np
import pytest

from naivetrace_b200 import abi, scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import Scene, diffuse, make_params

pytestmark = pytest.mark.gpu

BYTES_MIN = 16384  # primitives from which the 4-wide nodes have byte boxes


def _heightfield(prims, spheres, offset):
    """`prims` primitives in all: a bumpy grid (with flat axis-aligned parts) and analytic spheres."""
    n = 128
    rng = np.random.default_rng(5)
    h = 0.2 * scenes.fbm_heightfield(n, 5, rng)
    h[: n // 4] = 0.0
    xs = np.linspace(-2.0, 2.0, n)
    X, Z = np.meshgrid(xs, xs, indexing="ij")
    v = np.stack([X, h, Z], -1).reshape(-1, 3) + offset
    idx = np.arange(n * n).reshape(n, n)
    a, b, c, d = idx[:-1, :-1].ravel(), idx[1:, :-1].ravel(), idx[1:, 1:].ravel(), idx[:-1, 1:].ravel()
    t = np.concatenate([np.stack([a, d, c], 1), np.stack([a, c, b], 1)])
    s = Scene()
    m = s.add_material(diffuse(0.5))
    s.add_mesh(v, np.resize(t, (prims - spheres, 3)), m)
    for k in range(spheres):
        s.add_sphere(rng.uniform(-1.5, 1.5, 3) * [1, 0.2, 1] + offset, 0.05 + 0.02 * k, m)
    s.camera = scenes.CameraSpec(xres=8, yres=8)
    return s


def _rays(n, offset):
    rng = np.random.default_rng(n)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-2.5, 2.5, (n, 3)) * [1, 0.4, 1] + offset
    d = rng.normal(size=(n, 3))
    d[::7, 0] = 0.0       # in axis planes and along axes
    d[::7, 2] = -0.0
    d[3::11, 1] = 0.0
    d[np.linalg.norm(d, axis=1) == 0] = [0, -1, 0]
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = np.where(rng.random(n) < 0.5, 1e30, rng.uniform(0.1, 4.0, n))
    r[::13, 3] = 0.05
    return r


@pytest.mark.parametrize("prims", [BYTES_MIN - 1, BYTES_MIN, 2 * 127 * 127])
@pytest.mark.parametrize("spheres,offset", [(0, 0.0), (3, 0.0), (0, 1000.0)])
def test_byte_boxes_equal_binary(prims, spheres, offset, monkeypatch):
    scene = _heightfield(prims, spheres, offset)
    wide = GpuContext(scene, make_params())
    monkeypatch.setenv("TT_BVH_WIDTH", "2")
    binary = GpuContext(scene, make_params())
    assert wide.stats()["bvh_node_bytes"] == (64 if prims >= BYTES_MIN else 112)
    for n in (1, 31, 33, 257, 4097, 400003):  # warp remainders up to several refills per warp
        rays = _rays(n, offset)
        for a, b in zip(wide.intersect(rays), binary.intersect(rays)):
            assert np.array_equal(a, b)
        assert np.array_equal(wide.occluded(rays), binary.occluded(rays))
    assert wide.stats()["error_flags"] == 0


@pytest.mark.parametrize("algo", [abi.ALGO_PT, abi.ALGO_PT2])
@pytest.mark.parametrize("name", ["cornell_box_media_mix", "spheres_box"])
def test_renders_on_every_layout(algo, name, monkeypatch):
    """Media renders on the binary and the 8-wide layout: every kernel traverses the layout the
    context holds."""
    params = make_params(max_ray_depth=8, algo=algo)
    images = []
    for width in ("4", "2", "8"):
        monkeypatch.setenv("TT_BVH_WIDTH", width)
        g = GpuContext(getattr(scenes, name)(48, 40), params)
        g.render(4, seed=2)
        images.append(g.accumulators()[0])
        assert g.stats()["error_flags"] == 0
    assert np.array_equal(images[0], images[1])
    # The 8-wide layout's own boxes may decide a grazing ray otherwise.
    assert np.isclose(images[0], images[2], rtol=1e-5, atol=1e-6).mean() > 0.999


@pytest.mark.parametrize("prims", [1, 2, 3, 5, 4095, 4096, 4097, 9001])
def test_device_build_equals_host_build(prims, monkeypatch):
    """Around the cluster count where the device build goes on in one block: the same hits as on
    the host-built tree."""
    scene = _heightfield(prims, min(2, prims - 1), 0.0)
    device = GpuContext(scene, make_params())
    monkeypatch.setenv("TT_BVH_BUILD", "host")
    host = GpuContext(scene, make_params())
    rays = _rays(60001, 0.0)
    for a, b in zip(device.intersect(rays), host.intersect(rays)):
        assert np.array_equal(a, b)
    assert np.array_equal(device.occluded(rays), host.occluded(rays))
