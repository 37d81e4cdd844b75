"""The 4-wide layout with byte boxes where it differs most from the others: media around a large
mesh, rays through vertices and along edges, tiny clusters seen from far away, and trees too deep for
the 4-wide walk's stack."""
import numpy as np
import pytest

from naivetrace_b200 import abi, scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import MediumSpec, Scene, diffuse, make_params, volume_boundary

pytestmark = pytest.mark.gpu


def _grid(n, extent, height, offset=0.0, flat=0):
    """A bumpy n x n heightfield over [-extent/2, extent/2]^2: vertices and triangles.  The first `flat`
    rows lie at height 0, with a step behind them."""
    h = height * scenes.fbm_heightfield(n, 5, np.random.default_rng(5))
    h[:flat] = 0.0
    xs = np.linspace(-extent / 2, extent / 2, n)
    X, Z = np.meshgrid(xs, xs, indexing="ij")
    v = (np.stack([X, h, Z], -1).reshape(-1, 3) + offset).astype(np.float32)
    idx = np.arange(n * n).reshape(n, n)
    a, b, c, d = idx[:-1, :-1].ravel(), idx[1:, :-1].ravel(), idx[1:, 1:].ravel(), idx[:-1, 1:].ravel()
    return v, np.concatenate([np.stack([a, d, c], 1), np.stack([a, c, b], 1)]).astype(np.uint32)


def _mesh_scene(v, t):
    s = Scene()
    s.add_mesh(v, t, s.add_material(diffuse(0.5)))
    s.camera = scenes.CameraSpec(xres=8, yres=8)
    return s


def _both_layouts(scene, monkeypatch):
    wide = GpuContext(scene, make_params())
    monkeypatch.setenv("TT_BVH_WIDTH", "2")
    return wide, GpuContext(scene, make_params())


def _medium_scene(name, xres, yres):
    """A media scene with a heightfield of 32,258 triangles among its surfaces."""
    s = getattr(scenes, name)(xres, yres)
    v, t = _grid(128, 0.9, 0.2)
    s.add_mesh(v + np.float32([0.5, 0.15, 0.5]), t, s.add_material(diffuse(0.6)))
    return s


@pytest.mark.parametrize("algo", [abi.ALGO_PT, abi.ALGO_PT2])
@pytest.mark.parametrize("name", ["cornell_box_medium", "cornell_box_media_mix"])
def test_media_around_a_large_mesh(name, algo, monkeypatch):
    images = []
    for width in ("4", "2"):
        monkeypatch.setenv("TT_BVH_WIDTH", width)
        for profiling in (0, 1):  # whole paths, and every bounce as its own launches
            g = GpuContext(_medium_scene(name, 48, 40), make_params(max_ray_depth=8, algo=algo))
            assert g.stats()["bvh_node_bytes"] == 64
            g.set_profiling(profiling)
            g.render(4, seed=2)
            assert g.stats()["error_flags"] == 0
            images.append(g.accumulators()[0])
    for image in images[1:]:
        assert np.array_equal(images[0], image)
    assert np.any(images[0] != 0)


def _rays_at(points, distance, min_dy, rng):
    """Rays towards `points` from above, at most `distance` away."""
    n = len(points)
    d = rng.normal(size=(n, 3))
    d[:, 1] = np.abs(d[:, 1]) + min_dy
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = points + d * distance * rng.uniform(0.5, 1.0, (n, 1))
    q = points.astype(np.float64) - r[:, 0:3]
    r[:, 4:7] = q / np.linalg.norm(q, axis=1, keepdims=True)
    r[:, 7] = 1e30
    return r


# At a vertex or an edge the triangles around it lie within rounding of each other along the ray.  Which
# of them wins may depend on the walk (a box's entry, rounded at the scale of the ray's origin, can lie
# behind another triangle's hit), but no hit may be lost or invented, and the winners touch.
@pytest.mark.parametrize("offset", [0.0, 100.0])
@pytest.mark.parametrize("kind", ["vertex", "edge"])
def test_rays_at_vertices_and_edges(kind, offset, monkeypatch):
    v, t = _grid(200, 4.0, 0.2, offset, flat=50)
    wide, binary = _both_layouts(_mesh_scene(v, t), monkeypatch)
    assert wide.stats()["bvh_node_bytes"] == 64
    rng = np.random.default_rng(17)
    n, different = 1 << 20, 0
    for distance in (0.5, 5.0):
        corner = v[t[rng.integers(0, len(t), n)]]
        w = rng.random((n, 1)).astype(np.float32) if kind == "edge" else np.float32(0.0)
        rays = _rays_at(corner[:, 0] * (1 - w) + corner[:, 1] * w, distance, 0.2, rng)
        a, b = wide.intersect(rays)[0], binary.intersect(rays)[0]
        assert np.array_equal(a >= 0, b >= 0)
        assert np.array_equal(wide.occluded(rays), binary.occluded(rays))
        i = np.nonzero(a != b)[0]
        different += len(i)
        ta, tb = t[a[i]], t[b[i]]
        assert np.all((ta[:, :, None] == tb[:, None, :]).any(axis=(1, 2)))
    # One or two in a million at the edges of steep triangles far from the origin; 60 in a million if a
    # closest hit had to lie in a box that is entered before the nearest hit so far.
    if kind == "edge" and offset == 100.0:
        assert different <= 20
    assert wide.stats()["error_flags"] == 0


def test_tiny_cluster_from_far_away(monkeypatch):
    """Nodes smaller than a millionth of the ray's distance, where the widening of the exit distances
    outweighs a box's size: an empty slot may be met (it stands for the first child again)."""
    v, t = _grid(100, 0.05, 0.005)
    wide, binary = _both_layouts(_mesh_scene(v, t), monkeypatch)
    assert wide.stats()["bvh_node_bytes"] == 64
    rng = np.random.default_rng(3)
    corner = v[t[rng.integers(0, len(t), 1 << 18)]]
    w = rng.dirichlet((2, 2, 2), len(corner)).astype(np.float32)
    for distance in (10.0, 1000.0, 2000.0):
        rays = _rays_at((corner * w[:, :, None]).sum(1), distance, 1.0, rng)
        a, b = wide.intersect(rays)[0], binary.intersect(rays)[0]
        assert np.array_equal(a >= 0, b >= 0)
        assert (a >= 0).mean() > 0.2
    assert wide.stats()["error_flags"] == 0


def _nested(levels):
    """Clusters nested towards the origin, each a quarter of the one around it: per level a lone
    triangle near the inner ones and a longer row of ten beside them, deepest level first."""
    v, t = [], []
    rng = np.random.default_rng(1)
    for k in reversed(range(levels)):
        s = 0.25 ** k
        for x, y in [(0.02, 0.3)] + [(0.5 + 0.05 * i, 0.0) for i in range(10)]:
            z = 0.01 * rng.random(3)
            t.append([len(v), len(v) + 1, len(v) + 2])
            v += [[s * x, s * y, s * z[0]], [s * (x + 0.04), s * y, s * z[1]], [s * x, s * (y + 0.1), s * z[2]]]
    return np.array(v), np.array(t)


@pytest.mark.parametrize("levels,node_bytes", [(12, 112), (24, 64)])
def test_tree_too_deep_for_the_4_wide_walk(levels, node_bytes):
    """Where a path of the 4-wide tree could push more than the stack holds, the binary nodes serve all
    rays (64 bytes a node)."""
    v, t = _nested(levels)
    g = GpuContext(_mesh_scene(v, t), make_params())
    assert g.stats()["bvh_node_bytes"] == node_bytes
    rng = np.random.default_rng(2)
    tri = v.astype(np.float32)[t].astype(np.float64)[-11 * 8:]  # the eight outer levels
    rays = np.zeros((4096, 8), np.float32)
    w = rng.dirichlet((3, 3, 3), len(rays))
    target = (tri[rng.integers(0, len(tri), len(rays))] * w[:, :, None]).sum(1)
    rays[:, 0:3] = target + np.array([0.0, 0.0, 0.5]) + rng.uniform(-0.1, 0.1, (len(rays), 3))
    d = target - rays[:, 0:3]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 10.0
    prim, dist, _, _ = g.intersect(rays)
    # Every ray against every triangle in 64 bits; rays near an edge (at this distance) left out.
    tri = v.astype(np.float32)[t].astype(np.float64)
    o, d = rays[:, None, 0:3].astype(np.float64), rays[:, None, 4:7].astype(np.float64)
    e1, e2, s = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0], o - tri[:, 0]
    p = np.cross(d, e2)
    with np.errstate(divide="ignore", invalid="ignore"):
        inv = 1.0 / (p * e1).sum(-1)
        u, q = (s * p).sum(-1) * inv, np.cross(s, e1)
        w, tt = (d * q).sum(-1) * inv, (e2 * q).sum(-1) * inv
    edge = np.minimum(np.minimum(u, w), 1 - u - w)
    inside = (edge > 0) & (tt > 0)
    size = np.sqrt(0.5 * np.linalg.norm(np.cross(e1, e2), axis=1))
    clear = (~((np.abs(edge) * size < 1e-5) & (np.abs(edge) < 1))).all(1) & inside.any(1)
    tt[~inside] = np.inf
    assert clear.mean() > 0.2
    assert np.array_equal(prim[clear], tt.argmin(1)[clear])
    np.testing.assert_allclose(dist[clear], tt.min(1)[clear], rtol=1e-5)
    assert g.stats()["error_flags"] == 0


@pytest.mark.parametrize("wave_paths,profiling", [(20_011, 0), (20_011, 1)])
def test_captured_view_waves_after_guided_bounces(wave_paths, profiling):
    """Guided view batches: the replayed waves' last paths as whole paths, against one wave."""
    views = [(scenes.CameraSpec(pos=(0.5, 0.5, -1.4 + 0.1 * k), dir=(0, 0, 1), xres=90 + k, yres=80), 2 + k)
             for k in range(4)]
    batches, rays = [], []
    for paths, profile in ((0, 0), (wave_paths, profiling)):
        g = GpuContext(scenes.cornell_box(16, 16), make_params(max_ray_depth=10, wave_paths=paths))
        g.set_guiding(True, train=0, max_depth=2)
        w = np.random.default_rng(3).normal(scale=0.2, size=g.lib.tt_guide_num_params())
        g.guide_set_params(w.astype(np.float32))
        g.set_profiling(profile)
        batches.append(g.render_views(views, seed=3))
        s = g.stats()
        assert s["error_flags"] == 0
        rays.append([s[k] for k in ("paths", "extension_rays", "shadow_rays")])
    assert rays[0] == rays[1]
    for a, b in zip(*batches):
        # A pixel's samples are added in any order.
        assert np.allclose(a, b, rtol=1e-5, atol=1e-6)
