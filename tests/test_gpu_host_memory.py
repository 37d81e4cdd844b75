"""Images and ray batches from and to the caller's memory, pageable or page-locked."""
import ctypes as C
import time

import numpy as np
import pytest

from naivetrace_b200 import abi, scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import make_params

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _array(shape, locked):
    if not locked:
        return np.zeros(shape, np.float32)
    return torch.zeros(shape, dtype=torch.float32, pin_memory=True).numpy()


def _fp(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


def test_page_locked_image_is_copied_once():
    """Straight into page-locked memory (0.5 ms for 25 MB), not through the library's own blocks
    (as long as into pageable memory, 1.2 ms)."""
    g = GpuContext(scenes.cornell_box(1920, 1080), make_params(max_ray_depth=2))
    g.render(1, seed=1)
    fastest, images = [], []
    for locked in (True, False):
        rgb = _array(3 * g.npix, locked)
        times = []
        for _ in range(20):
            t = time.perf_counter()
            assert g.lib.tt_read_framebuffer(g.h, _fp(rgb), None) == abi.TT_OK
            times.append(time.perf_counter() - t)
        fastest.append(min(times))
        images.append(rgb)
    assert np.array_equal(*images)
    assert fastest[0] < 0.75 * fastest[1]


@pytest.mark.parametrize("n", [1, 70_001, 400_003])  # below and above the size that goes through blocks
def test_ray_batches_with_mixed_memory(n):
    """Each array of a batch may be pageable or page-locked."""
    g = GpuContext(scenes.cornell_box(8, 8), make_params(max_ray_depth=2))
    rng = np.random.default_rng(n)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = rng.uniform(0.1, 0.9, (n, 3))
    rays[:, 4:7] = rng.normal(size=(n, 3))
    rays[:, 4:7] /= np.linalg.norm(rays[:, 4:7], axis=1, keepdims=True)
    rays[:, 7] = 10.0
    expected, occluded = g.intersect(rays), g.occluded(rays)
    for kinds in ((1, 1, 1, 1, 1), (1, 0, 1, 0, 1), (0, 1, 0, 1, 0)):
        r, prim, t, u, v = (_array(s, k) for s, k in zip(((n, 8), n, n, n, n), kinds))
        r[:] = rays
        assert g.lib.tt_intersect_batch(g.h, _fp(r), n, prim.ctypes.data_as(C.POINTER(C.c_int32)), _fp(t), _fp(u),
                                        _fp(v)) == abi.TT_OK
        for a, b in zip((prim.view(np.int32), t, u, v), expected):
            assert np.array_equal(a, b)
        occ = _array((n + 3) // 4, kinds[1]).view(np.uint8)[:n]
        assert g.lib.tt_occluded_batch(g.h, _fp(r), n, occ.ctypes.data_as(C.POINTER(C.c_uint8))) == abi.TT_OK
        assert np.array_equal(occ.astype(bool), occluded)
