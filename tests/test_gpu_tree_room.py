"""max_device_bytes that holds everything a scene and its calls need but not
the four-wide tree: they run as with it, and few rays walk the binary tree."""
import numpy as np
import pytest

from nuray_gb300 import scenes
from nuray_gb300._lib import NuRayError, Scene

pytestmark = pytest.mark.gpu
SC = scenes.terrain_spheres(1, tiles=16, cells_per_tile=4, spheres=40, lights=8, n_mats=12, extent=80.0)
W, H, SPP = 64, 32, 64
P = f"renderer=ptnee imgw={W} imgh={H} spp={SPP} seed=2 campos=0,14,34 cameuler=0,-20,0 camfov=50 camasp=2 maxdepth=5"
STATE = W * H * SPP * (5 * 16 + 16 + 2 * 4 + 7 * 4 + 3 * 16) + W * H * (16 + 12)  # path state, film and image


def _scene(options=""):
    return Scene.from_arrays(SC["pos"], SC["mat"], SC["mats"], uv=SC["uv"], nrm=SC["nrm"], options=options)


def _check(S, T, rel):
    r = np.random.default_rng(0)
    pos = SC["pos"].reshape(-1, 3)
    o = r.uniform(pos.min(0), pos.max(0), (3000, 3)).astype(np.float32)
    d = r.standard_normal((3000, 3)).astype(np.float32)
    for a, b in zip(S.intersect(o, d), T.intersect(o, d)):
        assert np.mean(a == b) >= 0.999  # grazing rays may take another of two overlapping triangles
    a, b = S.render(P), T.render(P)
    assert np.mean(np.abs(a - b) <= 1e-5 * np.abs(a) + 1e-7) >= rel


def test_a_scene_without_room_for_the_tree(gpu_lib):
    S = _scene()
    T = _scene(f"max_device_bytes={S.info()['device_bytes'] - 1}")
    assert T.info()["device_bytes"] < S.info()["device_bytes"]
    T.close()
    with pytest.raises(NuRayError, match="NR_ERR_OOM"):
        _scene(f"max_device_bytes={S.info()['device_bytes'] // 2}")


def test_a_call_that_needs_the_trees_room(gpu_lib):
    """The path state fits only where the tree was: it is given up, and queries,
    renders and a replaced environment go on without it."""
    S = _scene()
    full = S.info()["device_bytes"]
    bare = _scene(f"max_device_bytes={full - 1}")
    tree = full - bare.info()["device_bytes"]
    assert tree > (64 << 10)
    T = _scene(f"max_device_bytes={full + STATE + (32 << 10) - tree // 2}")
    assert T.info()["device_bytes"] == full
    a, b = S.render(P), T.render(P)
    assert T.info()["device_bytes"] == full - tree
    # paths whose hit is one of two overlapping triangles may differ
    assert np.mean(np.abs(a - b) <= 1e-5 * np.abs(a) + 1e-7) >= 0.999
    _check(S, T, 0.999)
    img = np.ones((4, 8, 3), np.float32)
    S.set_env(img, 1.0)
    T.set_env(img, 1.0)
    _check(S, T, 0.999)
