"""What a scene holds for speed alone makes room for others: the ray sort's
workspace of an idle scene is freed when an allocation of another scene or
cache fails, and the four-wide tree is given up only where that makes the
request fit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nuray_gb300 import NuRayError, Scene, scenes
from nuray_gb300._lib import lib
from nuray_gb300.nrc import Cache

pytestmark = pytest.mark.gpu
SC = scenes.terrain_spheres(2, tiles=16, cells_per_tile=8, spheres=40, slices=10, stacks=8, lights=8, n_mats=12,
                            extent=128.0)
CAM = "campos=0,45,65 cameuler=0,-42,0 camfov=45 camasp=1.25 maxdepth=3 rrdepth=2 seed=5 tail=0"
BIG = f"renderer=ptnee imgw=320 imgh=256 spp=52 {CAM}"  # one wave of 4.26 M paths: sorted
SMALL = f"renderer=ptnee imgw=40 imgh=32 spp=2 {CAM}"


def _scene(options=""):
    return Scene.from_arrays(SC["pos"], SC["mat"], SC["mats"], uv=SC["uv"], nrm=SC["nrm"], options=options)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("who", ["cache", "scene"])
def test_an_idle_scenes_workspace_makes_room(gpu_lib, who):
    S, T = _scene(), _scene()
    want = S.render(BIG)
    launches = S.stats()["kernel_launches"]
    T.render(SMALL)
    before = _free()
    if who == "cache":
        c, x = Cache("seed=1"), np.zeros((4, 80), np.float32)
        before = _free()
        # 3.5 TB of scratch: refused before a row is read
        assert lib().nr_nrc_gradient(c._h, 2**31 - 1, x.ctypes.data, x.ctypes.data, None, None) == -3
    else:
        with pytest.raises(NuRayError, match="NR_ERR_OOM"):  # 2.05 G paths in one wave: 370 GB of path state
            T.render(f"renderer=ptnee imgw=320 imgh=256 spp=25000 wave=2147483647 {CAM}")
    assert _free() - before >= 24 * 320 * 256 * 52  # S's workspace: 24 bytes a path and more
    np.testing.assert_array_equal(S.render(BIG), want)
    assert S.stats()["kernel_launches"] == launches  # sorted again


def test_the_tree_stays_where_its_room_would_not_do(gpu_lib):
    full = _scene().info()["device_bytes"]
    S = _scene(f"max_device_bytes={full + (4 << 20)}")
    want = S.render(SMALL)
    with pytest.raises(NuRayError, match="NR_ERR_OOM"):
        S.render(BIG)
    assert S.info()["device_bytes"] == full
    np.testing.assert_array_equal(S.render(SMALL), want)
