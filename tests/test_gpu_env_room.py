"""An environment that does not fit the device is refused, and the scene keeps
the one it had."""
import numpy as np
import pytest

from nuray_gb300 import NuRayError, Scene, scenes

pytestmark = pytest.mark.gpu
P = ("renderer=ptnee imgw=64 imgh=48 spp=2 campos=0,14,34 cameuler=0,-20,0 camfov=50 camasp=1.3333 maxdepth=4")


@pytest.mark.parametrize("env", ["the scene's own", "one set before", "none"])
def test_an_environment_without_room(gpu_lib, env):
    sc = scenes.small_scene(4)

    def make(options=""):
        S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], textures=sc["textures"],
                              env_tex=sc["env_tex"], env_gain=sc["env_gain"], options=options)
        if env == "one set before":
            S.set_env(np.full((4, 8, 3), 0.5, np.float32), 2.0)
        if env == "none":
            S.set_env(None, 1.0)
        return S

    free = make()
    want = free.render(P)
    S = make(f"max_device_bytes={free.info()['device_bytes'] + (8 << 20)}")
    o, d = np.zeros((3, 3), np.float32), np.eye(3, dtype=np.float32)
    for _ in range(2):
        with pytest.raises(NuRayError, match="NR_ERR_OOM"):
            S.set_env(np.ones((1024, 2048, 3), np.float32), 1.0)  # 32 MB of texels
        np.testing.assert_array_equal(S.render(P), want)
        for a, b in zip(S.intersect(o, d), free.intersect(o, d)):
            np.testing.assert_array_equal(a, b)
        S.set_materials(sc["mats"])
    small = np.random.default_rng(0).uniform(0, 1, (8, 16, 3)).astype(np.float32)
    for scene in (S, free):
        scene.set_env(small, 1.5)
    np.testing.assert_array_equal(S.render(P), free.render(P))
