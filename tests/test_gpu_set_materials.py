"""nr_scene_set_materials rewrites the material table and the emitters'
radiance on the device: the scene then renders as one created with those
materials."""
import numpy as np
import pytest

from nuray_gb300 import NuRayError, Scene, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emitters", [0, 1, 8, 129, 700])
def test_set_materials_equals_a_new_scene(gpu_lib, emitters):
    sc = scenes.small_scene(5)
    r = np.random.default_rng(emitters)
    mats = [dict(m) for m in sc["mats"]] + [dict(type=5, c0=[1.0, 2.0, 3.0]), dict(type=5, c0=[3.0, 0.5, 0.25])]
    mat = np.where(np.isin(sc["mat"], [i for i, m in enumerate(mats) if m["type"] == 5]), 0, sc["mat"]).astype(np.int32)
    pick = r.choice(len(mat), emitters, replace=False)
    mat[pick] = len(mats) - 2 + (np.arange(emitters) % 2)

    def scene(m):
        return Scene.from_arrays(sc["pos"], mat, m, uv=sc["uv"], nrm=sc["nrm"], textures=sc["textures"],
                                 env_tex=sc["env_tex"], env_gain=sc["env_gain"])

    p = "renderer=ptnee imgw=40 imgh=32 spp=8 campos=0,14,34 cameuler=0,-20,0 camfov=50 camasp=1.25 maxdepth=5"
    S = scene(mats)
    before = S.render(p)
    new = [dict(m, c0=[float(np.float32(v)) for v in r.uniform(0.1, 0.9, 3) * (8 if m["type"] == 5 else 1)],
                alpha=float(r.uniform(0.1, 0.9)), tex0=-1) for m in mats]
    S.set_materials(new)
    np.testing.assert_array_equal(S.render(p), scene(new).render(p))
    with pytest.raises(NuRayError, match="type changed"):
        S.set_materials([dict(m, type=0) for m in new])
    S.set_materials(mats)
    np.testing.assert_array_equal(S.render(p), before)
