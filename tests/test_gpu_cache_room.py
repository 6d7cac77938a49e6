"""A cache call that asks for more scratch than the device has fails with
NR_ERR_OOM and leaves the cache as it was: the next call sizes its scratch
anew, and does not fail in its turn."""
import ctypes

import numpy as np
import pytest

from nuray_gb300 import Scene, scenes
from nuray_gb300._lib import check, lib
from nuray_gb300.nrc import INPUTS, Cache

pytestmark = pytest.mark.gpu
TOO_MANY = 2**31 - 1  # rows: some 3.5 TB of scratch, refused before a row is read
OOM = -3


def _rows(n):
    r = np.random.default_rng(n)
    return r.uniform(-1, 1, (n, INPUTS)).astype(np.float32), r.gamma(1.0, 1.0, (n, 3)).astype(np.float32)


def test_the_error_is_reported_once(gpu_lib):
    x, y = _rows(64)
    lo = ctypes.c_float()
    sc = scenes.small_scene(4, env=False, textures=False)
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"])
    for call in (lambda c: c.infer(x), lambda c: S.intersect(x[:, :3], x[:, 3:6]), lambda c: S.set_materials(sc["mats"]),
                 lambda c: S.render("renderer=ptnee imgw=8 imgh=8 spp=1 maxdepth=2")):
        c = Cache("seed=3")
        assert lib().nr_nrc_gradient(c._h, TOO_MANY, x.ctypes.data, y.ctypes.data, None, ctypes.byref(lo)) == OOM
        call(c)


@pytest.mark.parametrize("tc", [0, 1])
def test_calls_after_one_without_room(gpu_lib, tc):
    c, fresh = Cache(f"seed=3 tc={tc}"), Cache(f"seed=3 tc={tc}")
    x, y = _rows(3000)
    infer, (g, loss) = fresh.infer(x), fresh.gradient(x, y)
    c.infer(x)
    p, q = x.ctypes.data, y.ctypes.data
    out, lo = np.empty((3000, 3), np.float32), ctypes.c_float()
    assert lib().nr_nrc_infer(c._h, TOO_MANY, p, out.ctypes.data) == OOM
    np.testing.assert_array_equal(c.infer(x[:700]), infer[:700])
    assert lib().nr_nrc_gradient(c._h, TOO_MANY, p, q, None, ctypes.byref(lo)) == OOM
    g2, l2 = c.gradient(x, y)
    # float atomics in any order: sums of up to 3000 terms of either sign
    np.testing.assert_allclose(g2, g, rtol=1e-4, atol=1e-5 * np.abs(g).max())
    assert l2 == pytest.approx(loss, rel=1e-5)
    assert lib().nr_nrc_train_step(c._h, TOO_MANY, p, q, ctypes.byref(lo)) == OOM
    np.testing.assert_array_equal(c.infer(x), infer)  # no step was taken


def test_a_frame_after_a_call_without_room(gpu_lib):
    sc = scenes.small_scene(4)
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], textures=sc["textures"],
                          env_tex=sc["env_tex"], env_gain=sc["env_gain"])
    p = ("renderer=ptnee imgw=64 imgh=48 spp=2 campos=0,14,34 cameuler=0,-20,0 camfov=50 camasp=1.3333 maxdepth=4 "
         "nrc=1 nrc_steps=1")
    frames = []
    for fail in (False, True):
        c = Cache("seed=3")
        c.infer(_rows(64)[0])
        if fail:
            assert lib().nr_nrc_infer(c._h, TOO_MANY, frames[0].ctypes.data, frames[0].ctypes.data) == OOM
        c.attach(S)
        frames.append(S.render(p))  # predicted by the untrained cache
        check(lib().nr_scene_attach_nrc(S._h, None))
    np.testing.assert_array_equal(frames[0], frames[1])
