"""A cache call that asks for more scratch than the device has fails with
NR_ERR_OOM, and no call after it does."""
import ctypes

import numpy as np
import pytest

from nuray_gb300 import Scene, scenes
from nuray_gb300._lib import lib
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
