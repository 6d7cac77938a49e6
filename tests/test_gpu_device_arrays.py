"""Arrays in device, pinned or managed memory where a call takes host arrays:
the copies of staged arrays take them all, and so does every call."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nuray_gb300 import scenes
from nuray_gb300._lib import Scene, check, lib
from nuray_gb300.nrc import INPUTS, Cache

pytestmark = pytest.mark.gpu


def _place(a, where):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return {"host": t.clone, "pinned": t.pin_memory, "device": t.cuda}[where]()


@pytest.mark.parametrize("n", [1, 33, 5000])
@pytest.mark.parametrize("where_in", ["host", "pinned", "device"])
@pytest.mark.parametrize("where_out", ["host", "pinned", "device"])
def test_query_arrays(gpu_lib, n, where_in, where_out):
    sc = scenes.small_scene(3, env=False, textures=False)
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"])
    r = np.random.default_rng(n)
    lo, hi = sc["pos"].reshape(-1, 3).min(0), sc["pos"].reshape(-1, 3).max(0)
    o, d = r.uniform(lo, hi, (n, 3)).astype(np.float32), r.standard_normal((n, 3)).astype(np.float32)
    want = S.intersect(o, d)
    rays = [_place(a, where_in) for a in (o, d)]
    out = [_place(np.zeros_like(a), where_out) for a in want]
    torch.cuda.synchronize()
    check(lib().nr_intersect(S._h, n, *(t.data_ptr() for t in rays + out), 0))
    for t, w in zip(out, want):
        np.testing.assert_array_equal(t.cpu().numpy(), w)


@pytest.mark.parametrize("tc", [0, 1])
@pytest.mark.parametrize("where", ["host", "pinned", "device"])
def test_cache_arrays(gpu_lib, where, tc):
    n = 700
    r = np.random.default_rng(n)
    x, y = r.uniform(-1, 1, (n, INPUTS)).astype(np.float32), r.gamma(1.0, 1.0, (n, 3)).astype(np.float32)
    c = Cache(f"seed=3 tc={tc}")
    want, (g, loss) = c.infer(x), c.gradient(x, y)
    px, py, out, pg = (_place(a, where) for a in (x, y, np.zeros_like(want), np.zeros_like(g)))
    torch.cuda.synchronize()
    check(lib().nr_nrc_infer(c._h, n, px.data_ptr(), out.data_ptr()))
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    lo = ctypes.c_float()
    check(lib().nr_nrc_gradient(c._h, n, px.data_ptr(), py.data_ptr(), pg.data_ptr(), ctypes.byref(lo)))
    # float atomics in any order: sums of up to n terms of either sign
    np.testing.assert_allclose(pg.cpu().numpy(), g, rtol=1e-4, atol=1e-5 * np.abs(g).max())
    assert lo.value == pytest.approx(loss, rel=1e-5)
