"""Host arrays that a kernel cannot use where they lie (not on a float's
boundary, or a result that shares memory with an input or another result) give
the same answers: everything is read before anything is written."""
import ctypes

import numpy as np
import pytest

from nuray_gb300 import scenes
from nuray_gb300._lib import Scene, check, lib
from nuray_gb300.nrc import INPUTS, Cache

pytestmark = pytest.mark.gpu


def _at(buf, a, offset):
    """Copies a into the byte buffer at `offset` past a 64-byte boundary; the address."""
    start = (-buf.ctypes.data) % 64 + offset
    raw = a.view(np.uint8).reshape(-1)
    buf[start:start + raw.size] = raw
    return buf.ctypes.data + start


def _read(buf, offset, n, dtype):
    start = (-buf.ctypes.data) % 64 + offset
    return buf[start:start + 4 * n].copy().view(dtype)


@pytest.fixture(scope="module")
def rays(gpu_lib):
    sc = scenes.small_scene(3, env=False, textures=False)
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"])
    r = np.random.default_rng(4)
    lo, hi = sc["pos"].reshape(-1, 3).min(0), sc["pos"].reshape(-1, 3).max(0)

    def make(n):
        return r.uniform(lo, hi, (n, 3)).astype(np.float32), r.standard_normal((n, 3)).astype(np.float32)

    return S, make


@pytest.mark.parametrize("n", [1, 33, 5000])
@pytest.mark.parametrize("off", [0, 1, 2, 4, 7])
def test_query_arrays_at_any_byte(rays, n, off):
    S, make = rays
    o, d = make(n)
    want = S.intersect(o, d)
    bufs = [np.zeros(12 * n + 128, np.uint8) for _ in range(6)]
    p = [_at(b, a, off) for b, a in zip(bufs, (o, d) + tuple(np.zeros(n, np.float32) for _ in range(4)))]
    check(lib().nr_intersect(S._h, n, *p, 0))
    for b, w in zip(bufs[2:], want):
        np.testing.assert_array_equal(_read(b, off, n, w.dtype), w)


@pytest.mark.parametrize("n", [1, 33, 5000])
def test_query_results_over_the_inputs(rays, n):
    S, make = rays
    o, d = make(n)
    want = S.intersect(o, d)
    ob, db = o.copy(), d.copy()  # tri, t over the origins; b1, b2 over the directions
    p = [ob.ctypes.data, db.ctypes.data]
    check(lib().nr_intersect(S._h, n, *p, p[0], p[0] + 4 * n, p[1], p[1] + 8 * n, 0))
    of, df = ob.reshape(-1), db.reshape(-1)
    got = of[:n].view(np.int32), of[n:2 * n], df[:n], df[2 * n:]
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("n", [1, 33, 5000])
def test_query_results_over_each_other(rays, n):
    S, make = rays
    o, d = make(n)
    want = S.intersect(o, d)
    a = np.empty(n, np.float32)
    p = a.ctypes.data
    check(lib().nr_intersect(S._h, n, o.ctypes.data, d.ctypes.data, p, p, p, p, 0))
    np.testing.assert_array_equal(a, want[3])  # b2 is the last one written


@pytest.mark.parametrize("tc", [0, 1])
@pytest.mark.parametrize("n", [1, 129, 5000])
def test_cache_arrays(gpu_lib, n, tc):
    r = np.random.default_rng(n)
    x = r.uniform(-1, 1, (n, INPUTS)).astype(np.float32)
    y = r.gamma(1.0, 1.0, (n, 3)).astype(np.float32)
    c = Cache(f"seed=3 tc={tc}")
    want, (g, loss) = c.infer(x), c.gradient(x, y)
    for off in (1, 2, 7):
        xb, yb, ob = (np.zeros(a + 128, np.uint8) for a in (x.nbytes, y.nbytes, y.nbytes))
        px, py, po = _at(xb, x, off), _at(yb, y, off), _at(ob, y, off)
        check(lib().nr_nrc_infer(c._h, n, px, po))
        np.testing.assert_array_equal(_read(ob, off, 3 * n, np.float32).reshape(n, 3), want)
        g2, l2 = np.empty_like(g), ctypes.c_float()
        check(lib().nr_nrc_gradient(c._h, n, px, py, g2.ctypes.data, ctypes.byref(l2)))
        # float atomics in any order: sums of up to n terms of either sign
        np.testing.assert_allclose(g2, g, rtol=1e-4, atol=1e-5 * np.abs(g).max())
        assert l2.value == pytest.approx(loss, rel=1e-5)
    xo = x.copy()  # the outputs over the first rows
    check(lib().nr_nrc_infer(c._h, n, xo.ctypes.data, xo.ctypes.data))
    np.testing.assert_array_equal(xo.reshape(-1)[:3 * n].reshape(n, 3), want)
