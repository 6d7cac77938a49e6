"""Closest-hit queries with directions at the edge of the prepared ray's
arithmetic: a component of exactly -1e-9f makes the box test's denominator
d + 1e-9f zero."""
import numpy as np
import pytest

from nuray_gb300 import scenes
from nuray_gb300._lib import Scene, check, lib
from oracle.bind import Oracle

pytestmark = pytest.mark.gpu


def _noalloc(S, o, d):
    n = len(o)
    out = np.zeros(n, np.int32), *(np.zeros(n, np.float32) for _ in range(3))
    check(lib().nr_intersect_noalloc(S._h, n, *(a.ctypes.data for a in (o, d) + out)))
    return out


@pytest.fixture(scope="module")
def walks(gpu_lib, port_lib):
    """The scene with the four-wide tree, without it (no room), and the restatement."""
    sc = scenes.small_scene(3, env=False, textures=False)

    def make(options=""):
        return Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], options=options)

    S = make()
    return sc, S, make(f"max_device_bytes={S.info()['device_bytes'] - 1}"), Oracle("port", sc)


def _every_walk(walks, o, d):
    """The query walks' answers for the same rays: four-wide, binary (no tree,
    and calls of 2^19 rays) and the same from the static scratch."""
    _, S, T, _ = walks
    many = (1 << 19) // len(o) + 1
    big = S.intersect(np.tile(o, (many, 1)), np.tile(d, (many, 1)))
    return [S.intersect(o, d), T.intersect(o, d), _noalloc(S, o, d), _noalloc(T, o, d), [a[:len(o)] for a in big],
            [a[-len(o):] for a in big], S.intersect(o, d, exhaustive=True), T.intersect(o, d, exhaustive=True)]


@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1), (1, 2), (2, 0)])
def test_denominator_of_zero(walks, axes):
    """Boxes that hold the origin along such an axis are entered, as the
    reference enters them (its quotients are -inf and +inf): its hits."""
    sc, _, _, P = walks
    r = np.random.default_rng(sum(axes))
    lo, hi = sc["pos"].reshape(-1, 3).min(0), sc["pos"].reshape(-1, 3).max(0)
    o = r.uniform(lo, hi, (3000, 3)).astype(np.float32)
    d = r.standard_normal((3000, 3)).astype(np.float32)
    d[:, axes] = np.float32(-1e-9)
    want = P.intersect(o, d)
    assert np.any(want[0] >= 0)
    for got in _every_walk(walks, o, d):
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
