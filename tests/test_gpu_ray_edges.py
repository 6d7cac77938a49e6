"""Closest-hit queries with directions at the edge of the prepared ray's
arithmetic: a component of exactly -1e-9f makes the box test's denominator
d + 1e-9f zero; directions that are no numbers, or very long, walk by
closest_hit."""
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


def _rays(sc, n, seed):
    r = np.random.default_rng(seed)
    lo, hi = sc["pos"].reshape(-1, 3).min(0), sc["pos"].reshape(-1, 3).max(0)
    return r.uniform(lo, hi, (n, 3)).astype(np.float32), r.standard_normal((n, 3)).astype(np.float32)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1), (1, 2), (0, 1, 2)])
def test_a_direction_that_is_no_number_hits_nothing(walks, axes, bad):
    """Its determinant with any triangle is not finite. Rays beside it in the
    same warp have their own answers."""
    sc, S, _, _ = walks
    o, d = _rays(sc, 3000, 7)
    want = S.intersect(o, d)
    d[::3, axes] = bad
    for got in _every_walk(walks, o, d):
        assert np.all(got[0][::3] == -1)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a[1::3], b[1::3])
            np.testing.assert_array_equal(a[2::3], b[2::3])


def test_long_directions(walks):
    sc, _, _, P = walks
    o, d = _rays(sc, 3000, 8)
    d *= (10.0 ** np.random.default_rng(9).uniform(28, 32, (3000, 1))).astype(np.float32)
    want = P.intersect(o, d)
    assert np.any(want[0] >= 0)
    for got in _every_walk(walks, o, d):
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


def test_directions_of_zero(walks):
    """The biased determinant is then 1e-6 for every triangle, and t says nothing
    of where it lies: the exhaustive walk has the reference's answer, the
    pruned ones end."""
    sc, _, _, P = walks
    o, d = _rays(sc, 3000, 10)
    d[:] = 0
    want = P.intersect(o, d)
    got = _every_walk(walks, o, d)
    for a, b, c in zip(got[-2], got[-1], want):
        np.testing.assert_array_equal(a, c)
        np.testing.assert_array_equal(b, c)


@pytest.mark.parametrize("length", [31, 90])
def test_tree_of_chains(gpu_lib, length):
    """A tree (given to nr_scene_create_bvh) whose four-wide form fits the stack
    at 31 levels and not at 90: the same answers, for a direction of NaN too."""
    leaves = 4 * (length + 1)
    r = np.random.default_rng(length)
    x = np.arange(leaves)[:, None] * 0.5
    c = np.concatenate([x, r.uniform(-1, 1, (leaves, 2))], 1)
    pos = np.concatenate([c + [0, -0.5, -0.5], c + [0.1, 0.5, -0.5], c + [0.2, 0, 0.6]], 1).astype(np.float32)
    lo, hi = pos.reshape(-1, 3, 3).min(1), pos.reshape(-1, 3, 3).max(1)
    box, kids, first, count = [], [], [], []

    def sub(a, b, chain):
        me = len(box)
        box.append(np.concatenate([lo[a:b].min(0), hi[a:b].max(0)]))
        kids.append((-1, -1)), first.append(a), count.append(b - a)
        if b - a > 1:
            m = a + 4 if chain and b - a > 4 else (a + b) // 2
            first[me] = count[me] = 0
            kids[me] = (sub(a, m, False), sub(m, b, chain))
        return me

    sub(0, leaves, True)
    tree = tuple(np.array(a, t) for a, t in zip((box, kids, first, count, np.arange(leaves)),
                                                (np.float32, np.int32, np.int32, np.int32, np.int32)))
    mats = [dict(type=0, c0=[0.5] * 3), dict(type=5, c0=[1.0] * 3)]
    mat = np.zeros(leaves, np.int32)
    mat[-1] = 1
    S, T = Scene.from_arrays(pos, mat, mats, bvh=tree), Scene.from_arrays(pos, mat, mats)
    o = r.uniform([-1, -1, -1], [leaves / 2, 1, 1], (2000, 3)).astype(np.float32)
    d = r.standard_normal((2000, 3)).astype(np.float32)
    d[::2, 1:] *= 0.05  # along the chain
    d[::7] = np.nan
    for a, b in zip(S.intersect(o, d), T.intersect(o, d)):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(_noalloc(S, o, d), T.intersect(o, d)):
        np.testing.assert_array_equal(a, b)
    p = "renderer=ptnee imgw=16 imgh=8 spp=4 campos=" + f"{leaves / 2 - 1},0,4 " + "cameuler=0,0,0 camfov=60 camasp=2 maxdepth=4"
    a, b = S.render(p), T.render(p)
    assert np.all(np.isfinite(a))
    np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-7)
