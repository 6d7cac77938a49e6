"""The traversal walks at the edges of their range: trees of one leaf (no
inner node), of one and of a few inner nodes, against the CPU restatement."""
import numpy as np
import pytest

from nuray_gb300 import Scene
from oracle.bind import Oracle

pytestmark = pytest.mark.gpu

MATS = [dict(type=0, c0=[0.7, 0.6, 0.5]), dict(type=5, c0=[3.0, 3.0, 3.0])]


def _few_triangles(n, seed):
    """n triangles facing the camera at different depths, the last one an emitter behind it."""
    r = np.random.default_rng(seed)
    c = np.stack([r.uniform(-1, 1, n), r.uniform(-1, 1, n), r.uniform(-4, -2, n)], 1)
    pos = np.concatenate([c + [-0.6, -0.5, 0.1], c + [0.6, -0.5, 0.0], c + [0.0, 0.7, -0.1]], 1)
    mat = np.zeros(n, np.int32)
    if n > 1:
        pos[-1] = [-2, -2, 3, -2, 2, 3, 2, 2, 3]
        mat[-1] = 1
    pos = pos.astype(np.float32)
    return dict(pos=pos, uv=np.zeros((n, 6), np.float32), nrm=np.zeros((n, 9), np.float32), mat=mat, mats=MATS)


@pytest.mark.parametrize("trav", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 7, 12, 33])
def test_small_trees_match_port(gpu_lib, port_lib, n, trav):
    sc = _few_triangles(n, 100 + n)
    S, P = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"]), Oracle("port", sc)
    p = f"renderer=ptnee imgw=40 imgh=30 spp=4 campos=0,0,1 cameuler=0,0,0 camfov=60 camasp=1.3333 trav={trav}"
    pix = np.array([(x, y) for y in range(0, 30, 3) for x in range(0, 40, 3)], np.int32)
    # every float32 step of the estimator is the restatement's; libm calls differ in the last bits
    np.testing.assert_allclose(S.render_samples(p, pix, 4), P.render_samples(p, pix, 4), rtol=2e-3, atol=1e-4)
    r = np.random.default_rng(n)
    o = np.tile(np.array([0, 0, 1], np.float32), (500, 1))
    d = np.stack([r.uniform(-0.5, 0.5, 500), r.uniform(-0.5, 0.5, 500), -np.ones(500)], 1).astype(np.float32)
    for a, b in zip(S.intersect(o, d, exhaustive=trav == 0), P.intersect(o, d)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("policy", ["maxdepth=5 rrdepth=3", "prr=0.8", "maxdepth=1"])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (7, 5, 3), (97, 51, 4), (401, 303, 2), (640, 480, 5)])
def test_automatic_tail_gives_the_wavefront_image(gpu_lib, w, h, spp, policy):
    """By default one launch takes every path to its end from the bounce that
    is known to start with few of them: the whole wave of the small frames
    here (warps of 1 to 32 paths), some later bounce of the large one. The
    light samples are rounded before they are added in both kernels, so the
    image is that of tail=0 (the shading code inlined into the tail may
    contract other multiply-adds: a few ulp). Both count every ray."""
    from nuray_gb300 import scenes
    sc = scenes.small_scene(9)
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], textures=sc["textures"],
                          env_tex=sc["env_tex"], env_gain=sc["env_gain"])
    p = (f"renderer=ptnee imgw={w} imgh={h} spp={spp} campos=0,14,34 cameuler=0,-20,0 camfov=50 camasp={w / h:.4f} "
         + policy)
    a = S.render(p)
    sa = S.stats()
    b = S.render(p + " tail=0")
    sb = S.stats()
    np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-7)
    assert (sa["rays"], sa["shadow_rays"]) == (sb["rays"], sb["shadow_rays"])


@pytest.mark.parametrize("n", [1, 3, 31, 33, 6081, 65536, 65537, 194561, 524287, 524289])
def test_query_spread_covers_every_ray(gpu_lib, port_lib, n):
    """nr_intersect gives a warp 1 to 32 rays by their number, and another
    build of its kernel from 2^19 on: every ray has its own answer, equal to
    the restatement's on a sample, and the calls agree with each other."""
    from nuray_gb300 import scenes
    sc = scenes.small_scene(3, env=False, textures=False)
    S, P = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"]), Oracle("port", sc)
    r = np.random.default_rng(n)
    lo, hi = sc["pos"].reshape(-1, 3).min(0), sc["pos"].reshape(-1, 3).max(0)
    o = r.uniform(lo, hi, (n, 3)).astype(np.float32)
    o[::5] = o[::5] * 40  # origins outside the widened boxes' bound take the exact walk
    d = r.standard_normal((n, 3)).astype(np.float32)
    got = S.intersect(o, d)
    k = r.permutation(n)[:4000]
    for a, b in zip((x[k] for x in got), P.intersect(o[k], d[k])):
        assert np.mean(a == b) >= 0.999  # grazing rays may take another of two overlapping triangles
    m = min(n, 65536)
    from nuray_gb300._lib import check, lib
    oc, dc = np.ascontiguousarray(o[:m]), np.ascontiguousarray(d[:m])
    tri, t, b1, b2 = np.zeros(m, np.int32), *(np.zeros(m, np.float32) for _ in range(3))
    check(lib().nr_intersect_noalloc(S._h, m, *(x.ctypes.data for x in (oc, dc, tri, t, b1, b2))))
    for a, b in zip(got, (tri, t, b1, b2)):
        np.testing.assert_array_equal(a[:m], b)


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (1, 9, 3), (9, 1, 5), (7, 3, 3), (8, 4, 3), (9, 5, 1), (33, 18, 6), (64, 64, 12),
                                     (101, 67, 7)])
def test_pixel_order_gives_the_same_image(gpu_lib, w, h, spp):
    """Frames or sample counts that tiles of a warp do not divide take all
    samples of each pixel in turn, pixels in 8x4 tiles narrower and lower at
    the edges: every pixel once, its samples added in sample order, also
    where a wave ends between a pixel's samples."""
    from nuray_gb300 import scenes
    sc = scenes.small_scene(8)
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], textures=sc["textures"],
                          env_tex=sc["env_tex"], env_gain=sc["env_gain"])
    p = (f"renderer=ptnee imgw={w} imgh={h} spp={spp} campos=0,14,34 cameuler=0,-20,0 camfov=50 camasp={w / h:.4f} "
         "maxdepth=4")
    ref = S.render(p + " tile=0")
    for more in ("", " wave=1", " wave=50", " wave=777"):
        if "wave=1" in more and w * h * spp > 3000:
            continue
        np.testing.assert_array_equal(S.render(p + more), ref, err_msg=more)
    dl = np.random.default_rng(1).standard_normal((h, w, 3)).astype(np.float32)
    a, ia = S.adjoint(p, dl, want_image=True)
    b, ib = S.adjoint(p + " tile=0", dl, want_image=True)
    np.testing.assert_array_equal(ia, ib)
    # float atomics in any order: sums of up to 4 terms a path of either sign
    np.testing.assert_allclose(a, b, rtol=1e-4, atol=1e-5 * max(1e-6, np.abs(a).max()))
