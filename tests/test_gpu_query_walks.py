"""nr_intersect's walks have one answer: the four-wide tree's, the binary
tree's (calls of 2^19 rays, scenes without the other) and the static
scratch's are equal bit for bit, and with exhaustive pruning off so is the
restatement's. Rays in no order, of a camera, and off the surfaces."""
import numpy as np
import pytest

from nuray_gb300 import Scene, scenes
from nuray_gb300._lib import check, lib
from oracle.bind import Oracle

pytestmark = pytest.mark.gpu
N = 1 << 19


def _scene(name):
    if name == "mixed":
        return scenes.small_scene(3, env=False, textures=False)
    return scenes.terrain_spheres(2, tiles=16, cells_per_tile=8, spheres=40, slices=10, stacks=8, lights=8, n_mats=12,
                                  extent=128.0)


def _rays(S, sc, kind, r):
    lo, hi = sc["pos"].reshape(-1, 3).min(0), sc["pos"].reshape(-1, 3).max(0)
    if kind == "anywhere":
        return r.uniform(lo, hi, (N, 3)).astype(np.float32), r.standard_normal((N, 3)).astype(np.float32)
    eye = np.array([0.5 * (lo[0] + hi[0]), hi[1] + 0.5 * (hi[2] - lo[2]), hi[2]])
    at = np.stack([r.uniform(lo[0], hi[0], N), np.full(N, lo[1]), r.uniform(lo[2], hi[2], N)], 1)
    d = at - eye
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    o = np.broadcast_to(eye, (N, 3)).astype(np.float32).copy()
    if kind == "camera":
        return o, d
    t = S.intersect(o, d)[1]
    o = np.where((t < 1e17)[:, None], o + (t[:, None] - 1e-3) * d, o).astype(np.float32)
    return o, r.standard_normal((N, 3)).astype(np.float32)


@pytest.mark.parametrize("kind", ["anywhere", "camera", "surface"])
@pytest.mark.parametrize("name", ["mixed", "terrain"])
def test_the_walks_agree(gpu_lib, port_lib, name, kind):
    sc = _scene(name)

    def make(options=""):
        return Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], options=options)

    S = make()
    T = make(f"max_device_bytes={S.info()['device_bytes'] - 1}")  # no four-wide tree
    o, d = _rays(S, sc, kind, np.random.default_rng(5))
    binary = S.intersect(o, d)
    assert np.mean(binary[0] >= 0) > 0.1
    half = [S.intersect(o[a:a + N // 2], d[a:a + N // 2]) for a in (0, N // 2)]
    for a, b, c, e in zip(binary, *half, T.intersect(o[:N // 2], d[:N // 2])):
        np.testing.assert_array_equal(a, np.concatenate([b, c]))
        np.testing.assert_array_equal(a[:N // 2], e)
    for scene in (S, T):
        m = 65536
        out = np.zeros(m, np.int32), *(np.zeros(m, np.float32) for _ in range(3))
        check(lib().nr_intersect_noalloc(scene._h, m, *(a.ctypes.data for a in (o[:m], d[:m]) + out)))
        for a, b in zip(binary, out):
            np.testing.assert_array_equal(a[:m], b)
    m = 20000
    P = Oracle("port", sc)
    for a, b in zip(S.intersect(o[:m], d[:m], exhaustive=True), P.intersect(o[:m], d[:m])):
        np.testing.assert_array_equal(a, b)
