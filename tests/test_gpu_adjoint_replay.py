"""The adjoint's second pass follows the paths whose radiance the first pass
rendered, also through bounces that it traces again for want of records.
The scene is small enough that the biased determinant shortens most hits'
t (q / (q + 1e-6) below 0.99): which triangle wins then depends on the order
of a walk's leaves, and replays by another walk end elsewhere.

Radiance is linear in the emission, and nothing else emits here, so
sum(emission * its gradient) = sum(dL/dimage * image). With dL/dimage = +-1 a
pixel, paths that end elsewhere put the two sides apart by about
sqrt(share of such paths / spp) of the pixels' root sum of squares; FP32 sums
of some 4000 terms of either sign a block by less than 1e-5 of it."""
import numpy as np
import pytest

from nuray_gb300 import Scene, scenes

pytestmark = pytest.mark.gpu
SCALE = 3e-3


def _scene():
    sc = scenes.terrain_spheres(2, tiles=16, cells_per_tile=8, spheres=40, slices=10, stacks=8, lights=8, n_mats=12,
                                extent=128.0, mixed_materials=True)
    S = Scene.from_arrays((sc["pos"] * SCALE).astype(np.float32), sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"])
    ke = np.array([m.get("c0", [0, 0, 0]) if m["type"] == 5 else [0, 0, 0] for m in sc["mats"]], np.float64)
    return S, ke


@pytest.mark.parametrize("policy", ["maxdepth=4 rrdepth=2", "prr=0.6"])
@pytest.mark.parametrize("w,h,spp", [(160, 128, 4), (320, 256, 56)])  # unsorted bounces; sorted ones (4.6 M paths)
@pytest.mark.parametrize("trav", [0, 1])
def test_replayed_paths_are_the_rendered_ones(gpu_lib, w, h, spp, policy, trav):
    S, ke = _scene()
    p = (f"renderer=ptnee imgw={w} imgh={h} spp={spp} campos=0,{45 * SCALE},{65 * SCALE} cameuler=0,-42,0 camfov=45 "
         f"camasp=1.25 seed=5 trav={trav} {policy}")
    dl = np.random.default_rng(3).choice([-1.0, 1.0], (h, w, 1)).repeat(3, 2).astype(np.float32)
    per_bounce = w * h * spp * 17  # hits (16 bytes a path) and visibility
    for records in (None, 0, per_bounce + (1 << 16)):  # every bounce recorded, none, the first
        more = "" if records is None else f" adj_records={records}"
        g, img = S.adjoint(p + more, dl, want_image=True)
        lhs, rhs = float(np.sum(ke * g[:, 4:7])), float(np.sum(dl.astype(np.float64) * img))
        scale = float(np.sqrt(np.sum(img.astype(np.float64) ** 2)))
        assert scale > 0
        assert abs(lhs - rhs) <= 1e-3 * scale, (records, lhs, rhs, scale)
