"""Bounces of 4M paths or more sort their new rays by origin and direction
(scenes of 16,384 triangles or more); smaller waves leave them in queue
order. Either way every path has its own sums: the same image."""
import numpy as np
import pytest

from nuray_gb300 import Scene, scenes

pytestmark = pytest.mark.gpu

CAM = "campos=0,45,65 cameuler=0,-42,0 camfov=45 camasp=1.25 maxdepth=4 rrdepth=2 seed=5"


def _scene(options="", **more):
    sc = scenes.terrain_spheres(2, tiles=16, cells_per_tile=8, spheres=40, slices=10, stacks=8, lights=8, n_mats=12,
                                extent=128.0, mixed_materials=True)
    if more.get("env"):
        sc = scenes.with_env_textures(sc, 2, tex_size=32, env_size=(64, 32))
    S = Scene.from_arrays(sc["pos"], sc["mat"], sc["mats"], uv=sc["uv"], nrm=sc["nrm"], textures=sc["textures"],
                          env_tex=sc["env_tex"], env_gain=sc["env_gain"], options=options)
    assert S.info()["tris"] >= 16384
    return S


def _tight(w, h, paths, sh_mult, S, spare):
    """max_device_bytes: the scene, the path state of one wave and the outputs, and `spare` bytes."""
    return (S.info()["device_bytes"] + paths * (5 * 16 + 16 + 2 * 4 + 7 * 4 + 3 * 16 * sh_mult) + w * h * (16 + 12 + 3)
            + spare)


@pytest.mark.parametrize("envis", [0, 1])
@pytest.mark.parametrize("w,h,spp", [(320, 256, 49), (320, 256, 52), (641, 399, 33)])
def test_sorted_wave_gives_the_same_image(gpu_lib, w, h, spp, envis):
    """Waves of 4.01, 4.26 (one kernel per material from there) and 8.44 M
    paths: the same kernels sorted, and unsorted for want of room."""
    S = _scene(env=bool(envis))
    p = f"renderer=ptnee imgw={w} imgh={h} spp={spp} {CAM} envis={envis} tail=0"
    a = S.render(p)
    launches = S.stats()["kernel_launches"]
    T = _scene(f"max_device_bytes={_tight(w, h, w * h * spp, 1 + envis, S, 8 << 20)}", env=bool(envis))
    b = T.render(p)
    assert launches > T.stats()["kernel_launches"]  # the sort's own
    assert np.all(np.isfinite(a)) and a.mean() > 0
    np.testing.assert_array_equal(a, b)


def test_sorted_adjoint_gives_the_same_gradient(gpu_lib):
    S = _scene()
    p = f"renderer=ptnee imgw=320 imgh=256 spp=64 {CAM}"
    dl = np.random.default_rng(3).standard_normal((256, 320, 3)).astype(np.float32) / (320 * 256)
    a, ia = S.adjoint(p, dl, want_image=True)
    b, ib = S.adjoint(p + " wave=1000000", dl, want_image=True)
    np.testing.assert_allclose(ia, ib, rtol=1e-5, atol=1e-6)
    np.testing.assert_allclose(a, b, rtol=1e-3, atol=1e-4 * np.abs(a).max())  # float atomics in any order


def test_without_room_for_the_sort_the_render_still_runs(gpu_lib):
    """max_device_bytes that holds the scene and the path state of a 4.2M-path
    wave, but not the sort's workspace, nor that and the outputs at once."""
    p = f"renderer=ptnee imgw=320 imgh=256 spp=52 {CAM} tail=0"
    S = _scene()
    ref = S.render(p)
    for spare in (1 << 20, 60 << 20, 118 << 20, 119 << 20, 200 << 20):
        T = _scene(f"max_device_bytes={_tight(320, 256, 320 * 256 * 52, 1, S, spare)}")
        hdr, rgb8 = T.render(p, want_rgb8=True)
        np.testing.assert_array_equal(hdr, ref)
        np.testing.assert_array_equal(T.render(p), ref)
        T.close()


@pytest.mark.parametrize("w,h,spp", [(320, 256, 52), (641, 399, 33)])
@pytest.mark.parametrize("more", ["", "nrc=1", "nrc=1 nrc_steps=1", "nrc=1 nrc_steps=1 nrc_train_depth=0", "renderer=nrc"])
def test_waves_with_and_without_room_for_the_sort(gpu_lib, more, w, h, spp):
    """Several Adam steps a wave take consecutive chunks of the training
    records, and a full table keeps the first of them: such a wave is traced
    sorted but bucketed and shaded in path order. Every wave gives the unsorted
    one's first image, which no training has touched."""
    from nuray_gb300.nrc import Cache
    S = _scene()
    c = Cache("seed=1")
    p = f"renderer=ptnee imgw={w} imgh={h} spp={spp} {CAM} tail=0 "
    p = p.replace("renderer=ptnee", more) if "renderer" in more else p + more
    c.attach(S)
    a = S.render(p)
    with_order = S.stats()["kernel_launches"]
    S.render(p + " profile=1")
    assert S.stats()["kernel_launches"] == with_order
    # the same with room for the path state and the cache's records, but not for the sort (119 MB and more)
    records = (w * h * spp * 64 + 16384 * 4 * 196) if "nrc" in more else 0
    T = _scene("max_device_bytes=%d" % _tight(w, h, w * h * spp, 1, S, records + (16 << 20)))
    d = Cache("seed=1")
    d.attach(T)
    b = T.render(p)
    assert with_order > T.stats()["kernel_launches"]
    if "renderer" not in more:  # whose first pass trains before the samples
        np.testing.assert_array_equal(a, b)


def test_a_wave_whose_tail_keeps_its_order_is_not_sorted(gpu_lib):
    """4.05M paths, several Adam steps: two bounces in path order, then the tail, which appends records as its queue stands."""
    from nuray_gb300.nrc import Cache
    launches = []
    for more in ("nrc=1 nrc_steps=3", "nrc=1 nrc_steps=1"):
        S = _scene()
        c = Cache("seed=1")
        c.attach(S)
        S.render(f"renderer=ptnee imgw=320 imgh=256 spp=49 {CAM} {more} tail=2")
        launches.append(S.stats()["kernel_launches"])
    # 3 launches for each of two bounces' sorts; an Adam step is 4 launches
    assert launches[0] == launches[1] - 2 * 3 + 2 * 4
