"""What the framework's speed is measured on: calls that its users make, through its public entry points.

A case is a dict with a "kind" (the call), the scene it works on and its
sizes. Every state owns its scene handle or its cache, as a user's program
does; the host arrays of a scene are generated once per process. A seed
moves the camera a little and picks the random numbers (the Philox seed of a
frame, the rays of a query, the rows of a cache call).
"""
import functools
import math

import numpy as np
import torch

import nuray_gb300.scenes as scenes
from nuray_gb300 import Scene, inverse
from nuray_gb300._lib import MAT_GGXR, MAT_GLASS, MAT_LAMBERT, MAT_LIGHT
from nuray_gb300.nrc import INPUTS, OFF, Cache


# ---------------------------------------------------------------- scenes
def _box():
    """A room open to the viewer, two blocks (glossy and glass) and a ceiling light: 36 triangles."""
    pos, nrm, mat = [], [], []

    def quad(a, b, c, d, m):
        a, b, c, d = (np.array(v, float) for v in (a, b, c, d))
        n = np.cross(b - a, c - a)
        n /= np.linalg.norm(n)
        for t in ((a, b, c), (a, c, d)):
            pos.append(np.concatenate(t)), nrm.append(np.tile(n, 3)), mat.append(m)

    def block(cx, cz, s, h, turn, m):
        u = s * np.array([math.cos(turn), 0, math.sin(turn)])
        w = s * np.array([-math.sin(turn), 0, math.cos(turn)])
        c, up = np.array([cx, 0.0, cz]), np.array([0, h, 0.0])
        p = [c - u - w, c + u - w, c + u + w, c - u + w]
        q = [x + up for x in p]
        for i in range(4):
            j = (i + 1) % 4
            quad(p[i], q[i], q[j], p[j], m)
        quad(q[0], q[3], q[2], q[1], m)
        quad(p[0], p[1], p[2], p[3], m)

    x, y, z = 100.0, 200.0, 100.0
    quad((-x, 0, -z), (-x, 0, z), (x, 0, z), (x, 0, -z), 0)
    quad((-x, y, -z), (x, y, -z), (x, y, z), (-x, y, z), 0)
    quad((-x, 0, -z), (x, 0, -z), (x, y, -z), (-x, y, -z), 0)
    quad((-x, 0, z), (-x, 0, -z), (-x, y, -z), (-x, y, z), 1)
    quad((x, 0, -z), (x, 0, z), (x, y, z), (x, y, -z), 2)
    block(-40, -30, 28, 110, 0.3, 3)
    block(40, 25, 28, 60, -0.3, 4)
    quad((-30, y - 1, -30), (30, y - 1, -30), (30, y - 1, 30), (-30, y - 1, 30), 5)
    mats = [dict(type=MAT_LAMBERT, c0=[0.7, 0.7, 0.7]), dict(type=MAT_LAMBERT, c0=[0.63, 0.06, 0.05]),
            dict(type=MAT_LAMBERT, c0=[0.15, 0.48, 0.09]), dict(type=MAT_GGXR, c0=[0.8, 0.8, 0.8], alpha=0.2),
            dict(type=MAT_GLASS, c0=[0.04, 0.04, 0.04], ior=1.5), dict(type=MAT_LIGHT, c0=[12.0, 12.0, 12.0])]
    n = len(pos)
    return dict(pos=np.array(pos, np.float32), nrm=np.array(nrm, np.float32), uv=np.zeros((n, 6), np.float32),
                mat=np.array(mat, np.int32), mats=mats, textures=[], env_tex=-1, env_gain=1.0)


# eye, yaw, pitch and field of view of each scene's own camera
_VIEW = {"terrain": ((0, 90, 130), 0, -42, 45), "sky": ((0, 90, 130), 0, -42, 45), "inverse": ((0, 50, 75), 0, -38, 50),
         "mixed": ((0, 14, 34), 0, -20, 50), "box": ((0, 100, 95), 0, 0, 64)}
# triangles, and texture and environment texels, of each scene
_TRIS = {"terrain": 991296, "sky": 991296, "inverse": 207904, "mixed": 1720, "box": 36}
_TEXELS = {"sky": 32 * 512 * 512 + 2048 * 1024, "mixed": 6 * 32 * 32 + 64 * 32}


@functools.lru_cache(maxsize=None)
def _scene(name):
    if name == "terrain":  # the benchmark's scene
        return scenes.terrain_spheres(0)
    if name == "sky":  # the same with an HDR sky, textures and dielectrics
        return scenes.with_env_textures(_scene("terrain"), 0)
    if name == "inverse":  # the inverse-rendering scene: 64 materials, GGX reflect and Lambert
        return inverse.c5_scene(0)
    if name == "mixed":  # every material type, a sky and small textures
        return scenes.small_scene(1)
    return _box()


def _open(name):
    s = _scene(name)
    return Scene.from_arrays(s["pos"], s["mat"], s["mats"], uv=s["uv"], nrm=s["nrm"], textures=s["textures"],
                             env_tex=s["env_tex"], env_gain=s["env_gain"], options="bvh=gpu")


def _view(name, seed):
    """The scene's camera, moved by up to 4 % of its distance and 3 degrees."""
    (x, y, z), yaw, pitch, fov = _VIEW[name]
    r = np.random.default_rng([seed, 17])
    d = 0.04 * math.sqrt(x * x + y * y + z * z)
    x, y, z = (a + d * b for a, b in zip((x, y, z), r.uniform(-0.5, 0.5, 3)))
    yaw, pitch = yaw + r.uniform(-3, 3), pitch + r.uniform(-3, 3)
    return [float(np.float32(round(v, 5))) for v in (x, y, z)], float(round(yaw, 5)), float(round(pitch, 5)), float(fov)


def _camera(name, w, h, seed):
    (x, y, z), yaw, pitch, fov = _view(name, seed)
    return (f"imgw={w} imgh={h} campos={x:.5f},{y:.5f},{z:.5f} cameuler={yaw:.5f},{pitch:.5f},0 camfov={fov:g} "
            f"camasp={w / h:.6f}")


def _policy(c):
    # depth 0: the reference's own policy, Russian roulette from the first vertex and no depth limit
    return f"maxdepth={c['depth']} rrdepth=3" if c["depth"] else "prr=0.8"


# ---------------------------------------------------------------- the cases
def _frame(name, scene, w, h, spp, depth, **more):
    return dict(name=name, kind="frame", scene=scene, w=w, h=h, spp=spp, depth=depth, envis=more.get("envis", False),
                rgb8=more.get("rgb8", False), nrc=more.get("nrc", False))


def listed():
    return [
        # the benchmark's frame in the steps a viewer shows it: 1M triangles, one wave of 33 M paths
        _frame("frame_1080p_16spp", "terrain", 1920, 1080, 16, 8),
        # one frame of a progressive or real-time viewer: a sample per pixel
        _frame("frame_540p_1spp", "terrain", 960, 540, 1, 8),
        # a textured outdoor scene under a sampled HDR sky, with dielectrics
        _frame("sky_540p_16spp", "sky", 960, 540, 16, 8, envis=True),
        # an interior with the reference's own policy (unbounded paths), as its command line renders to 8 bits
        _frame("box_480p_16spp", "box", 640, 480, 16, 0, rgb8=True),
        # a thumbnail of a small scene with every material type: the smallest render
        _frame("mixed_48x32_4spp", "mixed", 48, 32, 4, 0),
        # a frame whose sides and samples divide by no tile
        _frame("frame_853x481_3spp", "terrain", 853, 481, 3, 5),
        # a real-time frame that trains and asks the radiance cache
        _frame("cached_540p_1spp", "terrain", 960, 540, 1, 8, nrc=True),
        # one step of an inverse-rendering loop: materials in, image and gradient out
        dict(name="inverse_512_32spp", kind="inverse", scene="inverse", w=512, h=512, spp=32, depth=4),
        # picking: the first hits of a view's pixel centres, host arrays
        dict(name="pick_64k_rays", kind="pick", scene="inverse", w=256, h=256),
        # occlusion or visibility rays from the surfaces, device arrays
        dict(name="rays_2m", kind="rays", scene="terrain", n=2000003),
        # the cache by itself: predictions, and a training step
        dict(name="cache_infer_64k", kind="infer", n=65536),
        dict(name="cache_train_16k", kind="train", n=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["inverse", "pick", "rays", "infer", "train"])
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 1, 262144))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 64, 65536))
    if kind == "rays":
        return dict(kind=kind, scene=rng.choice(["terrain", "inverse", "mixed"]), n=_log(rng, 1000, 8000000))
    w = _log(rng, 40, 1920)
    h = max(24, int(w * rng.uniform(0.5, 1.0)))
    if rng.random() < 0.5:  # sides that tiles divide, as most users' do
        w, h = (w + 7) // 8 * 8, (h + 7) // 8 * 8
    if kind == "pick":
        return dict(kind=kind, scene=rng.choice(["inverse", "mixed", "box"]), w=min(w, 512), h=min(h, 512))
    if kind == "inverse":
        w, h = min(w, 640), min(h, 640)
        return dict(kind=kind, scene="inverse", w=w, h=h, spp=min(64, _log(rng, 1, 64), max(1, 8000000 // (w * h))),
                    depth=rng.choice([3, 4, 5]))
    scene = rng.choice(["terrain", "terrain", "sky", "box", "mixed"])
    most = {"terrain": 24, "sky": 12, "box": 16, "mixed": 16}[scene] * 1000000
    spp = min(_log(rng, 1, 64), max(1, most // (w * h)))
    nrc = scene == "terrain" and rng.random() < 0.25
    return dict(kind=kind, scene=scene, w=w, h=h, spp=spp, depth=rng.choice([0, 4, 8]) if not nrc else 8,
                envis=scene in ("sky", "mixed") and rng.random() < 0.5, rgb8=rng.random() < 0.3, nrc=nrc)


# ---------------------------------------------------------------- inputs
def _pick_rays(name, w, h, seed):
    """Rays through the pixel centres of the scene's view, as a user's picking code makes them."""
    eye, yaw, pitch, fov = _view(name, seed)
    a, b = math.radians(yaw), math.radians(pitch)
    gaze = np.array([math.sin(a) * math.cos(b), math.sin(b), -math.cos(a) * math.cos(b)])
    hand = np.cross(gaze, (0, 1, 0))
    hand /= np.linalg.norm(hand)
    up = np.cross(hand, gaze)
    xs, ys = np.meshgrid((np.arange(w) + 0.5) / w * 2 - 1, (np.arange(h) + 0.5) / h * 2 - 1)
    f = math.tan(math.radians(fov) / 2)
    d = gaze + (xs.ravel() * f * w / h)[:, None] * hand - (ys.ravel() * f)[:, None] * up
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.tile(np.array(eye), (w * h, 1)).astype(np.float32), d.astype(np.float32)


def _surface_rays(name, n, seed):
    """Cosine-weighted rays leaving uniformly drawn triangles, in no order."""
    s = _scene(name)
    g = torch.Generator(device="cuda").manual_seed(seed)
    pos, nrm = torch.from_numpy(s["pos"]).cuda(), torch.from_numpy(s["nrm"]).cuda()
    k = torch.randint(pos.shape[0], (n,), generator=g, device="cuda")
    b = torch.rand((n, 2), generator=g, device="cuda")
    b = torch.where(b.sum(1, keepdim=True) > 1, 1 - b, b)
    p, m = pos[k].view(n, 3, 3), torch.nn.functional.normalize(nrm[k].view(n, 3, 3)[:, 0], dim=1)
    at = p[:, 0] + b[:, :1] * (p[:, 1] - p[:, 0]) + b[:, 1:] * (p[:, 2] - p[:, 0])
    d = m + 0.999 * torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    return (at + 1e-3 * m).contiguous(), torch.nn.functional.normalize(d, dim=1).contiguous()


def _rows(n, seed):
    """Encoded vertices (frequencies of a position, directions, roughness, albedo) and radiance targets."""
    r = np.random.default_rng([seed, 23])
    p = r.uniform(0, 1, (n, 3, 1)) * 2.0 ** np.arange(12) * np.pi
    x = np.concatenate([np.stack([np.sin(p), np.cos(p)], -1).reshape(n, 72), r.uniform(0, 1, (n, 8))], 1)
    y = r.gamma(0.7, 0.8, (n, 3)) * (0.2 + x[:, 77:80])
    return x.astype(np.float32), y.astype(np.float32)


def prepare(case, seed):
    c = dict(case)
    k = c["kind"]
    if k in ("infer", "train"):
        x, y = _rows(c["n"], seed)
        return dict(case=c, cache=Cache(f"seed={seed % 65536}"), x=x, y=y)
    s = dict(case=c, scene=_open(c["scene"]))
    if k == "pick":
        s["o"], s["d"] = _pick_rays(c["scene"], c["w"], c["h"], seed)
    elif k == "rays":
        s["o"], s["d"] = _surface_rays(c["scene"], c["n"], seed)
        s["tri"] = torch.empty(c["n"], dtype=torch.int32, device="cuda")
        s["hit"] = torch.empty((3, c["n"]), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
    else:
        s["params"] = f"renderer=ptnee {_camera(c['scene'], c['w'], c['h'], seed)} spp={c['spp']} {_policy(c)} seed={seed}"
        if k == "inverse":
            r = np.random.default_rng([seed, 29])
            mats = [dict(m) for m in _scene(c["scene"])["mats"]]
            for m in mats:
                if m["type"] != MAT_LIGHT:
                    m["c0"] = [float(v) for v in np.clip(np.array(m["c0"]) * r.uniform(0.8, 1.2, 3), 0, 1)]
            s["mats"] = mats
            s["target"] = r.uniform(0, 1, (c["h"], c["w"], 3)).astype(np.float32)
            s["again"] = s["params"].replace(f" seed={seed}", f" seed={seed + 1000}")
        else:
            s["params"] += " envis=1" if c["envis"] else ""
            if c["nrc"]:
                s["params"] += " nrc=1"
                s["cache"] = Cache("")
                s["cache"].attach(s["scene"])
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "frame":
        out = s["scene"].render(s["params"], want_rgb8=c["rgb8"])
        out = dict(hdr=out[0], rgb8=out[1]) if c["rgb8"] else dict(hdr=out)
        if c["nrc"]:
            out["weights"] = s["cache"].get_params()
        return out
    if k == "inverse":
        s["scene"].set_materials(s["mats"])
        image = s["scene"].render(s["params"])
        return dict(image=image, grad=s["scene"].adjoint(s["again"], (image - s["target"]) * np.float32(2.0 / image.size)))
    if k == "pick":
        return dict(zip(("tri", "t", "b1", "b2"), s["scene"].intersect(s["o"], s["d"])))
    if k == "rays":
        h = s["hit"]
        s["scene"].intersect_device(c["n"], s["o"].data_ptr(), s["d"].data_ptr(), s["tri"].data_ptr(), h[0].data_ptr(),
                                    h[1].data_ptr(), h[2].data_ptr())
        return dict(tri=s["tri"], hit=h)
    if k == "infer":
        return dict(out=s["cache"].infer(s["x"]))
    loss = s["cache"].train_step(s["x"], s["y"])
    return dict(loss=loss, weights=s["cache"].get_params())


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: the scene, the inputs and the outputs, once each. Flops: per
    ray, both boxes of every level of a balanced binary tree (21 each) and two
    triangles (45 each); per vertex the light sample, the material's value
    and density twice and its sample (400); the cache's multiplies."""
    c = case
    k = c["kind"]
    net = 2.0 * (80 * 64 + 3 * 64 * 64 + 64 * 3)
    weights = 4.0 * sum(n for _, n in OFF.values())
    if k == "infer":
        return dict(bytes=c["n"] * (4.0 * INPUTS + 12) + weights, flops=c["n"] * net)
    if k == "train":
        return dict(bytes=c["n"] * (4.0 * INPUTS + 12) + 8 * weights, flops=3.0 * c["n"] * net)
    tris = _TRIS[c["scene"]]
    ray = 2 * 21 * math.log2(tris) + 2 * 45
    scene = 100.0 * tris + 12.0 * _TEXELS.get(c["scene"], 0)
    if k in ("pick", "rays"):
        n = c["n"] if k == "rays" else c["w"] * c["h"]
        return dict(bytes=48.0 * tris + 40.0 * n, flops=n * ray)
    # extension rays of a path: outdoors about half of the paths leave at each vertex, a room keeps most
    going = 0.8 if c["scene"] == "box" else 0.55
    depth = c["depth"] or 64
    rays = sum(going ** i for i in range(depth))
    per_path = rays * (1 + 0.5 * (2 if c.get("envis") else 1)) * ray + rays * 400
    pixels = c["w"] * c["h"]
    flops = pixels * c["spp"] * per_path
    if k == "inverse":
        return dict(bytes=2 * scene + 36.0 * pixels, flops=2 * flops + pixels * c["spp"] * rays * 800)
    return dict(bytes=scene + (15.0 if c["rgb8"] else 12.0) * pixels, flops=flops)


# ---------------------------------------------------------------- the same in 64 bits
def _mlp(p, x, y):
    """Output, relative L2 loss and its gradient of the 80-64-64-64-64-3 ReLU network in float64."""
    w = {k: p[o:o + n].clone().requires_grad_(True) for k, (o, n) in OFF.items()}
    a = x
    for i in range(4):
        a = torch.relu(a @ w[f"W{i}"].view(64, -1).T + w[f"b{i}"])
    o = (a @ w["W4"].view(8, 64).T + w["b4"])[:, :3]
    loss = ((o - y) ** 2 / (o.detach() ** 2 + 0.01)).mean()
    loss.backward()
    g = torch.zeros_like(p)
    for k, (at, n) in OFF.items():
        g[at:at + n] = w[k].grad
    return o.detach(), loss.detach(), g


def _first_hits(pos, o, d):
    """t, b1, b2 of the nearest triangle over all of them: o + t d against p0
    + b1 e1 + b2 e2 with the determinant biased by 1e-6, as the reference's
    triangles have it; 1e18, 0, 0 for a miss."""
    p0, e1, e2 = pos[:, 0], pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0]
    cr = torch.linalg.cross
    n = cr(e1, e2)
    ta, tb, tc = (n * p0).sum(1), torch.cat([-cr(e2, p0), e2], 1), torch.cat([cr(e1, p0), -e1], 1)
    out = torch.empty((3, o.shape[0]), dtype=torch.float64, device=o.device)
    for i in range(0, o.shape[0], 2048):
        O, D = o[i:i + 2048], d[i:i + 2048]
        # (d x e2).e1 = -d.n, (d x e2).(o - p0), ((o - p0) x e1).d and ((o - p0) x e1).e2
        q = -(D @ n.T) + 1e-6
        L = torch.cat([D, cr(O, D)], 1)
        u = (L @ tb.T) / q
        v = (L @ tc.T) / q
        t = (O @ n.T - ta) / q
        t = torch.where((t > 0) & (u >= 0) & (v >= 0) & (u + v <= 1), t, 1e18)
        best, k = t.min(1)
        hit, j = best < 1e18, torch.arange(k.shape[0], device=o.device)
        out[:, i:i + 2048] = torch.stack([best, torch.where(hit, u[j, k], 0.0), torch.where(hit, v[j, k], 0.0)])
    return out


def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "pick" and c["w"] * c["h"] * _TRIS[c["scene"]] < 2e10:
        o, d = _pick_rays(c["scene"], c["w"], c["h"], seed)
        pos = torch.from_numpy(_scene(c["scene"])["pos"]).cuda().double().view(-1, 3, 3)
        h = _first_hits(pos, torch.from_numpy(o).cuda().double(), torch.from_numpy(d).cuda().double())
        return dict(tri=None, t=h[0], b1=h[1], b2=h[2])
    if k not in ("infer", "train"):
        return None  # a path tracer's image: no value in 64 bits within seconds
    x, y = (torch.from_numpy(a).cuda().double() for a in _rows(c["n"], seed))
    # the cache's own first weights are an input here
    p = torch.from_numpy(Cache(f"seed={seed % 65536}").get_params()).cuda().double()
    o, loss, g = _mlp(p, x, y)
    if k == "infer":
        return dict(out=o)
    # Adam's first step: lr 1e-3, beta 0.9 and 0.99, eps 1e-8
    return dict(loss=float(loss), weights=p - 1e-3 * g / (g.abs() + 1e-8))
