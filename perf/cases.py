"""Performance cases: what programs have this renderer do, from one preview sample to a full frame.

Each case goes through the public Python classes (SceneBuffers, EnvMap, Pathtracer, RadianceCache,
RenderServer), as a program that uses the package calls them.  Scenes are the seeded generators of
nbounce_gb300.scenes with their own proportions; sizes are those of the benchmark workloads
(256x256 at 16 spp, 1920x1080 at 64 spp, the 1M-triangle soup, 16,384 training rows, the job mix of
the server) and odd sizes between them.

kinds
  render  a still image or one step of a progressive preview: invalidate, then n samples per pixel
  cache   a real-time loop with the learned radiance cache: 1-spp frames along a camera path, each of
          which trains the cache, then a snapshot of its weights
  trace   the traversal query on the caller's own rays, on the device (baking, visibility) or with
          host buffers (picking)
  train   optimiser steps of the cache network on the caller's batches, then a snapshot
  infer   the cache network on the caller's encoded rows
  serve   a burst of render requests through the job server, images delivered to host memory
"""
import math

import numpy as np
import torch

import nbounce_gb300 as nb
from nbounce_gb300 import _lib as L
from nbounce_gb300 import scenes
from nbounce_gb300.server import RenderServer


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def _render(name, scene, detail, env, w, h, spp, bounces=8, nee=False, rr=0):
    return dict(name=name, kind="render", scene=scene, detail=detail, env=env, width=w, height=h, spp=spp,
                bounces=bounces, nee=nee, rr=rr)


def listed():
    return [
        # a thumbnail-sized preview while the camera moves: latency and launches
        _render("preview_64x48_1spp", "spheres", 0, "constant", 64, 48, 1),
        # the reference's window (1920x1080 scaled by 0.3, rounded down to 8): one dispatch per shown frame
        _render("window_576x320_1spp", "instanced", 1 / 16, "equirect", 576, 320, 1),
        # the 64-icosphere benchmark frame
        _render("spheres_256x256_16spp", "spheres", 0, "constant", 256, 256, 16, bounces=6),
        # sun-lit still with environment next-event estimation, cube map, roulette from bounce 3, odd size
        _render("nee_cube_1013x571_3spp", "instanced", 1 / 16, "cube", 1013, 571, 3, nee=True, rr=3),
        # the headline frame's shape: 16 meshes in 1024 instances, 1080p, 64 spp, 8 bounces
        _render("frame_1920x1080_64spp", "instanced", 1 / 4, "equirect", 1920, 1080, 64),
        # real-time loop with the radiance cache
        dict(name="cache_1920x1080_4frames", kind="cache", detail=1 / 16, width=1920, height=1080, frames=4,
             spread=0.01),
        # camera-like rays against the 1M-triangle soup, closest hit
        dict(name="rays_camera_2048x2048", kind="trace", tris=1 << 20, rays=2048 * 2048, coherent=True, any_hit=False,
             host=False),
        # scattered occlusion rays (ambient occlusion, light baking)
        dict(name="rays_scattered_any_4000037", kind="trace", tris=1 << 20, rays=4000037, coherent=False, any_hit=True,
             host=False),
        # picking: a few rays from host memory, hits back in host memory
        dict(name="rays_host_1531", kind="trace", tris=20480, rays=1531, coherent=False, any_hit=False, host=True),
        # one frame's training in the cache workload's configuration: 65,536 records in 4 Adam steps
        dict(name="train_4x16384", kind="train", rows=16384, steps=4),
        # lookups of about half a 1080p frame, a ragged count
        dict(name="infer_1000003", kind="infer", rows=1000003),
        # a burst of thumbnails and previews from several users
        dict(name="serve_12_jobs", kind="serve", jobs=12, detail=1 / 64, largest=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "cache", "trace", "trace", "train", "infer", "serve"])
    if kind == "render":
        w, h = _log(rng, 33, 1920), _log(rng, 27, 1080)
        spp = min(_log(rng, 1, 64), max(1, (1 << 24) // (w * h)))
        scene = rng.choice(["spheres", "instanced", "instanced"])
        detail = 1 / rng.choice([16, 64, 512]) if scene == "instanced" else 0
        return {k: v for k, v in
                _render("", scene, detail, rng.choice(["constant", "equirect", "cube"]), w, h, spp,
                        bounces=rng.choice([3, 6, 8]), nee=rng.random() < 0.33, rr=rng.choice([0, 0, 3])).items()
                if k != "name"}
    if kind == "cache":
        return dict(kind="cache", detail=1 / rng.choice([64, 512]), width=_log(rng, 97, 1920),
                    height=_log(rng, 65, 1080), frames=rng.choice([1, 2, 4]), spread=rng.choice([0.01, -1.0]))
    if kind == "trace":
        host = rng.random() < 0.25
        coherent = rng.random() < 0.5
        rays = _log(rng, 65, 100000) if host else _log(rng, 1000, 1 << 22)
        if coherent:  # a camera grid
            side = max(8, int(math.sqrt(rays)))
            rays = side * side
        return dict(kind="trace", tris=_log(rng, 2000, 1 << 19), rays=rays, coherent=coherent,
                    any_hit=rng.random() < 0.5, host=host)
    if kind == "train":
        return dict(kind="train", rows=_log(rng, 1000, 40000), steps=rng.choice([1, 2, 4]))
    if kind == "infer":
        return dict(kind="infer", rows=_log(rng, 1000, 2000000))
    return dict(kind="serve", jobs=rng.randint(2, 16), detail=1 / 512, largest=rng.choice([256, 320, 512]))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _eye(seed):
    """The workload's camera, a little elsewhere for each seed."""
    rng = np.random.default_rng([seed, 7])
    return rng.uniform(-1.0, 1.0, 3) * np.array([3.0, 1.0, 3.0])


def _scene(scene, detail, seed, width, height):
    if scene == "spheres":
        d = scenes.spheres_scene(seed=0x5EED0 + seed, width=width, height=height)
        eye, target = np.array([0.0, 6.0, 34.0]), (0.0, -1.0, 0.0)
    else:
        d = scenes.instanced_scene(seed=0x5EED1 + seed, scale=detail, width=width, height=height, env_size=(16, 8))
        eye, target = np.array([0.0, 14.0, 62.0]), (0.0, -2.0, 0.0)
    w2c, c2w = scenes.camera_matrices(eye + _eye(seed), target, width, height)
    return nb.SceneBuffers.from_desc(d), nb.camera_struct(w2c, c2w)


def _env(env, seed):
    if env == "constant":
        return nb.EnvMap((0.5, 0.6, 0.8))
    sky = scenes.sky_envmap(seed + 1, 1024, 512)
    return nb.EnvMap(texels=sky) if env == "equirect" else nb.EnvMap(cube=scenes.cube_from_equirect(sky, 256))


class _DeviceImage:
    """The path tracer's image as an array that torch can view; a view keeps the path tracer, whose memory it is."""

    def __init__(self, pt):
        self.pt = pt
        p, w, h = pt.output_texture()
        self.__cuda_array_interface__ = {"shape": (h, w, 4), "typestr": "<f4", "data": (p, False), "version": 3}


def _weights(seed):
    """A plausible network: uniform weights of variance 2 / fan-in, the unused output rows zero."""
    rng = np.random.default_rng([seed, 11])
    w = (rng.uniform(-1.0, 1.0, nb.cache.N_PARAMS) * math.sqrt(6.0 / 64.0)).astype(np.float32)
    w[5 * 4096 + 3 * 64:] = 0.0
    return w


def _rows(n, seed):
    """Encoded rows as the cache sees them (values in [0, 1], input 62 is the constant 1) and positive targets."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(n, nb.cache.N_INPUTS, generator=g, device="cuda")
    x[:, 62] = 1.0
    return x, torch.rand(n, 3, generator=g, device="cuda") * 2.0


def _soup_rays(case, seed):
    """(n, 8) rays on the device: a pinhole grid in front of the soup, or scattered through it."""
    n = case["rays"]
    rays = torch.zeros(n, 8, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["coherent"]:
        side = int(round(math.sqrt(n)))
        c = (torch.arange(side, device="cuda") + torch.rand(1, generator=g, device="cuda")) / side * 2.0 - 1.0
        y, x = torch.meshgrid(c, c, indexing="ij")
        d = torch.stack([x * math.tan(math.pi / 6), y * math.tan(math.pi / 6), -torch.ones_like(x)], -1).reshape(-1, 3)
        rays[:, 2] = 3.0
    else:
        rays[:, :3] = torch.rand(n, 3, generator=g, device="cuda") * 2.0 - 1.0
        d = torch.randn(n, 3, generator=g, device="cuda")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return rays


def _jobs(case, seed):
    """A burst of the server's job mix: thumbnails to `largest`, a few with environment NEE; the seed moves the
    cameras."""
    rng, place = np.random.default_rng(case["jobs"]), np.random.default_rng([seed, 13])
    n, m = case["largest"], []
    for _ in range(case["jobs"]):
        w, h = ((n, n), (n // 2, n // 2), (n, n * 3 // 4), (n // 2 + 7, n // 4 + 5))[rng.integers(4)]
        m.append((int(rng.integers(2)), int(w), int(h), int((1, 4, 16)[rng.integers(3)]),
                  L.NB_JOB_ENV_NEE if rng.uniform() < 0.25 else 0, place.uniform(-4.0, 4.0, 3)))
    return m


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "render":
        w, h = case["width"], case["height"]
        s["scene"], s["camera"] = _scene(case["scene"], case["detail"], seed, w, h)
        s["env"] = _env(case["env"], seed)
        s["pt"] = nb.Pathtracer(w, h, nb.Globals(bounces=case["bounces"]))
        s["pt"].set_sampling(env_nee=case["nee"])
        s["pt"].set_rr_start_bounce(case["rr"])
        s["image"] = torch.as_tensor(_DeviceImage(s["pt"]), device="cuda")
    elif kind == "cache":
        w, h = case["width"], case["height"]
        s["scene"], _ = _scene("instanced", case["detail"], seed, w, h)
        s["env"] = _env("equirect", seed)
        s["cameras"] = [nb.camera_struct(*scenes.camera_matrices(e, t, w, h))
                        for e, t in scenes.camera_path(max(2, case["frames"]), seed=seed)][:case["frames"]]
        s["cache"] = nb.RadianceCache(seed=1 + seed % 1000003, spread=case["spread"])
        s["pt"] = nb.Pathtracer(w, h, nb.Globals(bounces=8))
        s["pt"].set_cache(s["cache"])
        s["image"] = torch.as_tensor(_DeviceImage(s["pt"]), device="cuda")
    elif kind == "trace":
        s["scene"] = nb.SceneBuffers.from_desc(scenes.soup_scene(case["tris"], seed=0x5EED2 + seed))
        s["rays"] = _soup_rays(case, seed)
        if case["host"]:
            s["rays"] = s["rays"].cpu().numpy()
        else:
            s["hits"] = torch.empty(case["rays"], 4, device="cuda")
            s["instances"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
    elif kind in ("train", "infer"):
        s["cache"] = nb.RadianceCache()
        s["cache"].set_weights(_weights(seed))
        if kind == "train":
            s["batches"] = [_rows(case["rows"], seed * 64 + k) for k in range(case["steps"])]
        else:
            s["x"] = _rows(case["rows"], seed)[0]
            s["out"] = torch.empty(case["rows"], 3, device="cuda")
    else:
        s["server"] = RenderServer()
        slots = [s["server"].add_scene(_scene(k, case["detail"], seed, 64, 64)[0]) for k in ("spheres", "instanced")]
        s["env"] = s["server"].add_env(_env("equirect", seed))
        eyes, s["jobs"] = ((0.0, 6.0, 34.0), (0.0, 14.0, 62.0)), []
        for k, w, h, spp, flags, move in _jobs(case, seed):
            w2c, c2w = scenes.camera_matrices(np.array(eyes[k]) + move, (0.0, -1.0, 0.0), w, h)
            s["jobs"].append((slots[k], w2c, c2w, w, h, spp, flags, np.zeros((h, w, 4), np.float32)))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "render":
        s["pt"].invalidate()
        if case["spp"] == 1:
            s["pt"].dispatch(s["scene"], s["camera"], s["env"])
        else:
            s["pt"].render(s["scene"], s["camera"], s["env"], case["spp"])
        return s["image"]
    if kind == "cache":
        for camera in s["cameras"]:
            s["pt"].invalidate()
            s["pt"].dispatch(s["scene"], camera, s["env"])
        return {"image": s["image"], "weights": s["cache"].get_weights()}
    if kind == "trace":
        if case["host"]:
            hits, instances = s["scene"].trace_host(s["rays"], any_hit=case["any_hit"],
                                                    incoherent=not case["coherent"])
            return {"t": hits[:, 0], "uv": hits[:, 1:3], "triangle": hits.view(np.int32)[:, 3],
                    "instance": instances.view(np.int32)}
        h = s["hits"]
        s["scene"].trace_device(s["rays"].data_ptr(), case["rays"], h.data_ptr(), s["instances"].data_ptr(),
                                any_hit=case["any_hit"], incoherent=not case["coherent"])
        return {"t": h[:, 0], "uv": h[:, 1:3], "triangle": h.view(torch.int32)[:, 3], "instance": s["instances"]}
    if kind == "train":
        losses = [s["cache"].train_step(x, y, case["rows"]) for x, y in s["batches"]]
        return {"loss": np.array(losses, np.float32), "weights": s["cache"].get_weights()}
    if kind == "infer":
        s["cache"].infer(s["x"], case["rows"], s["out"])
        return s["out"]
    srv = s["server"]
    ids = [srv.submit(slot, s["env"], w2c, c2w, w, h, spp, out=out, flags=flags)
           for slot, w2c, c2w, w, h, spp, flags, out in s["jobs"]]
    for i in ids:
        info = srv.wait(i)
        if info["status"] != 0:
            raise RuntimeError(f"job {i} failed with status {info['status']}")
        srv.release(i)
    return [job[-1] for job in s["jobs"]]


# ------------------------------------------------------------------------------------------
# the work a case cannot do without
# ------------------------------------------------------------------------------------------
TRI_BYTES = 48 + 1.5 * 32 + 12 + 80 / 10  # a triangle, its share of vertex attributes, indices and tree nodes
INSTANCED_TRIS = 4.9e6                    # unique triangles of instanced_scene at detail 1
MLP_FLOPS = 2 * 20672                     # one row through the 64 -> 5 x 64 -> 3 network
MLP_GRAD_FLOPS = 2 * (20672 + 16576 + 20672)


def _query_flops(tris):
    """One traversal query: a root-to-leaf path of an 8-wide tree (8 box tests of 12 operations a node) and
    two triangle tests of 50."""
    return 96.0 * max(1.0, math.log(max(tris, 2), 8)) + 100.0


def _scene_tris(scene, detail):
    return 1282 if scene == "spheres" else INSTANCED_TRIS * max(detail, 1 / 512)


def _render_work(scene, detail, w, h, spp, nee):
    tris = _scene_tris(scene, detail)
    paths = float(w) * h * spp
    queries = paths * 1.5 * (2.0 if nee else 1.0)  # 1.5 closest-hit queries a path, as the benchmark frame has
    return min(tris * TRI_BYTES, queries * 128.0) + 16.0 * w * h, queries * (_query_flops(tris) + 200.0)


def work(case):
    kind = case["kind"]
    if kind == "render":
        b, f = _render_work(case["scene"], case["detail"], case["width"], case["height"], case["spp"], case["nee"])
    elif kind == "cache":
        px = case["width"] * case["height"]
        b, f = _render_work("instanced", case["detail"], case["width"], case["height"], 1, False)
        b, f = b * case["frames"], case["frames"] * (f + 0.3 * px * MLP_FLOPS + min(65536, px) * MLP_GRAD_FLOPS)
    elif kind == "trace":
        n = case["rays"]
        b = n * 52.0 + min(case["tris"] * (48 + 8), n * 128.0)
        f = n * _query_flops(case["tris"])
    elif kind == "train":
        n = case["rows"] * case["steps"]
        b, f = n * 67 * 4.0 + case["steps"] * nb.cache.N_PARAMS * 24.0, float(n * MLP_GRAD_FLOPS)
    elif kind == "infer":
        b, f = case["rows"] * 67 * 4.0, float(case["rows"] * MLP_FLOPS)
    else:
        b = f = 0.0
        for k, w, h, spp, flags, _ in _jobs(case, 1):
            x, y = _render_work(("spheres", "instanced")[k], case["detail"], w, h, spp, flags != 0)
            b, f = b + x, f + y
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------------
# the same outputs in 64 bits
# ------------------------------------------------------------------------------------------
def _exact_trace(case, seed):
    """Closest hits by testing every ray against every triangle (backface-culled Moller-Trumbore, hits from
    distance 0.1 on), in 64 bits on the 32-bit inputs.  The triangle numbers follow the tree's order, which
    brute force does not have."""
    v, faces = scenes.triangle_soup(case["tris"], 0x5EED2 + seed)
    p = torch.from_numpy(np.ascontiguousarray(v["pos"][faces.astype(np.int64)])).cuda().double()
    v0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    rays = _soup_rays(case, seed).double()
    miss = float(np.finfo(np.float32).max)
    t_out = torch.full((len(rays),), miss, dtype=torch.float64, device="cuda")
    uv = torch.zeros(len(rays), 2, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 25) // len(v0))
    for i in range(0, len(rays), step):
        o, d = rays[i:i + step, None, :3], rays[i:i + step, None, 4:7]
        h = torch.linalg.cross(d.expand(-1, len(v0), -1), e2[None])
        det = (e1[None] * h).sum(-1)
        sv = o - v0[None]
        u = (sv * h).sum(-1) / det
        q = torch.linalg.cross(sv, e1[None].expand_as(sv))
        w = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (det >= 1e-8) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t >= 0.1)
        best, at = torch.where(ok, t, torch.inf).min(dim=1)
        hit = torch.isfinite(best)
        t_out[i:i + step] = torch.where(hit, best, miss)
        both = torch.stack([u.gather(1, at[:, None])[:, 0], w.gather(1, at[:, None])[:, 0]], -1)
        uv[i:i + step] = torch.where(hit[:, None], both, 0.0)
    return {"t": t_out, "uv": uv, "triangle": None, "instance": None}


def _layers(w):
    """The flat weights as 64-bit [out, in] matrices."""
    out, at = [], 0
    for o, i in nb.cache.LAYER_SHAPES:
        out.append(w[at:at + o * i].reshape(o, i))
        at += o * i
    return out


def _forward(layers, x):
    for w in layers[:-1]:
        x = torch.relu(x @ w.T)
    return x @ layers[-1].T[:, :3]


def _exact_train(case, seed):
    """Adam (0.01, 0.9, 0.99, 1e-8) on the relative L2 loss whose denominator is held constant."""
    w = torch.from_numpy(_weights(seed)).cuda().double()
    m, v, losses = torch.zeros_like(w), torch.zeros_like(w), []
    cfg = nb.cache.default_config()
    lr, b1, b2, eps = cfg.learning_rate, cfg.beta1, cfg.beta2, cfg.epsilon
    for k in range(case["steps"]):
        x, y = (a.double() for a in _rows(case["rows"], seed * 64 + k))
        w.requires_grad_(True)
        p = _forward(_layers(w), x)
        loss = ((p - y) ** 2 / (p.detach() ** 2 + 0.01)).sum() / (3 * case["rows"])
        g, = torch.autograd.grad(loss, w)
        w = w.detach()
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        w = w - lr * (m / (1 - b1 ** (k + 1))) / ((v / (1 - b2 ** (k + 1))).sqrt() + eps)
        losses.append(float(loss.detach()))
    return {"loss": np.array(losses), "weights": w.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "trace" and not case["any_hit"] and case["rays"] * case["tris"] <= 2e9:
        return _exact_trace(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "infer":
        return _forward(_layers(torch.from_numpy(_weights(seed)).cuda().double()), _rows(case["rows"], seed)[0].double())
    return None  # a path-traced image takes minutes in 64 bits; which occluder is found first is not defined
