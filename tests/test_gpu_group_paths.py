"""Queries and waves that the library traces with 8 lanes per ray against the same ones traced with a
ray per lane: the hits, images, ray counts and cache weights are the same bits.

A ray per lane is had from a call with more rays than the limits, and for renders from the instrumented
traversal (enable_trace_counters), which traces a ray per lane whatever the size."""
import numpy as np
import pytest

import nbounce_gb300 as nb
from nbounce_gb300 import scenes

pytestmark = pytest.mark.gpu

LIMIT = 65536  # above it no call or wave is traced in groups: 32,768 paths, 16,384 rays, 24,576 scattered ones
EDGES = (16384, 16385, 24576, 24577, 32768)


@pytest.fixture(scope="module")
def world():
    sph = scenes.spheres_scene(width=64, height=64)
    ins = scenes.instanced_scene(n_instances=200, width=64, height=64, env_size=(64, 32), scale=1 / 128)
    room = scenes.room_scene(width=64, height=64)
    w = {}
    for k, d in (("spheres", sph), ("instanced", ins), ("room", room)):
        env = nb.EnvMap(d.env_color) if d.env_texels is None else nb.EnvMap(texels=d.env_texels)
        w[k] = (nb.SceneBuffers.from_desc(d), env)
    return w


CAMS = {"spheres": ((0.0, 6.0, 34.0), (0.0, -1.0, 0.0)), "instanced": ((0.0, 14.0, 62.0), (0.0, -2.0, 0.0)),
        "room": ((0.0, 5.0, 4.6), (0.0, 4.0, -5.0))}


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("kind", ["spheres", "instanced"])
def test_few_rays_equal_many(world, kind, any_hit):
    n = LIMIT + 37
    rays = scenes.incoherent_rays(n, seed=9)
    rays[:, :3] *= np.float32([30.0, 12.0, 30.0])
    rays[5, 4] = np.nan
    rays[6, 0] = np.inf
    rays[7, 4:7] = (0.0, -1.0, 0.0)
    scene = world[kind][0]
    hits, inst = scene.trace_host(rays, any_hit=any_hit, incoherent=True)  # a ray per lane
    assert (hits[:, 0] < 3e38).mean() > 0.05
    for m in (1, 3, 4, 5, 31, 33, 2431, *EDGES, LIMIT - 1, LIMIT):
        for incoherent in (False, True):
            h, i = scene.trace_host(rays[:m], any_hit=any_hit, incoherent=incoherent)
            assert np.array_equal(h.view(np.uint32), hits[:m].view(np.uint32)) and np.array_equal(i, inst[:m]), m


def _render(scene, env, kind, w, h, spp, bounces, nee, rr, per_lane, batch=0):
    pt = nb.Pathtracer(w, h, nb.Globals(bounces=bounces))
    pt.set_sampling(env_nee=nee)
    pt.set_rr_start_bounce(rr)
    pt.enable_trace_counters(per_lane)
    if batch:
        pt.set_batch_paths(batch)
    pt.render(scene, nb.camera_struct(*scenes.camera_matrices(*CAMS[kind], w, h)), env, spp)
    return pt.download(), pt.last_stats()


# waves around the limits: all bounces in one launch (up to 32,768 paths), from bounce 1 on (twice
# that), from later bounces on, and short queues within a larger wave
@pytest.mark.parametrize("kind,w,h,spp,bounces,nee,rr", [
    ("spheres", 1, 1, 1, 8, False, 0), ("spheres", 3, 5, 1, 0, False, 0), ("instanced", 33, 27, 2, 8, True, 0),
    ("instanced", 255, 257, 1, 8, False, 0), ("instanced", 256, 256, 1, 3, True, 3), ("room", 256, 257, 1, 8, False, 0),
    ("instanced", 257, 256, 1, 8, True, 0), ("spheres", 300, 437, 1, 6, False, 0), ("room", 363, 361, 1, 12, False, 0),
    ("instanced", 511, 513, 1, 8, False, 3), ("spheres", 640, 480, 2, 6, True, 0), ("instanced", 801, 603, 3, 8, True, 0),
    ("instanced", 801, 603, 3, 8, False, 0), ("instanced", 181, 181, 1, 8, False, 0), ("spheres", 128, 256, 1, 8, True, 0),
    ("instanced", 127, 259, 1, 8, True, 0), ("room", 129, 255, 1, 8, False, 3)])
def test_render_equals_ray_per_lane(world, kind, w, h, spp, bounces, nee, rr):
    scene, env = world[kind]
    a, sa = _render(scene, env, kind, w, h, spp, bounces, nee, rr, False)
    b, sb = _render(scene, env, kind, w, h, spp, bounces, nee, rr, True)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert sa == sb


def test_several_waves_per_render(world):
    scene, env = world["instanced"]
    a = _render(scene, env, "instanced", 100, 75, 11, 8, False, 0, False, batch=3 * 7500)
    b = _render(scene, env, "instanced", 100, 75, 11, 8, False, 0, True)
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32)) and a[1] == b[1]


@pytest.mark.parametrize("w,h,spread", [(64, 48, 0.01), (256, 256, -1.0), (400, 300, 0.01), (700, 500, np.inf)])
def test_cache_frames_equal_ray_per_lane(world, w, h, spread):
    scene, env = world["instanced"]
    out = []
    for per_lane in (False, True):
        pt = nb.Pathtracer(w, h, nb.Globals(bounces=8))
        cache = nb.RadianceCache(seed=3, spread=spread, train_records=8192, train_steps=2)
        pt.set_cache(cache)
        pt.enable_trace_counters(per_lane)
        for k in range(3):
            pt.invalidate()
            pt.dispatch(scene, nb.camera_struct(*scenes.camera_matrices((0.0, 14.0, 60.0 + k), (0.0, -2.0, 0.0), w, h)),
                        env)
        stats = cache.stats()
        out.append((pt.download(), cache.get_weights(), pt.last_stats(), stats["queries"], stats["records_found"]))
    for x, y in zip(*out):
        assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=True)


def test_host_and_device_queries_alternate(world):
    """Host queries of changing sizes (through the scene's own buffer up to 65,536 rays, through device
    buffers beyond) and device queries on the same scene give the same hits; nb_scene_status follows the
    last query; calls from several threads take turns."""
    import threading

    import torch
    scene = world["instanced"][0]
    n = LIMIT + 5
    rays = scenes.incoherent_rays(n, seed=21)
    rays[:, :3] *= np.float32([30.0, 12.0, 30.0])
    dev = torch.from_numpy(rays).cuda()
    hits = torch.empty(n, 4, device="cuda")
    inst = torch.empty(n, dtype=torch.int32, device="cuda")
    scene.trace_device(dev.data_ptr(), n, hits.data_ptr(), inst.data_ptr(), incoherent=True)
    assert scene.status() == 0
    want, want_i = hits.cpu().numpy().view(np.uint32), inst.cpu().numpy().view(np.uint32)
    for m in (1, 700, 30000, 5, n, 1, LIMIT):
        h, i = scene.trace_host(rays[:m], incoherent=True)
        assert np.array_equal(h.view(np.uint32), want[:m]) and np.array_equal(i, want_i[:m])
        h, none = scene.trace_host(rays[:m], with_instances=False)
        assert none is None and np.array_equal(h.view(np.uint32), want[:m]) and scene.status() == 0
    assert scene.trace_host(rays[:0])[0].shape == (0, 4)
    bad = []

    def query(lo):
        for _ in range(20):
            h, _ = scene.trace_host(rays[lo:lo + 900])
            if not np.array_equal(h.view(np.uint32), want[lo:lo + 900]):
                bad.append(lo)

    threads = [threading.Thread(target=query, args=(1000 * k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
