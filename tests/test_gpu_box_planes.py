"""The box test of a ray per lane at the edges of its margins, against the same rays traced with 8 lanes
per ray (whose box test has another offset and margin, and is held to the oracle elsewhere): the closest
distance is the same bits, and a ray has any hit or none."""
import numpy as np
import pytest

import nbounce_gb300 as nb
from nbounce_gb300 import scenes

pytestmark = pytest.mark.gpu

LIMIT = 65536  # above it no call is traced in groups (below 16,384 all are)


def _edge_rays(desc, scale, seed):
    """8,000 rays: axis-parallel, components around the reciprocal's nudge, exact powers of two, components
    over 16 decades, and origins on box planes (a vertex's coordinate) with a tiny component there."""
    rng = np.random.default_rng(seed)
    n = 8000
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(-1.2, 1.2, (n, 3)) * scale
    d = rng.normal(size=(n, 3))
    rows, which = np.arange(n), rng.integers(0, 3, n)
    small = np.array([0.0, 1e-21, 1e-20, 1.9e-20, 2e-20, 2.1e-20, 1e-19, 2.0 ** -60, 1e-12, 1e-6])
    d[rows, which] = np.where(d[rows, which] < 0, -1.0, 1.0) * small[rng.integers(0, len(small), n)]
    q = n // 4
    d[:q] = np.where(d[:q] < 0, -1.0, 1.0) * 2.0 ** rng.integers(-10, 11, (q, 3))
    d[q:q + n // 8] *= 10.0 ** rng.integers(-8, 9, (n // 8, 3))
    v = desc.vertices["pos"][rng.integers(0, len(desc.vertices), n)]
    on = rows % 3 == 0
    rays[rows[on], which[on]] = v[rows[on], which[on]]
    rays[:, 4:7] = d
    return rays


@pytest.mark.parametrize("scale", [1.0, 1024.0, 2.0 ** 20])
def test_edge_rays_equal_groups(scale):
    desc = scenes.soup_scene(20000, seed=11)
    desc.vertices["pos"] *= np.float32(scale)
    scene = nb.SceneBuffers.from_desc(desc)
    rays = _edge_rays(desc, scale, 7)
    ref = scene.trace_host(rays)[0][:, 0]
    assert (ref < 3e38).sum() > 300
    many = np.tile(rays, (LIMIT // len(rays) + 1, 1))
    for incoherent in (False, True):
        t = scene.trace_host(many, incoherent=incoherent)[0][:, 0].reshape(-1, len(rays))
        assert np.array_equal(t.view(np.uint32), np.broadcast_to(ref, t.shape).copy().view(np.uint32)), incoherent
        hit = scene.trace_host(many, any_hit=True, incoherent=incoherent)[0][:, 0].reshape(-1, len(rays)) < 3e38
        assert np.array_equal(hit, np.broadcast_to(ref < 3e38, hit.shape)), incoherent
