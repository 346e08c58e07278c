"""Queries whose answer the visiting order decides: the first hit found by an any-hit query among
overlapping instances, and the closest hit among coincident triangles (a hit replaces another only if it
is strictly closer).  The library visits children near to far by their entry distance, and at the same
distance in the order of their slots; the answers are held to tests/golden/hit_order.npz whatever the
number of rays in a call, which decides how many lanes trace a ray."""
import os

import numpy as np
import pytest

import nbounce_gb300 as nb
from nbounce_gb300 import scenes

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "hit_order.npz")
MANY = 65536  # rays of a call that is traced a ray per lane (up to 16,384 or 24,576 rays: 8 lanes per ray)


def _instance(rng, start, end, scale=1.0, t=(0.0, 0.0, 0.0)):
    """Scale and translation only, by powers of two and dyadic numbers: the same floats on every machine."""
    t = np.asarray(t, np.float64)
    l2w, w2l = np.eye(4), np.eye(4)
    l2w[:3, :3] *= scale
    l2w[:3, 3] = t
    w2l[:3, :3] /= scale
    w2l[:3, 3] = -t / scale
    return dict(l2w=l2w.astype(np.float32), w2l=w2l.astype(np.float32), color=np.ones(4, np.float32),
                roughness=np.float32(0.5), metallic=np.float32(0.0), emissive=np.float32(0.0), index_start=start,
                index_end=end)


def _vertices(pos):
    return scenes.pack_vertices(pos, np.tile([0.0, 1.0, 0.0], (len(pos), 1)), np.tile([1.0, 0.0, 0.0, 1.0], (len(pos), 1)))


def crowd():
    """400 overlapping octahedra."""
    rng = np.random.default_rng(17)
    pos = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]], np.float64)
    faces = np.array([[0, 2, 4], [2, 1, 4], [1, 3, 4], [3, 0, 4], [2, 0, 5], [1, 2, 5], [3, 1, 5], [0, 3, 5]], np.uint32)
    prims = [_instance(rng, 0, faces.size, (0.25, 0.5, 1.0, 2.0)[rng.integers(4)], rng.integers(-64, 65, 3) / 16.0)
             for _ in range(400)]
    return nb.SceneBuffers.from_scene(_vertices(pos), faces.ravel(), prims)


def coincident():
    """Six meshes in place, each with the same 4,000 triangles among others of its own."""
    rng = np.random.default_rng(19)

    def soup(n):
        c = rng.integers(-1000, 1001, (n, 1, 3))
        return ((c + rng.integers(-80, 81, (n, 3, 3))) / 1000.0).reshape(-1, 3)

    shared, pos, idx, prims, n_pos, n_idx = soup(4000), [], [], [], 0, 0
    for k in range(6):
        p = np.concatenate([shared, soup(4000 // (2 + k))])
        tri = rng.permutation(len(p) // 3)
        pos.append(p)
        idx.append((3 * tri[:, None] + np.arange(3)).ravel() + n_pos)
        prims.append(_instance(rng, n_idx, n_idx + len(p)))
        n_pos, n_idx = n_pos + len(p), n_idx + len(p)
    return nb.SceneBuffers.from_scene(_vertices(np.concatenate(pos)), np.concatenate(idx).astype(np.uint32), prims)


def rays(n, seed, extent):
    """(n, 8): origins in the cube of that half extent, directions of any kind."""
    rng = np.random.default_rng(seed)
    out = np.zeros((n, 8), np.float32)
    out[:, :3] = rng.integers(-4096, 4097, (n, 3)) / 4096.0 * extent
    out[:, 4:7] = (rng.integers(-1000, 1001, (n, 3)) + np.array([0.5, 0.25, 0.125])) / 1024.0
    return out


@pytest.fixture(scope="module")
def golden():
    return np.load(GOLDEN)


@pytest.mark.parametrize("incoherent", [False, True])
@pytest.mark.parametrize("make,any_hit", [(crowd, True), (crowd, False), (coincident, False), (coincident, True)])
def test_hits_are_the_recorded_ones(golden, make, any_hit, incoherent):
    scene, key = make(), f"{make.__name__}_{'any' if any_hit else 'closest'}"
    r, want = golden[make.__name__ + "_rays"], golden[key]
    assert len(r) <= 16384
    for n in (len(r), MANY + 1):
        many = np.resize(r, (n, 8))
        hits, inst = scene.trace_host(many, any_hit=any_hit, incoherent=incoherent)
        got = np.column_stack([hits.view(np.uint32), inst])
        assert np.array_equal(got, np.resize(want, (n, 5))), (n, int((got != np.resize(want, (n, 5))).any(1).sum()))
