"""The instrumented traversal's triangle count against a number known without a traversal: parallel
triangles that each fill half of their box, crossed by rays through the other halves.  Such a ray enters
every box, hits nothing and so tests every triangle once, whatever the tree."""
import numpy as np
import pytest

import nbounce_gb300 as nb
from nbounce_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZE = 48  # pixels of a side


def _scene(n, z0, mirror):
    """n right triangles in planes z0 ... z0 + 0.5, x and y in [-1, 1], right angle at (-1, -1)."""
    z = z0 + 0.5 * np.arange(n) / n
    pos = np.array([[[-1, -1, k], [1, -1, k], [-1, 1, k]] for k in z]).reshape(-1, 3)
    b = scenes._Builder()
    grey = dict(color=np.ones(4, np.float32), roughness=np.float32(0.0), metallic=np.float32(1.0), emissive=np.float32(0.0))
    stack = b.add_mesh(scenes.pack_vertices(pos, np.tile([0.0, 0.0, 1.0], (3 * n, 1)), np.tile([1.0, 0, 0, 1], (3 * n, 1))),
                       np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))
    insts = [scenes._instance(stack, np.eye(4), grey)]
    if mirror:  # a perfect one, facing +y
        insts.append(scenes._instance(b.add_mesh(*scenes.quad_mesh((0.5, -20.0, 0.0), (0, 0, 8), (8, 0, 0))), np.eye(4), grey))
    v, i, meshes = b.finish()
    return nb.SceneBuffers.from_desc(scenes.SceneDesc(v, i, meshes, insts))


def _counters(scene, eye, target, spp):
    pt = nb.Pathtracer(SIZE, SIZE, nb.Globals(bounces=3))
    pt.enable_trace_counters(True)
    w2c, c2w = scenes.camera_matrices(eye, target, SIZE, SIZE, fov_y=np.radians(0.5))
    pt.render(scene, nb.camera_struct(w2c, c2w), nb.EnvMap((0.5, 0.6, 0.8)), spp)
    return pt.trace_counters(3)


@pytest.mark.parametrize("spp", [1, 32])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 61])
def test_camera_rays_test_every_triangle(n, spp):
    """Whole-warp chunks."""
    c = _counters(_scene(n, 0.0, False), (0.5, 0.5, -10.0), (0.5, 0.5, 0.0), spp)
    rays = SIZE * SIZE * spp
    assert c[0]["rays"] == c[0]["instance_entries"] == rays and c[1]["rays"] == 0
    assert c[0]["triangle_tests"] == n * rays
    assert c[0]["leaf_warp_triangles"] <= c[0]["triangle_tests"] <= 32 * c[0]["leaf_warp_triangles"]


@pytest.mark.parametrize("spp", [1, 32])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 61])
def test_reflected_rays_test_every_triangle(n, spp):
    """Lane refill: the rays that leave the mirror; on the way they may test its two triangles too."""
    c = _counters(_scene(n, 20.2, True), (0.5, 10.0, -30.0), (0.5, -20.0, 0.0), spp)
    rays = SIZE * SIZE * spp
    assert c[0]["rays"] == c[1]["rays"] == rays and c[2]["rays"] == 0
    assert c[0]["triangle_tests"] == 2 * rays
    assert n * rays <= c[1]["triangle_tests"] <= (n + 2) * rays
    assert c[1]["leaf_warp_triangles"] <= c[1]["triangle_tests"] <= 32 * c[1]["leaf_warp_triangles"]
