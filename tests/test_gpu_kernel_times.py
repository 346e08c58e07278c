"""nb_pathtracer_kernel_times counts the launches that a render makes: a small wave of one sample per pixel
is one traversal launch, of several samples that and an accumulation; a larger one has launches of all kinds."""
import pytest

import nbounce_gb300 as nb
from nbounce_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,counts", [(64, 48, 1, (0, 1, 0, 0)), (64, 48, 4, (0, 1, 0, 1)), (300, 300, 1, (1, None, 5, 1))])
def test_launch_counts(w, h, spp, counts):
    d = scenes.spheres_scene(width=w, height=h)
    pt = nb.Pathtracer(w, h, nb.Globals(bounces=4))
    pt.enable_timing(True)
    pt.render(nb.SceneBuffers.from_desc(d), nb.camera_struct(d.world_to_clip, d.clip_to_world), nb.EnvMap(d.env_color), spp)
    t = pt.kernel_times()
    got = tuple(t[k + "_launches"] for k in ("raygen", "trace", "shade", "accumulate"))
    assert all(c is None or c == g for c, g in zip(counts, got)), got
