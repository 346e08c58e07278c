"""No bounce's queue goes to the 8-lane kernel without a look at its length: a wave above the limit, which is
lower for few bounces and with NEE, has the per-bounce traversal and shading launches of all of its bounces,
so that an enclosed scene, whose paths survive, is not traced at 2.5 times the instructions per ray."""
import pytest

import nbounce_gb300 as nb
from nbounce_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nee", [False, True])
@pytest.mark.parametrize("w,h,bounces", [(182, 181, 8), (256, 256, 8), (300, 437, 12), (640, 480, 3), (160, 160, 2),
                                          (100, 100, 0)])
def test_every_bounce_has_its_kernels(w, h, bounces, nee):
    d = scenes.room_scene(width=w, height=h)
    pt = nb.Pathtracer(w, h, nb.Globals(bounces=bounces))
    pt.set_sampling(env_nee=nee)
    pt.enable_timing(True)
    pt.render(nb.SceneBuffers.from_desc(d), nb.camera_struct(d.world_to_clip, d.clip_to_world),
              nb.EnvMap((0.5, 0.6, 0.8)), 1)
    t = pt.kernel_times()
    assert t["shade_launches"] == bounces + 1
    # per bounce, NEE's last shadow rays, and at least one check
    assert t["trace_launches"] >= bounces + 1 + nee + min(bounces, 1)
