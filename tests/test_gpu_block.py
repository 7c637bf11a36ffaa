"""block_kernel (csrc/render.cu): whole small renders, and the ends of larger
ones, inside thread blocks. It runs the wavefront's own steps, so its images
are bit for bit those of the wavefront alone, which rmn_render_profile_get
renders with."""
import numpy as np
import pytest

from raym0nade_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _case(name, w, h, spp, depth):
    if name == "terrain":
        s = scenes.heightfield(65, seed=4)
        s.env = scenes.sky_env(128, 64)
        cam = scenes.heightfield_camera(w, h, spp)
    elif name == "textured":
        s, cam = scenes.textured_room(), scenes.textured_camera(w, h, spp)
    else:
        s = scenes.cornell_glass() if name == "glass" else scenes.cornell()
        cam = scenes.cornell_camera(w, h, spp)
    cam.max_depth = depth
    return s, cam


# one unit, one worker, fewer workers than a block, an odd count over several
# blocks, about as many units as workers the device holds (155,648) and as the
# kernel takes from the start (400,000), and renders whose wavefront runs first
@pytest.mark.parametrize("name,w,h,spp,depth", [
    ("cornell", 1, 1, 1, 1), ("cornell", 1, 1, 2, 16), ("cornell", 33, 17, 5, 3), ("cornell", 97, 61, 9, 16),
    ("cornell", 240, 216, 9, 8), ("cornell", 241, 217, 9, 8), ("cornell", 365, 365, 9, 8),
    ("cornell", 366, 366, 9, 8), ("cornell", 200, 150, 65, 16),
    ("glass", 5, 3, 1, 16), ("glass", 61, 47, 3, 16), ("glass", 90, 80, 16, 12),
    ("textured", 7, 5, 4, 16), ("textured", 120, 90, 8, 16), ("textured", 200, 160, 32, 8),
    ("terrain", 31, 29, 7, 16), ("terrain", 160, 90, 16, 16), ("terrain", 320, 200, 40, 16),
])
def test_block_kernel_equals_the_wavefront(name, w, h, spp, depth):
    scene, cam = _case(name, w, h, spp, depth)
    m = api.Model(scene)
    args = api.RenderArgs.from_camera(cam, seed=17)
    got = api.render(m, args)
    want, _ = api.render_profile(m, args)
    for k in ("radiance_Dd", "radiance_Ds", "radiance_Id", "radiance_Is", "Gbuffer", "dropped"):
        a, b = getattr(got, k).cpu().numpy(), getattr(want, k).cpu().numpy()
        assert np.array_equal(a.view(np.int32), b.view(np.int32)), k
