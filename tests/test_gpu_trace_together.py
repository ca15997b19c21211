"""The launch that traces a bounce's shadow rays with the next bounce's closest-hit rays, against separate
launches (what timing by kernel family uses): the same image bit for bit, for queues from a few rays to more
than the grid's lanes, one bounce to many, opaque and transparent shadows, and with the ground plane."""
import numpy as np
import pytest

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu

CASES = [  # scene, width, height, samples, trace depth, opaque shadows, ground plane
    ("tiny", 1, 1, 1, 4, True, False), ("tiny", 33, 7, 1, 1, True, False), ("tiny", 160, 120, 3, 2, False, True),
    ("small", 97, 101, 1, 5, True, False), ("small", 131, 75, 1, 5, True, True), ("small", 640, 480, 2, 3, True, False),
    ("layered", 64, 48, 2, 5, False, False), ("layered", 200, 150, 3, 8, False, False)]


@pytest.mark.parametrize("name,w,h,spp,depth,opaque,ground", CASES)
def test_together_equals_apart(agb, name, w, h, spp, depth, opaque, ground):
    from aurora_gb300 import api, scenes
    if name == "layered":
        s = scenes.config_layered(width=w, height=h, spp=spp, trace_depth=depth, blas=2, instances=12,
                                  tri_range=(300, 900), decal_size=64)
    else:
        s = getattr(scenes, "config_" + name)(width=w, height=h, spp=spp, trace_depth=depth)
    s.frame["is_force_opaque_shadows_enabled"] = 1 if opaque else 0
    if ground:
        s.ground_plane = _abi.ground_plane(position=(0.0, -0.01, 0.0))
    out = []
    with api.Renderer() as r:
        r.upload(s)
        for apart in (True, False):
            r.set_profiling(apart)
            st = r.render(0, spp, stats=True)
            out.append((r.read(_abi.ACCUM_KAHAN), st["closest_rays_per_bounce"], st["shadow_rays_per_bounce"]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1:] == out[1][1:]
