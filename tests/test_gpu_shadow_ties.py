"""Transparent shadows where an opaque and a half-transparent surface lie in the same place (a decal instance
on its carrier): the any-hit shader of HitShaderEntryPoints.slang:490-552 takes every surface a shadow ray crosses,
in any order, so the opaque one blocks the ray whichever of them has the lower instance index, is met first, or
has a further transparent surface in front of it.  The image is the one with the opaque surface alone."""
import numpy as np
import pytest

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu


def scene(kinds, depth):
    """A lit ground quad under occluders that the camera does not see: O opaque, T half-transparent in the same
    place, N a smaller half-transparent one nearer to the ground, whose shadow lies within theirs."""
    from aurora_gb300 import scenes
    s = scenes.SceneDesc("ties")
    ground, cover = s.add_mesh(*scenes.quad(5.0)), s.add_mesh(*scenes.quad(1.0))
    # Black occluders: no light but the ground's own reaches the image.
    s.materials = scenes.materials(3, base=np.float32([0.8, 0, 0]), specular=np.float32([1, 0, 0]))
    s.materials["opacity"][2] = (0.5, 0.3, 0.8)
    s.instances.append(dict(mesh=ground, material=0, xform=scenes.translation(0, 0, 0), layers=[]))
    for k in kinds:
        xform = scenes.translation(0, 1.5 if k == "N" else 2.0, 0)
        xform[[0, 5, 10]] = 0.9 if k == "N" else 1.0
        s.instances.append(dict(mesh=cover, material=1 if k == "O" else 2, xform=xform, layers=[]))
    s.env = scenes.environment(*[(0, 0, 0)] * 4)
    s.width, s.height, s.spp = 64, 40, 2
    view = scenes.look_at((0, 1.2, 6), (0, 0, 0))
    s.frame = scenes.frame_data(view, scenes.perspective(20, 1.6), trace_depth=depth, force_opaque_shadows=False,
                                lights=[((0, -1.0, 0), (1, 1, 1), 2.0, 0.02)], scene_bounds=s.bounds())
    return s


def render(s, builder):
    from aurora_gb300 import api
    with api.Renderer() as r:
        _abi.check(r._lib.agb_set_bvh_builder(r.ctx, builder))
        r.upload(s)
        r.render(0, s.spp)
        return r.read(_abi.ACCUM_RUNNING_MEAN)


@pytest.mark.parametrize("kinds", ["OT", "TO", "OTN", "TON", "NTO", "TNO", "TOT", "TTO"])
@pytest.mark.parametrize("builder", [_abi.BVH_HOST, _abi.BVH_GPU])
@pytest.mark.parametrize("depth", [1, 3])
def test_coincident_blocker_blocks(agb, oracle, kinds, builder, depth):
    alone = scene("O", depth)
    want = oracle.OracleScene(alone).render(0, alone.spp)["mean"]
    dark = np.mean(np.all(want[..., :3] == 0, axis=2))
    assert 0.02 < dark < 0.9
    got = render(scene(kinds, depth), builder)
    np.testing.assert_array_equal(got[..., :3], render(alone, builder)[..., :3])
    assert oracle.rel_mse(got, want) < 1e-6
