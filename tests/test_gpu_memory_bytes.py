"""agb_context_memory counts the allocations that a context holds: the serving loop charges a pooled view by
it, and a view's image size changes from request to request."""
import numpy as np
import pytest

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu


def test_smaller_image_keeps_what_the_larger_one_allocated(agb):
    """No render buffer is given back when an image gets smaller, so the figure stays; the same image again
    allocates nothing."""
    from aurora_gb300 import api, scenes
    s = scenes.config_tiny(width=32, height=24, spp=1)
    with api.Renderer() as r:
        r.upload(s)
        with api.View(r) as v:
            v.set_frame(s.frame)
            seen = []
            for w, h in ((640, 360), (64, 36), (640, 360)):
                v.render(0, 1, width=w, height=h)
                v.wait()
                seen.append(v.memory_bytes())
    print("bytes", seen)
    assert seen[0] >= 640 * 360 * 72  # the accumulation alone: four float4 and a float2 a pixel
    assert seen[1] == seen[0] and seen[2] == seen[0]


@pytest.mark.parametrize("builder", [_abi.BVH_HOST, _abi.BVH_GPU])
def test_geometry_counted_once(agb, builder):
    """A mesh's arrays (positions, normals, texture coordinates, vertex records, indices, triangles) are in the
    figure once, whichever way they were allocated; its nodes, at most one a triangle, beside them."""
    from aurora_gb300 import api, scenes
    pos, nrm, uv, idx = scenes.icosphere(5, radius=1.0)
    v, t = len(pos), len(idx) // 3
    arrays = v * (12 + 12 + 8 + 32) + len(idx) * 4 + t * 48
    s = scenes.SceneDesc("ico")
    s.add_mesh(pos, nrm, uv, idx)
    with api.Renderer() as r:
        _abi.check(r._lib.agb_set_bvh_builder(r.ctx, builder))
        before = r.memory_bytes()
        r.upload_geometry_only(s)
        grown = r.memory_bytes() - before
    assert arrays <= grown <= arrays + 64 * t + 16384  # and the mesh table, rounding
