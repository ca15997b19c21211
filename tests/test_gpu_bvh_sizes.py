"""The GPU builder's two parts (large nodes over many CTAs, subtrees of at most 512 primitives in one CTA
each) at the sizes where they meet: valid trees, as good as the host builder's."""
import numpy as np
import pytest

from test_gpu_bvh import check_and_cost, read_bvh

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu


def mesh(kind, triangles, seed):
    rng = np.random.default_rng(seed)
    if kind == "soup":
        c = rng.uniform(-5, 5, (triangles, 1, 3))
    elif kind == "line":      # centroids on one axis: two axes of no extent
        c = np.zeros((triangles, 1, 3))
        c[:, 0, 1] = np.arange(triangles)
    elif kind == "spread":    # each SAH split peels a few off: the depth budget forces midpoints
        c = np.zeros((triangles, 1, 3))
        c[:, 0, 0] = 1.2 ** rng.uniform(0, 380, triangles)
    else:                     # "point": no extent at all
        c = np.zeros((triangles, 1, 3))
    size = 0.0 if kind == "point" else 0.1
    p = c + rng.normal(0, 1, (1 if kind == "point" else triangles, 3, 3)) * (size if size else 1.0)
    return p.reshape(-1, 3).astype(np.float32)


CASES = [("soup", n) for n in (1, 4, 5, 511, 512, 513, 1025, 2048, 2049, 4097, 20001)] + \
    [("line", 513), ("line", 3000), ("spread", 512), ("spread", 5000), ("point", 513), ("point", 2500)]


@pytest.mark.parametrize("kind,triangles", CASES)
def test_sizes_valid_and_close_to_host(agb, kind, triangles):
    from aurora_gb300 import api, scenes
    pos = mesh(kind, triangles, triangles)
    costs = {}
    for builder in (_abi.BVH_HOST, _abi.BVH_GPU):
        s = scenes.SceneDesc(kind)
        s.add_mesh(pos, None, None, np.arange(3 * triangles, dtype=np.uint32))
        with api.Renderer() as r:
            _abi.check(r._lib.agb_set_bvh_builder(r.ctx, builder))
            r.upload_geometry_only(s)
            nodes, tris, root, depth = read_bvh(r, 0)
        costs[builder] = check_and_cost(nodes, tris, root, depth, triangles)
    assert costs[_abi.BVH_GPU] <= 1.15 * costs[_abi.BVH_HOST] + 1e-6
