"""Instance boxes of a lopsided mesh: the TLAS box of an instance is the union of the transformed boxes five levels
down its mesh's tree, also where a small outlying part of a large mesh (a subtree that the builder numbers behind
all the large nodes) hangs right under the root."""
import numpy as np
import pytest

from test_gpu_bvh import read_bvh, read_tlas

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu


def cover_boxes(nodes, root, levels=5):
    refs = nodes[:, 12:14].view(np.int32)
    out, level = [], [root]
    for depth in range(levels):
        nxt = []
        for k in level:
            n = nodes[k]
            boxes = ((n[[0, 2, 8]], n[[1, 3, 9]]), (n[[4, 6, 10]], n[[5, 7, 11]]))
            for side in (0, 1):
                if refs[k][side] >= 0 and depth + 1 < levels:
                    nxt.append(int(refs[k][side]))
                else:
                    out.append(boxes[side])
        level = nxt
    return out


# Triangles of the bulk: one subtree, one large node, and (every subtree holds at most 512) over 4,096 large nodes.
@pytest.mark.parametrize("bulk", [300, 3000, 2_110_000])
def test_instance_box_is_the_cover_of_five_levels(agb, bulk):
    from aurora_gb300 import api, scenes
    rng = np.random.default_rng(bulk)
    c = rng.uniform(0, 1, (bulk, 1, 3)).astype(np.float32)
    d = np.linspace(0, 40, 400, dtype=np.float32)[:, None, None] * np.float32([1, 1, 0]) + np.float32([100, 0, 0])
    c = np.concatenate([c, d])
    pos = (c + rng.uniform(0, 0.01, (len(c), 3, 3)).astype(np.float32)).reshape(-1, 3)
    s = scenes.SceneDesc("lopsided")
    mesh = s.add_mesh(pos, None, None, np.arange(len(pos), dtype=np.uint32))
    h = np.float32(np.sqrt(0.5))
    turned = np.float32([h, -h, 0, 0, h, h, 0, 0, 0, 0, 1, 0])
    s.materials = scenes.materials(1)
    for xform in (turned, scenes.translation(1000, 0, 0)):
        s.instances.append(dict(mesh=mesh, material=0, xform=xform, layers=[]))
    s.width = s.height = 4
    s.frame = scenes.frame_data(np.eye(4), scenes.perspective(45, 1))
    with api.Renderer() as r:
        _abi.check(r._lib.agb_set_bvh_builder(r.ctx, _abi.BVH_GPU))
        r.upload(s)
        nodes, _, root, _ = read_bvh(r, 0)
        tlas, order, troot, _ = read_tlas(r)
    m = turned.reshape(3, 4).astype(np.float64)
    lo, hi = np.full(3, np.inf), np.full(3, -np.inf)
    for b in cover_boxes(nodes, root):
        for corner in range(8):
            p = np.array([b[corner >> k & 1][k] for k in range(3)], np.float64)
            w = m[:, :3] @ p + m[:, 3]
            lo, hi = np.minimum(lo, w), np.maximum(hi, w)
    n = tlas[troot]
    sides = [int(order[~int(ref) >> 3]) for ref in n[12:14].view(np.int32)]
    k = sides.index(0)
    box = ((n[[0, 2, 8]], n[[1, 3, 9]]), (n[[4, 6, 10]], n[[5, 7, 11]]))[k]
    # FP32 corners (a few parts in 10^7 of 180) and the box's own padding of 1e-5 of the two sides.
    np.testing.assert_allclose(box[0], lo, rtol=0, atol=5e-3)
    np.testing.assert_allclose(box[1], hi, rtol=0, atol=5e-3)
