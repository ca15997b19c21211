"""A mixed batch (several scenes, sizes and trace depths, one wave and many) without statistics, as the serving
loop renders it - one launch traces a bounce's shadow rays with the next bounce's closest-hit rays - against the same
requests alone and against the batch with statistics (a launch per stage): bit-identical images, with opaque and
with transparent shadows."""
import numpy as np
import pytest

from test_gpu_batch import frame_for, render_alone, requests, scene_set

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opaque", [True, False])
@pytest.mark.parametrize("max_paths", [1 << 22, 3000])
def test_batch_without_statistics_matches_requests_alone(agb, max_paths, opaque):
    from aurora_gb300 import api
    scs = scene_set()
    if not opaque:
        for s in scs:
            s.materials["opacity"][::3] = (0.5, 0.3, 0.8)  # surfaces that shadow rays pass, in every scene
    rs = []
    try:
        for s in scs:
            r = api.Renderer()
            r.upload(s)
            rs.append(r)
        reqs = requests(scs)
        views, items, want = [], [], []
        for k, w, h, spp, seed, jit, aovs in reqs:
            f = frame_for(scs[k], w, h, jit, aovs)
            f["is_force_opaque_shadows_enabled"] = 1 if opaque else 0
            want.append(render_alone(rs[k], f, w, h, spp, seed)[0])
            v = api.View(rs[k])
            v.set_frame(f)
            views.append(v)
            items.append(dict(view=v, width=w, height=h, spp=spp, seed_offset=seed))
        assert len({int(np.asarray(scs[k].frame)["trace_depth"]) for k, *_ in reqs}) > 2
        with api.Batch(max_paths=max_paths) as b:
            for stats in (False, True):
                b.render(items, stats=stats)
                for (k, w, h, *_), v, img in zip(reqs, views, want):
                    np.testing.assert_array_equal(v.read(_abi.ACCUM_RUNNING_MEAN, w, h), img[0])
                    np.testing.assert_array_equal(v.read(_abi.ACCUM_KAHAN, w, h), img[1])
        for v in views:
            v.close()
    finally:
        for r in rs:
            r.close()
