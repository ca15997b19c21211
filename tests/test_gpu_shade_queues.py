"""Shading queues around 128 paths per SM, up to which they are dealt out in groups over all SMs, and far from it:
the image of several samples in one wave (a longer queue) and of a wave per sample, bit for bit, with
distant lights and without."""
import numpy as np
import pytest

from aurora_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [-1, 0, 1, 40])
@pytest.mark.parametrize("name", ["tiny", "layered"])
def test_waves_of_one_sample_equal_one_wave(agb, rows, name):
    import torch
    from aurora_gb300 import api, scenes
    width = torch.cuda.get_device_properties(0).multi_processor_count
    w, h, spp = (width, 128 + rows, 3) if rows < 40 else (7, 1, 40)
    if name == "layered":
        s = scenes.config_layered(width=w, height=h, spp=spp, trace_depth=4, blas=2, instances=12,
                                  tri_range=(300, 900), decal_size=64)
    else:
        s = scenes.config_tiny(width=w, height=h, spp=spp, trace_depth=4)
    out = []
    with api.Renderer() as r:
        r.upload(s)
        for paths in (0, w * h):
            r.render(0, spp, max_paths=paths)
            out.append(r.read(_abi.ACCUM_KAHAN).copy())
    np.testing.assert_array_equal(out[0], out[1])
