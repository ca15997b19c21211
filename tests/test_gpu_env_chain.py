"""The reference-layout environment table's two sequential parts (the FP32 sum in index order and the
sweep that pairs below-average with above-average texels) at the sizes and values where their
block-wise evaluation can go wrong: bit-identical to the oracle's sequential loops."""
import numpy as np
import pytest

from test_gpu_env import env_scene

pytestmark = pytest.mark.gpu


def image(kind, h, w, seed):
    rng = np.random.default_rng(seed)
    if kind == "ties":      # addends that are half an ulp of the running sum again and again
        return rng.integers(0, 4, (h, w, 3)).astype(np.float32) * np.float32(0.5)
    if kind == "constant":  # every texel at or next to the average
        return np.full((h, w, 3), 0.75, np.float32)
    if kind == "black_top":  # a run of zeros before the first texel that is not one
        img = rng.uniform(0, 3, (h, w, 3)).astype(np.float32)
        img[: h // 2 + 1] = 0.0
        return img
    if kind == "one_sun":   # one large that takes every small
        img = rng.uniform(0, 1e-3, (h, w, 3)).astype(np.float32)
        img[h // 3, w // 2] = 5e6
        return img
    if kind == "tiny":      # sums that start subnormal and climb through the binades
        return np.exp(rng.uniform(-100, -60, (h, w, 3))).astype(np.float32)
    return np.exp(rng.normal(0, 2, (h, w, 3))).astype(np.float32)


CASES = [("lognormal", 64, 32), ("lognormal", 64, 33), ("lognormal", 91, 181), ("lognormal", 300, 700),
         ("lognormal", 1, 2), ("lognormal", 1, 9), ("lognormal", 5, 1639), ("ties", 90, 180), ("ties", 64, 256),
         ("constant", 64, 128), ("black_top", 130, 257), ("one_sun", 100, 201), ("tiny", 64, 128)]


@pytest.mark.parametrize("kind,h,w", CASES)
def test_sequential_table_parts_match_oracle(agb, oracle, kind, h, w):
    from aurora_gb300 import api
    img = image(kind, h, w, h * 1000 + w)
    with api.Renderer() as r:
        r.upload(env_scene(img))
        table, integral = r.environment_alias()
    ref, ref_integral = oracle.alias_build(img)
    assert np.float32(integral) == np.float32(ref_integral)
    for field in ("alias", "prob", "pdf"):
        np.testing.assert_array_equal(table[field], ref[field], err_msg=field)
