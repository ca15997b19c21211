"""The optimiser step, which updates the parameters and packs them both ways in one pass: two Adam steps against
FP64 from the device's own gradients, and the packed weights against those of a denoiser that was given
the same parameters (its answer bit for bit; its gradients, whose sums have no fixed order, to 1e-2 of
their norm, where a misplaced weight changes them by their own size).  A step's FP32 rounding of a parameter: half
an ulp of it, and of the update (at most 1.5 lr here) about ten roundings: 2^-23 |p| + lr 2^-19 for two steps."""
import ctypes

import numpy as np
import pytest

from test_gpu_unet import denoiser, param_count, random_features

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,lr", [(1, 16, 16, 1e-3), (3, 32, 48, 2e-3)])
def test_step_updates_and_packs(agb, B, H, W, lr):
    import torch
    from aurora_gb300 import _abi
    rng = np.random.default_rng(B + H)
    x = torch.from_numpy(random_features(rng, B, H, W).view(np.int16)).cuda()
    t = torch.from_numpy(rng.uniform(0, 2, (B, H, W, 4)).astype(np.float32)).cuda()
    n, loss = param_count(agb), ctypes.c_float()
    dn, other = denoiser(agb), denoiser(agb, 4)

    def read(h, what):
        a = np.zeros(n, np.float32)
        _abi.check(what(h, a.ctypes.data, n))
        return a

    def answer(h):
        out = torch.zeros((B, H, W, 4), device="cuda")
        _abi.check(agb.agb_denoiser_forward(h, x.data_ptr(), B, H, W, out.data_ptr()))
        return out.cpu().numpy()

    def gradients(h):
        _abi.check(agb.agb_denoiser_train_step(h, x.data_ptr(), t.data_ptr(), B, H, W, 0.0, 0, ctypes.byref(loss)))
        return read(h, agb.agb_denoiser_grads)

    try:
        p = read(dn, agb.agb_denoiser_params).astype(np.float64)
        m, v = np.zeros(n), np.zeros(n)
        b1, b2, one = np.float32(0.9), np.float32(0.999), np.float32(1)
        for step in (1, 2):
            _abi.check(agb.agb_denoiser_train_step(dn, x.data_ptr(), t.data_ptr(), B, H, W, lr, 1, ctypes.byref(loss)))
            g = read(dn, agb.agb_denoiser_grads).astype(np.float64)
            m = float(b1) * m + float(one - b1) * g
            v = float(b2) * v + float(one - b2) * g * g
            c1, c2 = (float(one - np.float32(float(b) ** step)) for b in (b1, b2))
            p -= float(np.float32(lr)) * (m / c1) / (np.sqrt(v / c2) + float(np.float32(1e-8)))
        got = read(dn, agb.agb_denoiser_params)
        assert (np.abs(got - p) <= 2.0 ** -23 * np.abs(p) + lr * 2.0 ** -19).all()
        _abi.check(agb.agb_denoiser_set_params(other, got.ctypes.data, n))
        assert np.array_equal(answer(dn), answer(other))
        ga, gb = gradients(dn), gradients(other)
        assert np.linalg.norm(ga - gb) < 1e-2 * np.linalg.norm(gb)
    finally:
        agb.agb_denoiser_destroy(dn)
        agb.agb_denoiser_destroy(other)
