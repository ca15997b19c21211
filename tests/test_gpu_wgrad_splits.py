"""The weight gradient's split into items and halves: unit counts that leave items of one unit, of an odd
number and of unequal length, one and two items per SM, and every tile width, against FP64.  Tolerance as
for the other shapes: 1e-5 of the sum of |x dy| (FP32 sums of exact BF16 products; dW starts from zero, so no
rounding to a larger value that was there enters)."""
import pytest

pytestmark = pytest.mark.gpu

# batch, height, width, input channels, output channels
CASES = [(1, 1, 2, 16, 16), (1, 50, 128, 64, 64), (1, 51, 128, 64, 64), (1, 103, 126, 64, 48), (3, 101, 130, 64, 64),
         (2, 153, 100, 32, 32), (1, 305, 66, 16, 64), (2, 211, 258, 48, 32), (1, 97, 140, 128, 96), (2, 120, 260, 64, 128)]


@pytest.mark.parametrize("B,H,W,cin,cout", CASES)
def test_splits_match_fp64(agb, B, H, W, cin, cout):
    import torch
    from aurora_gb300 import _abi
    g = torch.Generator(device="cuda").manual_seed(B * H + W + cin)
    x = torch.randn(B, H, W, cin, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(B, H, W, cout, generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.zeros(9, cin, cout, device="cuda")
    torch.cuda.synchronize()
    _abi.check(agb.agb_conv3x3_wgrad_bf16(x.data_ptr(), None, dy.data_ptr(), dw.data_ptr(), B, H, W, cin, 0, cout, 0,
                                          None))
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    d = dy.double().reshape(-1, cout)
    for t in range(9):
        a = xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, cin)
        want, scale = a.T @ d, a.abs().T @ d.abs() + 1e-30
        err = ((dw[t].double() - want).abs() / scale).max().item()
        assert err < 1e-5, (t, err)
