"""The weight gradient of narrow images, whose units take two or four rows: widths on both sides of one, two,
three and four K steps, heights that leave part of a unit, two sources, an upsampled one (a row a unit), and
a last unit of fewer steps in a wide row; against FP64.  Tolerance as for the other shapes: 1e-5 of the sum
of |x dy| (FP32 sums of exact BF16 products)."""
import pytest

pytestmark = pytest.mark.gpu

# batch, height, width, channels of the two sources, output channels, first source upsampled
CASES = [(1, 1, 2, 16, 0, 16, 0), (2, 3, 4, 32, 0, 32, 0), (1, 5, 30, 64, 0, 64, 0), (3, 33, 32, 128, 0, 256, 0),
         (4, 32, 32, 256, 0, 256, 0), (2, 31, 34, 48, 16, 48, 0), (1, 2, 62, 16, 0, 128, 0), (2, 63, 64, 128, 128, 128, 0),
         (1, 21, 66, 32, 0, 64, 0), (1, 9, 96, 128, 0, 96, 0), (2, 7, 98, 64, 64, 64, 0), (1, 17, 160, 64, 0, 64, 0),
         (2, 16, 32, 256, 128, 128, 1), (1, 34, 64, 64, 64, 64, 1), (1, 6, 20, 32, 0, 16, 1)]


@pytest.mark.parametrize("B,H,W,c0,c1,cout,up", CASES)
def test_rows_match_fp64(agb, B, H, W, c0, c1, cout, up):
    import torch
    from aurora_gb300 import _abi
    g = torch.Generator(device="cuda").manual_seed(B * H + W + c0 + cout)
    x0 = torch.randn(B, H >> up, W >> up, c0, generator=g, device="cuda").to(torch.bfloat16)
    x1 = torch.randn(B, H, W, c1, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(B, H, W, cout, generator=g, device="cuda").to(torch.bfloat16)
    cin = c0 + c1
    dw = torch.zeros(9, cin, cout, device="cuda")
    torch.cuda.synchronize()
    _abi.check(agb.agb_conv3x3_wgrad_bf16(x0.data_ptr(), x1.data_ptr() if c1 else None, dy.data_ptr(), dw.data_ptr(),
                                          B, H, W, c0, c1, cout, up, None))
    full = x0.double()
    if up:
        full = full.repeat_interleave(2, 1).repeat_interleave(2, 2)
    xp = torch.nn.functional.pad(torch.cat([full, x1.double()], -1), (0, 0, 1, 1, 1, 1))
    d = dy.double().reshape(-1, cout)
    for t in range(9):
        a = xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, cin)
        want, scale = a.T @ d, a.abs().T @ d.abs() + 1e-30
        err = ((dw[t].double() - want).abs() / scale).max().item()
        assert err < 1e-5, (t, err)
