"""The convolution's four-row tiles (64 output channels from 128 input channels on) at heights, widths and
batch sizes around their edges, plain and upsampled with a skip, against FP64: 1e-5 of the sum of |x w|, as for
the other shapes."""
import pytest

pytestmark = pytest.mark.gpu

# batch, height, width, first input's channels, second's, output channels, first input upsampled
CASES = [(1, 1, 2, 128, 0, 64, False), (1, 5, 258, 128, 0, 64, False), (3, 67, 130, 144, 0, 64, False),
         (2, 94, 514, 128, 0, 128, False), (1, 154, 700, 128, 64, 64, True), (4, 62, 256, 96, 32, 192, True)]


@pytest.mark.parametrize("B,H,W,c0,c1,cout,up", CASES)
def test_rows_match_fp64(agb, B, H, W, c0, c1, cout, up):
    import torch
    import torch.nn.functional as F
    from aurora_gb300 import _abi
    g = torch.Generator(device="cuda").manual_seed(B * H + W + cout)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    x0 = rnd(B, H // 2 if up else H, W // 2 if up else W, c0).to(torch.bfloat16)
    x1 = rnd(B, H, W, c1).to(torch.bfloat16) if c1 else None
    w, bias = (rnd(9, c0 + c1, cout) * 0.1).to(torch.bfloat16).float(), rnd(cout)
    pack = torch.zeros(9 * (c0 + c1) * cout, dtype=torch.int16, device="cuda")
    out = torch.zeros(B, H, W, cout, device="cuda")
    torch.cuda.synchronize()
    _abi.check(agb.agb_pack_conv_weights(w.data_ptr(), c0 + c1, cout, 0, pack.data_ptr(), None))
    _abi.check(agb.agb_conv3x3_bf16(x0.data_ptr(), x1.data_ptr() if c1 else None, pack.data_ptr(), bias.data_ptr(),
                                    None, out.data_ptr(), B, H, W, c0, c1, cout, 1 if up else 0, 0, None))
    x = x0.double().permute(0, 3, 1, 2)
    if up:
        x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
    if c1:
        x = torch.cat([x, x1.double().permute(0, 3, 1, 2)], 1)
    k = w.double().reshape(3, 3, c0 + c1, cout).permute(3, 2, 0, 1).contiguous()
    want = F.conv2d(x, k, bias.double(), padding=1)
    scale = F.conv2d(x.abs(), k.abs(), bias.double().abs(), padding=1)
    err = ((out.double().permute(0, 3, 1, 2) - want).abs() / scale).max().item()
    assert err < 1e-5, err
