"""Narrow images that share a convolution's tiles: widths and batch sizes around one, two and more images a
tile and around a last tile that is not full, plain, upsampled with a skip, and pooled.  The sums are those
of the images one by one, bit for bit; against FP64 1e-5 of the sum of |x w|, as for the other shapes."""
import pytest

pytestmark = pytest.mark.gpu

# batch, height, width, first input's channels, second's, output channels, first input upsampled
CASES = [(50, 1, 2, 16, 0, 16, False), (9, 5, 26, 32, 0, 32, False), (4, 32, 32, 128, 0, 256, False),
         (7, 6, 34, 144, 0, 64, False), (4, 64, 64, 64, 0, 128, False), (3, 7, 84, 16, 16, 48, False),
         (3, 9, 124, 64, 0, 64, False), (2, 10, 126, 32, 0, 64, False), (2, 4, 128, 128, 0, 64, False),
         (5, 12, 32, 256, 128, 128, True), (4, 34, 64, 64, 64, 64, True)]


@pytest.mark.parametrize("B,H,W,c0,c1,cout,up", CASES)
def test_images_match_single_ones_and_fp64(agb, B, H, W, c0, c1, cout, up):
    import torch
    import torch.nn.functional as F
    from aurora_gb300 import _abi
    g = torch.Generator(device="cuda").manual_seed(B * H + W + cout)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    x0 = rnd(B, H // 2 if up else H, W // 2 if up else W, c0).to(torch.bfloat16)
    x1 = rnd(B, H, W, c1).to(torch.bfloat16)
    w, bias = (rnd(9, c0 + c1, cout) * 0.1).to(torch.bfloat16).float(), rnd(cout)
    pack = torch.zeros(9 * (c0 + c1) * cout, dtype=torch.int16, device="cuda")
    out, single = torch.zeros(2, B, H, W, cout, device="cuda")
    torch.cuda.synchronize()
    _abi.check(agb.agb_pack_conv_weights(w.data_ptr(), c0 + c1, cout, 0, pack.data_ptr(), None))

    def conv(a, b, o):
        _abi.check(agb.agb_conv3x3_bf16(a.data_ptr(), b.data_ptr() if c1 else None, pack.data_ptr(), bias.data_ptr(),
                                        None, o.data_ptr(), len(o), H, W, c0, c1, cout, int(up), 0, None))

    conv(x0, x1, out)
    for i in range(B):
        conv(x0[i:i + 1], x1[i:i + 1], single[i:i + 1])
    assert torch.equal(out, single)
    if H % 2 == 0:
        low, pool = (torch.zeros(B, H // d, W // d, cout, dtype=torch.bfloat16, device="cuda") for d in (1, 2))
        torch.cuda.synchronize()
        _abi.check(agb.agb_conv3x3_pool_bf16(x0.data_ptr(), x1.data_ptr() if c1 else None, pack.data_ptr(),
                                             bias.data_ptr(), low.data_ptr(), pool.data_ptr(), B, H, W, c0, c1, cout,
                                             int(up), 0, None))
        q = low.float()
        assert torch.equal(low, out.to(torch.bfloat16))
        assert torch.equal(pool, ((q[:, ::2, ::2] + q[:, ::2, 1::2] + q[:, 1::2, ::2] + q[:, 1::2, 1::2]) * 0.25)
                           .to(torch.bfloat16))
    x = x0.double().permute(0, 3, 1, 2)
    if up:
        x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
    x = torch.cat([x, x1.double().permute(0, 3, 1, 2)], 1)
    k = w.double().reshape(3, 3, c0 + c1, cout).permute(3, 2, 0, 1).contiguous()
    want = F.conv2d(x, k, bias.double(), padding=1)
    scale = F.conv2d(x.abs(), k.abs(), bias.double().abs(), padding=1)
    err = ((out.double().permute(0, 3, 1, 2) - want).abs() / scale).max().item()
    assert err < 1e-5, err
