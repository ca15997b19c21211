"""How long the weight gradient's sums are in narrow images.  The tensor core's FP32 accumulation drops what lies
below the accumulator's last place, so with products of one sign the mean signed error grows with the number of rows
that are summed in place before the partial sum goes to dW (which rounds to nearest).  An upsampled source is
summed by single rows; the same source handed over at full resolution is the same sum, and in images of no more
rows than the items of two per SM its items are single rows as well.  So its mean error must not be larger:
both runs sum the same values in the same parts, and only the order in which the parts reach dW differs, whose
rounding averages out over the 9 cin cout outputs.  Allowed for that: a quarter, and a twentieth of the
relative spacing 2^-24 (the mean of 36,864 roundings of about two spacings each is below a fiftieth)."""
import pytest

pytestmark = pytest.mark.gpu

# height, width (of the gradient), channels, output channels: one accumulator set and two
CASES = [(32, 32, 64, 64), (24, 32, 64, 64), (16, 16, 64, 64), (32, 64, 64, 64), (48, 32, 64, 48), (32, 32, 64, 128)]


@pytest.mark.parametrize("H,W,cin,cout", CASES)
def test_sums_no_longer_than_single_rows(agb, H, W, cin, cout):
    import torch
    from aurora_gb300 import _abi
    up_err, full_err = [], []
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(1, H // 2, W // 2, cin, generator=g, device="cuda").exp().to(torch.bfloat16)
        dy = torch.randn(1, H, W, cout, generator=g, device="cuda").exp().to(torch.bfloat16)
        full = x.repeat_interleave(2, 1).repeat_interleave(2, 2).contiguous()
        xp = torch.nn.functional.pad(full.double(), (0, 0, 1, 1, 1, 1))
        d = dy.double().reshape(-1, cout)
        want = torch.stack([xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, cin).T @ d for t in range(9)])
        for src, up, out in ((x, 1, up_err), (full, 0, full_err)):
            dw = torch.zeros(9, cin, cout, device="cuda")
            torch.cuda.synchronize()
            _abi.check(agb.agb_conv3x3_wgrad_bf16(src.data_ptr(), None, dy.data_ptr(), dw.data_ptr(), 1, H, W, cin, 0,
                                                  cout, up, None))
            out.append(((dw.double() - want) / want).mean().item())
    single, mean = sum(up_err) / len(up_err), sum(full_err) / len(full_err)
    print(f"{H}x{W} {cin}->{cout}: mean signed error {mean / 2**-24:.3f} of 2^-24, by single rows {single / 2**-24:.3f}")
    assert abs(mean) <= 1.25 * abs(single) + 0.05 * 2 ** -24


# batch, height, width, input and output channels: halves that meet inside a unit, at a unit whose further rows lie below
# the image, in items of one unit (of one to four rows) and of several
MEETING = [(1, 3, 2, 64, 64), (1, 7, 30, 64, 48), (1, 33, 32, 64, 64), (4, 32, 32, 64, 64), (4, 31, 20, 32, 64),
           (4, 64, 64, 64, 64), (9, 37, 64, 16, 32), (33, 37, 64, 64, 64)]


@pytest.mark.parametrize("B,H,W,cin,cout", MEETING)
def test_halves_match_fp64(agb, B, H, W, cin, cout):
    """Tolerance as for the other shapes: 1e-5 of the sum of |x dy| (FP32 sums of exact BF16 products)."""
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
