"""3 x 3 convolutions on CTA pairs (csrc/conv_pair.cuh): ragged images, odd numbers of pixel tiles, channel counts that end inside a
block of 64 or a step of 16, output widths of every tile, epilogues; against 64-bit sums."""
import pytest
import torch
import torch.nn.functional as F

from vllm_omni_b200.ops import _native as nv, conv as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 64, 80), (3, 47, 61), (2, 16, 200), (5, 33, 41), (40, 7, 9), (20, 8, 130), (9, 3, 401)])
@pytest.mark.parametrize("cin,cout", [(16, 384), (96, 96), (96, 3), (72, 200), (192, 192), (128, 256), (8, 40)])
@pytest.mark.parametrize("epilogue", [None, "silu", "residual"])
def test_against_64_bits(n, h, w, cin, cout, epilogue):
    if epilogue and (cin, cout) not in ((96, 96), (8, 40), (96, 3), (72, 200), (128, 256)):
        pytest.skip("epilogues at five widths")
    g = torch.Generator(device="cuda").manual_seed(n * h + w + cin)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    wide = rnd(n, h, w, cin + 8)                                       # channels past cin are not part of the input
    wt, b = rnd(cout, cin, 3, 3) * (9 * cin) ** -0.5, rnd(cout)
    pw, pb = C.pack_conv_weight(wt, b)
    res = rnd(n, h, w, pw.shape[0]) if epilogue == "residual" else None
    out = C.conv2d_nhwc(wide, pw, pb, 3, cin, act="silu" if epilogue == "silu" else None, residual=res)
    x64, w64 = wide[..., :cin].double().permute(0, 3, 1, 2), wt.double()
    ref = F.conv2d(x64, w64, b.double(), padding=1)
    mass = F.conv2d(x64.abs(), w64.abs(), padding=1)
    err = 0.0
    if epilogue == "silu":
        err, ref = ref.abs() * 2.0 ** -11, F.silu(ref)                 # tanh.approx
    if res is not None:
        ref = ref + res[..., :cout].double().permute(0, 3, 1, 2)
    # result rounded to bf16; fp32 sums of at most 9 * cin / 16 MMA steps
    bound = 1.2 * (ref.abs() * 2.0 ** -8 + mass * (9 * cin / 16 + 1) * 2.0 ** -23) + err + 1e-6
    got = out[..., :cout].double().permute(0, 3, 1, 2)
    assert torch.isfinite(out).all() and ((got - ref).abs() <= bound).all()
    nv.check_status()


@pytest.mark.parametrize("channels", [8, 32, 40, 64, 96, 128, 136, 192, 256, 264, 384, 512, 520, 1024])
@pytest.mark.parametrize("pixels", [1, 77, 2369, 4099, 4736, 9472, 9473, 18944, 18945, 37889])     # lanes per pixel change at 256 * SMs / lanes
def test_rmsnorm_silu(channels, pixels):
    g = torch.Generator(device="cuda").manual_seed(channels + pixels)
    x, gamma = torch.randn(pixels, channels, generator=g, device="cuda").bfloat16(), torch.randn(channels, generator=g, device="cuda").bfloat16()
    z = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True)) * gamma.double()
    for silu in (False, True):
        y, ref = C.rmsnorm_silu_nhwc(x, gamma, silu=silu), F.silu(z) if silu else z
        # one rounding to bf16 of fp32 arithmetic; tanh.approx in silu
        assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + z.abs() * 2.0 ** -11 * silu + 1e-5).all()


# both places where the epilogue makes the norm (a thread has all channels of a pixel; two threads share them), widths that leave columns of a tile empty, a
# width whose channels span tiles (norm of its own); one image that is doubled in place, several and flat ones that are not
@pytest.mark.parametrize("cin,cout", [(96, 96), (16, 24), (192, 96), (40, 192), (192, 136), (64, 384), (72, 3)])
@pytest.mark.parametrize("n,h,w,up", [(1, 64, 80, False), (1, 33, 41, True), (1, 16, 8, True), (2, 33, 41, False), (2, 20, 24, True), (1, 5, 400, True)])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_and_doubling_in_the_launch(n, h, w, up, cin, cout, residual):
    g = torch.Generator(device="cuda").manual_seed(n * h + w + cin)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, wt = rnd(n, h, w, (cin + 7) // 8 * 8), rnd(cout, cin, 3, 3) * (9 * cin) ** -0.5
    pw, pb = C.pack_conv_weight(wt, rnd(cout))
    gamma = rnd(pw.shape[0])
    s = 2 if up else 1
    res = rnd(n, s * h, s * w, pw.shape[0]) if residual else None
    want = C.conv2d_nhwc(x.repeat_interleave(s, 1).repeat_interleave(s, 2), pw, pb, 3, cin, residual=res)       # the same products in the same order
    for silu in (True, False):
        norm = C.rmsnorm_silu_nhwc(want, gamma, silu=silu).double()
        for keep in (True, False):
            y, z = C.conv3x3_norm_nhwc(x, pw, pb, cin, residual=res, up=up, gamma=gamma, silu=silu, keep=keep)
            nv.check_status()
            assert torch.equal(y, want) if keep else y is None or torch.equal(y, want)
            # sums of squares in another order may round the other way: one unit in the last place of bf16
            assert ((z.double() - norm).abs() <= norm.abs() * 2.0 ** -7 + 1e-6).all()
    y, z = C.conv3x3_norm_nhwc(x, pw, pb, cin, residual=res, up=up)
    assert z is None and torch.equal(y, want)
    assert torch.equal(want[..., cout:], torch.zeros_like(want[..., cout:]) if res is None else res[..., cout:])
