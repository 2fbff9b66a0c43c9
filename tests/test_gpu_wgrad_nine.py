"""The weight gradient's forms: all nine taps of a tile in one CTA, which layers of 128 and
more channels take, and those of one kx with 64 or 32 output channels: values against
torch, and the bounded waits of the first."""
import pytest

pytestmark = pytest.mark.gpu


def _nine_taps(cin, cout, B, H, W):
    """The dispatch's rule: unless CTAs of one kx are all resident, two to an SM."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = -(-cin // 64) * -(-cout // 64)
    cols = 9 * -(-cout // 128) * (-(-cin // 128) if cin > 64 else 1)
    split = max(1, min(B * (H // 8) * (W // 16), (2 * sms + cols - 1) // cols))
    return 3 * tiles * split > 2 * sms


def _data(cin, cout, B, H, W):
    import torch
    g = torch.Generator(device="cuda").manual_seed(cin + 7 * cout)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).bfloat16()
    dy = torch.randn((B, H, W, cout), device="cuda", generator=g).bfloat16()
    return x, dy


# 128 x 128: several blocks per CTA; 64 x 64 images: one to four; partial tiles of output
# (96, 80, 112) and input channels (144, 80); 8 x 16 images: one block per CTA
@pytest.mark.parametrize("cin,cout,B,H,W", [
    (128, 128, 2, 128, 128), (128, 128, 4, 64, 64), (128, 256, 1, 64, 64), (256, 256, 2, 64, 48),
    (384, 128, 2, 64, 64), (256, 96, 2, 64, 64), (192, 80, 1, 72, 80), (144, 112, 2, 64, 64),
    (80, 144, 3, 64, 48), (256, 384, 9, 8, 16)])
def test_nine_tap_gradient_matches_torch(cin, cout, B, H, W):
    """Within 1e-3 of the range of a float32 gradient, the bound of the other shapes; added
    to what dw holds."""
    import torch
    from ctas_b200 import learned
    assert _nine_taps(cin, cout, B, H, W)
    x, dy = _data(cin, cout, B, H, W)
    dw = torch.full((cout, 9, cin), 2.0, device="cuda")
    learned.conv3x3_wgrad(x, dy, dw)
    ref = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (cout, cin, 3, 3),
                                      dy.double().permute(0, 3, 1, 2), padding=1)
    ref = ref.permute(0, 2, 3, 1).reshape(cout, 9, cin)
    torch.cuda.synchronize()
    assert float((dw - 2.0 - ref).abs().max()) <= 1e-3 * float(ref.abs().max())


# one kx: 32 output channels a CTA (few blocks; 48, 80 and 112 leave partial tiles, 16 is
# below one), 64 where there are more blocks or CTAs
@pytest.mark.parametrize("cin,cout,B,H,W", [
    (16, 16, 1, 8, 16), (32, 48, 1, 16, 32), (64, 80, 1, 16, 32), (128, 112, 1, 8, 32),
    (48, 32, 2, 32, 32), (64, 64, 1, 32, 32), (64, 64, 2, 64, 256), (32, 64, 4, 64, 128),
    (192, 64, 1, 32, 32), (64, 128, 2, 64, 64), (80, 48, 1, 64, 128), (256, 256, 1, 8, 16)])
def test_one_kx_gradient_matches_torch(cin, cout, B, H, W):
    import torch
    from ctas_b200 import learned
    assert not _nine_taps(cin, cout, B, H, W)
    x, dy = _data(cin, cout, B, H, W)
    dw = torch.full((cout, 9, cin), -1.0, device="cuda")
    learned.conv3x3_wgrad(x, dy, dw)
    ref = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (cout, cin, 3, 3),
                                      dy.double().permute(0, 3, 1, 2), padding=1)
    ref = ref.permute(0, 2, 3, 1).reshape(cout, 9, cin)
    torch.cuda.synchronize()
    assert float((dw + 1.0 - ref).abs().max()) <= 1e-3 * float(ref.abs().max())


def test_channel_slices():
    """Both operands as channel slices of wider buffers."""
    import torch
    from ctas_b200 import learned
    cin, cout, B, H, W = 128, 128, 2, 64, 64
    assert _nine_taps(cin, cout, B, H, W)
    x, dy = _data(192, 256, B, H, W)
    dw = torch.zeros((cout, 9, cin), device="cuda")
    learned.conv3x3_wgrad(x, dy, dw, cin=cin, x_co=64, cout=cout, dy_co=128)
    ref = torch.nn.grad.conv2d_weight(x[..., 64:].double().permute(0, 3, 1, 2), (cout, cin, 3, 3),
                                      dy[..., 128:].double().permute(0, 3, 1, 2), padding=1)
    ref = ref.permute(0, 2, 3, 1).reshape(cout, 9, cin)
    torch.cuda.synchronize()
    assert float((dw - ref).abs().max()) <= 1e-3 * float(ref.abs().max())


def test_waits_run_out_and_context_survives():
    """The first copies left out: the waits end, the next convolution reports it, and the
    kernel then gives the values of before."""
    import torch
    from ctas_b200 import _lib, ct, learned
    cin, cout, B, H, W = 128, 128, 2, 64, 64
    assert _nine_taps(cin, cout, B, H, W)
    x, dy = _data(cin, cout, B, H, W)

    def run():
        dw = torch.zeros((cout, 9, cin), device="cuda")
        learned.conv3x3_wgrad(x, dy, dw)
        torch.cuda.synchronize()
        return dw

    before, L = run(), _lib.load()
    _lib.check(L.ctas_nn_test_timeout(1))
    try:
        run()
    finally:
        _lib.check(L.ctas_nn_test_timeout(0))
    w = torch.zeros((128, 9, 128), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ct.CtasError) as e:
        learned.conv3x3(x, w, None, relu=False)
    assert e.value.code == _lib.E_TIMEOUT
    torch.cuda.synchronize()
    after = run()
    assert torch.allclose(before, after, rtol=1e-5, atol=1e-5 * float(before.abs().max()))
