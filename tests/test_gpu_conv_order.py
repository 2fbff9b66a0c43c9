"""Summation order of the row-streaming convolution: taps of one output row after
another, in each the columns and in each the channels.  The forms round differently, so
a layer keeps its form: every shape whose weights fit takes this one."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 32), (16, 64), (32, 32), (32, 64), (64, 32), (64, 64),
                                      (96, 32), (128, 32)])
@pytest.mark.parametrize("B,H,W", [(1, 8, 128), (2, 40, 256)])
def test_row_form_serves_layer(cin, cout, B, H, W):
    """2^30 at (ky, kx) = (0, 0), 1 at (0, 1) and -2^30 at (2, 0): 0 where the 1 is added
    to 2^30 in float32, 1 in the tiled form, which adds the taps of kx = 0 first."""
    import torch
    from ctas_b200 import learned
    x = torch.zeros((B, H, W, cin), device="cuda")
    x[..., 0], x[..., cin - 1] = 2.0 ** 15, 1.0
    w = torch.zeros((cout, 9, cin), device="cuda")
    w[:, 0, 0], w[:, 1, cin - 1], w[:, 6, 0] = 2.0 ** 15, 1.0, -2.0 ** 15
    y = learned.conv3x3(x.bfloat16(), w.bfloat16(), None, relu=False)
    torch.cuda.synchronize()
    assert (y[:, 1:-1, 1:-1] == 0).all()
    assert (y[:, 0, 1:] == -2.0 ** 30 + 0).all() and (y[:, -1, 1:] == 2.0 ** 30).all()


@pytest.mark.parametrize("B,H,W,relu,masked", [(1, 8, 128, True, False), (2, 24, 256, False, True),
                                               (1, 40, 384, True, False)])
def test_128_to_32_matches_torch(B, H, W, relu, masked):
    """The row form with one staging buffer per warp: within 1e-2 of the output range of
    a float32 convolution, the bound of the other shapes."""
    import torch
    import torch.nn.functional as F
    from ctas_b200 import learned
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn((B, H, W, 128), device="cuda", generator=g).bfloat16()
    w = (torch.randn((32, 9, 128), device="cuda", generator=g) * 0.1).bfloat16()
    b = torch.randn(32, device="cuda", generator=g)
    mask = torch.randn((B, H, W, 32), device="cuda", generator=g).bfloat16() if masked else None
    y = learned.conv3x3(x, w, b, mask=mask, relu=relu)
    tw = w.float().reshape(32, 3, 3, 128).permute(0, 3, 1, 2)
    ref = F.conv2d(x.float().permute(0, 3, 1, 2), tw, b, padding=1).permute(0, 2, 3, 1)
    ref = F.relu(ref) if relu else ref
    ref = ref * (mask.float() > 0) if masked else ref
    torch.cuda.synchronize()
    assert float((y.float() - ref).abs().max()) <= 1e-2 * float(ref.abs().max())
