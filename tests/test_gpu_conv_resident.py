"""The tiled convolution with its weights kept in shared memory and with weights loaded
along with each input box, which images of few tiles take: both against torch, and equal
bits on the same pixels."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (64, 64), (64, 128), (128, 64), (96, 32),
                                      (32, 96)])
def test_few_and_many_tiles(cin, cout):
    """One image of 32 tiles, and a batch of as many images as exceed two tiles per SM (W not
    a multiple of 128): within 1e-2 of the output range of a float32 convolution, the
    bound of the other shapes, and the image's output the same in both."""
    import torch
    import torch.nn.functional as F
    from ctas_b200 import learned
    H, W = 64, 64
    B = 2 * torch.cuda.get_device_properties(0).multi_processor_count // 32 + 1
    g = torch.Generator(device="cuda").manual_seed(cin + cout)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).bfloat16()
    w = (torch.randn((cout, 9, cin), device="cuda", generator=g) * 0.1).bfloat16()
    b = torch.randn(cout, device="cuda", generator=g)
    many = learned.conv3x3(x, w, b, relu=False)
    few = learned.conv3x3(x[-1:].contiguous(), w, b, relu=False)
    tw = w.float().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
    ref = F.conv2d(x.float().permute(0, 3, 1, 2), tw, b, padding=1).permute(0, 2, 3, 1)
    torch.cuda.synchronize()
    assert float((many.float() - ref).abs().max()) <= 1e-2 * float(ref.abs().max())
    assert torch.equal(few.view(torch.int16), many[-1:].view(torch.int16))


def test_waits_run_out_with_resident_weights():
    """The first input box left out: the waits end, the next call reports it, and the
    output is then that of before."""
    import torch
    from ctas_b200 import _lib, ct, learned
    B = 2 * torch.cuda.get_device_properties(0).multi_processor_count // 32 + 1
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn((B, 64, 64, 64), device="cuda", generator=g).bfloat16()
    w = (torch.randn((128, 9, 64), device="cuda", generator=g) * 0.1).bfloat16()
    before, L = learned.conv3x3(x, w, None), _lib.load()
    torch.cuda.synchronize()
    _lib.check(L.ctas_nn_test_timeout(1))
    try:
        learned.conv3x3(x, w, None)
        torch.cuda.synchronize()
    finally:
        _lib.check(L.ctas_nn_test_timeout(0))
    with pytest.raises(ct.CtasError) as e:
        learned.conv3x3(x, w, None)
    assert e.value.code == _lib.E_TIMEOUT
    after = learned.conv3x3(x, w, None)
    torch.cuda.synchronize()
    assert torch.equal(before.view(torch.int16), after.view(torch.int16))
