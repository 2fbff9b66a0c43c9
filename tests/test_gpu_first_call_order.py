"""First calls of a handle on a stream of its own, while the legacy stream is busy: the
zeroing of the work buffers that such a call allocates stays ahead of the filter's
stores into them."""
import numpy as np
import pytest

from ctas_b200 import _lib, ct

pytestmark = pytest.mark.gpu
N, W, S, C = 120, 300, 6, 1.5


def _rows(seed):
    return np.random.default_rng(seed).standard_normal((S, N, W)).astype(np.float32)


def _bits(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("arc", [180.0, 360.0])
def test_first_filter_outlives_busy_legacy_stream(arc):
    """sino_dev of a fresh handle on a side stream; the filtered rows are still there
    when everything queued on the legacy stream has run."""
    import torch
    x = torch.from_numpy(_rows(1)).cuda()
    want, got = torch.empty((2, W, W), device="cuda")
    with ct.CTrec((N, W), ct.Contrast.PHS, arc) as rec:
        rec.sino_dev(x[0])
        rec.repeat_dev(want, C)
        torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with ct.CTrec((N, W), ct.Contrast.PHS, arc) as rec:
        torch.cuda._sleep(40_000_000)  # about 20 ms on the legacy stream
        with torch.cuda.stream(side):
            rec.sino_dev(x[0])
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            rec.repeat_dev(got, C)
        torch.cuda.synchronize()
    assert np.array_equal(_bits(got), _bits(want))


@pytest.mark.parametrize("store", [0, 1])
@pytest.mark.parametrize("cycles", [0, 200_000, 2_000_000, 40_000_000])
def test_first_stack_beside_busy_legacy_stream(cycles, store):
    """reconstruct_stack_dev of a fresh handle on a side stream, the legacy stream busy for
    0 to 20 ms: the bits of the same call on an idle device."""
    import torch
    x = torch.from_numpy(_rows(2)).cuda()
    out = []
    for busy in (0, cycles):
        y = torch.full((S, W, W), float("nan"), device="cuda")
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with ct.CTrec((N, W), ct.Contrast.PHS, 180.0, store=store, flags=_lib.FLAG_GROUPS) as rec:
            if busy:
                torch.cuda._sleep(busy)
            with torch.cuda.stream(side):
                rec.reconstruct_stack_dev(x, y, C)
            side.synchronize()
            out.append(_bits(y))
            torch.cuda.synchronize()
    assert np.array_equal(out[0], out[1])


def test_batch_made_beside_busy_legacy_stream():
    """A batch made and run on a side stream while the legacy stream is busy."""
    import torch
    x = torch.from_numpy(_rows(3)).cuda()
    out = []
    for busy in (0, 40_000_000):
        y = torch.full((2, W, W), float("nan"), device="cuda")
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        if busy:
            torch.cuda._sleep(busy)
        with torch.cuda.stream(side):
            batch = ct.Batch([(x[0], y[0], C), (x[1], y[1], -C)], ct.Contrast.PHS, 180.0,
                             ct.Filter("HANN"))
            batch.run()
        side.synchronize()
        out.append(_bits(y))
        batch.close()
        torch.cuda.synchronize()
    assert np.array_equal(out[0], out[1])
