"""Chunks of the streamed volume call: a filter and a backprojection launch per chunk, and
the bits of one call per slice."""
import numpy as np
import pytest

from ctas_b200 import _lib, ct, volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,N,W,flags,launches", [
    (4, 60, 1090, False, 8),   # callbacks and copies bound the call: they overlap slice by slice
    (5, 60, 1090, False, 6),
    (4, 60, 1090, True, 2),    # a whole group where groups are asked for
    (16, 60, 1090, False, 8)])
def test_volume_chunks(S, N, W, flags, launches):
    x = np.random.default_rng(S).standard_normal((S, N, W)).astype(np.float32)
    kw = {"flags": _lib.FLAG_GROUPS} if flags else {}
    with ct.CTrec((N, W), ct.Contrast.PHS, 180.0, ct.Filter("HANN"), no_writeback=True, **kw) as rec:
        single = np.stack([rec.reconstruct(x[s].copy(), None, 1.5) for s in range(S)])
        before = rec.kernel_launches()
        got = volume.reconstruct_arrays(rec, x, 1.5)
        assert rec.kernel_launches() - before == launches
        assert np.array_equal(got.view(np.uint32), single.view(np.uint32))
