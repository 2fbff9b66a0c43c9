"""Host stack calls whose chunks and groups the estimates choose: the bits of one call per
slice, filtered rows written back included, at sizes where whole stacks, some chunks or
no chunk are grouped."""
import numpy as np
import pytest

from ctas_b200 import ct

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("N,W,counts,arc,store", [
    (24, 1090, (3, 4, 5, 9, 17, 18, 22), 180.0, 0), (24, 700, (4, 7, 16, 31, 45), 180.0, 0),
    (24, 1090, (4, 6, 18), 360.0, 0), (24, 900, (4, 5, 20, 33), 180.0, 1),
    (400, 300, (3, 40, 47), 180.0, 0), (1500, 1400, (4, 6, 9), 180.0, 0)])
def test_host_stack_equals_single_calls(N, W, counts, arc, store, pinned):
    import torch
    S, c = max(counts), 2.25
    x = np.random.default_rng(W).standard_normal((S, N, W)).astype(np.float32)
    with ct.CTrec((N, W), ct.Contrast.PHS, arc, ct.Filter("HANN"), store=store) as rec:
        back = x.copy()
        single = np.stack([rec.reconstruct(back[s], None, c) for s in range(S)])
        for n in counts:
            t = torch.empty((n, N, W), pin_memory=pinned), torch.empty((n, W, W), pin_memory=pinned)
            y, out = (v.numpy() for v in t)
            y[:], out[:] = x[:n], np.nan
            rec.reconstruct_stack(y, out, c)
            assert np.array_equal(_bits(out), _bits(single[:n])), n
            assert np.array_equal(_bits(y), _bits(back[:n])), n


@pytest.mark.parametrize("S,N,W,launches", [(4, 60, 2048, 8), (3, 60, 2048, 6), (8, 3000, 1400, 4)])
def test_chunks_follow_what_bounds_the_call(S, N, W, launches):
    """A filter and a backprojection launch per chunk: chunks of one slice where copies
    bound the call (they overlap), of a group of four where the kernels do."""
    import torch
    y, out = (torch.zeros(s, pin_memory=True).numpy() for s in ((S, N, W), (S, W, W)))
    with ct.CTrec((N, W), ct.Contrast.PHS, 180.0, no_writeback=True) as rec:
        rec.reconstruct_stack(y, out, 1.0)
        before = rec.kernel_launches()
        rec.reconstruct_stack(y, out, 1.0)
        assert rec.kernel_launches() - before == launches
