"""sino(), then a stack call that fails, then repeat(): the rows of sino() or an error,
never the rows of a buffer that the stack call has replaced or could not get."""
import numpy as np
import pytest

from ctas_b200 import _lib, ct

pytestmark = pytest.mark.gpu


def _x(S, N, W):
    return np.random.default_rng(W).uniform(0.1, 1.0, (S, N, W)).astype(np.float32)


def _refused(call):
    with pytest.raises(_lib.CtasError) as e:
        call()
    return e.value.code


@pytest.mark.parametrize("S,flags", [(3, 0), (3, _lib.FLAG_GROUPS), (9, _lib.FLAG_GROUPS)])
def test_after_bad_data(S, flags):
    import torch
    N, W = 60, 301
    x = _x(1, N, W)[0]
    bad, out = -np.ones((S, N, W), np.float32), np.empty((S, W, W), np.float32)
    with ct.CTrec((N, W), ct.Contrast.ABS, 180.0, flags=flags, chunk_slices=S) as rec:
        y = torch.empty((W, W), device="cuda")
        rec.sino_dev(torch.from_numpy(x).cuda())
        want = rec.repeat_dev(y, 1.5).cpu().clone()
        assert _refused(lambda: rec.reconstruct_stack(bad, out, 1.5)) == _lib.E_DATA
        assert _refused(lambda: rec.repeat_dev(y, 1.5)) == _lib.E_STATE
        rec.sino_dev(torch.from_numpy(x).cuda())
        assert _refused(lambda: rec.reconstruct_stack(bad, out, 1.5)) == _lib.E_DATA
        assert torch.equal(rec.repeat_dev(y, 1.5).cpu(), want)     # the buffers are large enough


def test_after_too_little_memory():
    import torch
    N, W, S = 1800, 1024, 16
    x, y = torch.from_numpy(_x(1, N, W)).cuda(), torch.empty((W, W), device="cuda")
    big, out = torch.zeros((S, N, W), device="cuda"), torch.empty((S, W, W), device="cuda")
    with ct.CTrec((N, W), ct.Contrast.PHS, 180.0) as rec:
        rec.sino_dev(x[0])
        rec.repeat_dev(y, 1.5)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (60 << 20), dtype=torch.uint8, device="cuda")
        assert _refused(lambda: rec.reconstruct_stack_dev(big, out, 1.5)) == _lib.E_NOMEM
        del hog
        torch.cuda.empty_cache()
        assert _refused(lambda: rec.repeat_dev(y, 1.5)) == _lib.E_STATE
