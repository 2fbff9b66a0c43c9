"""Stack calls on a nearly full device: where the buffers of four-slice groups do not fit
but those of one slice at a time do, the call runs so, with the same bits."""
import numpy as np
import pytest

from ctas_b200 import ct

pytestmark = pytest.mark.gpu
N, W, S, C = 1800, 1024, 16, 1.5
MB = 1 << 20


def test_stack_falls_back_to_single_slices():
    import torch
    x = torch.from_numpy(np.random.default_rng(3).standard_normal((S, N, W)).astype(np.float32)).cuda()
    want, got = (torch.empty((S, W, W), device="cuda") for _ in range(2))
    with ct.CTrec((N, W), ct.Contrast.PHS, 180.0) as rec:   # loads and tunes the kernels
        rec.reconstruct_stack_dev(x, want, C)
        assert rec.last_tile() == -1
        rec.reconstruct_dev(x[0], got[0], C)
        torch.cuda.synchronize()
    want = want.cpu().view(torch.int32)
    row = 4 * 1040 * N                                      # a slice's padded rows
    single = S * row + S * 4 * W * W                        # filtered rows, slices
    with ct.CTrec((N, W), ct.Contrast.PHS, 180.0) as rec:
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - single - 12 * MB, dtype=torch.uint8,
                          device="cuda")
        if not single + 6 * MB < torch.cuda.mem_get_info()[0] < single + 2 * row + 6 * MB:
            pytest.skip("free device memory is not this process's alone")
        rec.reconstruct_stack_dev(x, got, C)
        torch.cuda.synchronize()
        assert rec.last_tile() != -1                        # one slice at a time
        assert torch.equal(got.cpu().view(torch.int32), want)
        del hog
        torch.cuda.empty_cache()
        got.fill_(float("nan"))
        rec.reconstruct_stack_dev(x, got, C)                # and in groups again
        torch.cuda.synchronize()
        assert rec.last_tile() == -1
        assert torch.equal(got.cpu().view(torch.int32), want)
