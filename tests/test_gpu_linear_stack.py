"""Linear interpolation in stacks: slices in four-slice groups add their samples in another
order than single calls do (one sum of interpolated samples, where the one-slice kernel
sums samples and differences apart), so they agree to rounding, not to the bit."""
import numpy as np
import pytest

from ctas_b200 import _lib, ct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,N,W,c", [(5, 97, 200, 1.25), (6, 180, 301, -4.5), (8, 64, 96, 0.0),
                                     (6, 40, 500, 2.0)])
def test_linear_stack_close_to_single_calls(S, N, W, c):
    """Each way's sum of N products of at most m = 2 max|q| carries at most 2 N roundings
    of partial sums below N m, half an ulp each: 4 N 2^-24 m between both ways' means.  The
    slices that groups leave over equal the single calls."""
    q = np.random.default_rng(S).standard_normal((S, N, W)).astype(np.float32)
    with ct.CTrec((N, W), ct.Contrast.FLT, 180.0, interp=1, flags=_lib.FLAG_GROUPS) as rec:
        rec.setPhysics(0.0, 0.0)
        single = np.stack([rec.reconstruct(q[s].copy(), None, c) for s in range(S)])
        got = rec.reconstruct_stack(q.copy(), None, c)
        assert rec.last_kernel() == 2
    bound = 4 * N * 2.0 ** -24 * 2 * np.abs(q).max()
    assert np.abs(got.astype(np.float64) - single).max() <= bound
    assert np.abs(single).max() > 100 * bound
    if S % 4 in (1, 2) and W > 448:
        n = S - S % 4
        assert np.array_equal(got[n:].view(np.uint32), single[n:].view(np.uint32))
