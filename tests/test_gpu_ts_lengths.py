"""Tomosynthesis rows whose transform length is 3 or 5 times a power of two: the
oracle's exact circular convolution, at the edges of the ranges of widths that take
each length, with the bounds of the other widths (1e-5 of the filtered rows' range,
1e-4 with the running sum of refraction contrast)."""
import numpy as np
import pytest

import oracle as O
from ctas_b200 import ct, ts

pytestmark = pytest.mark.gpu


# lengths 48, 80; 96, 160 (limits 24, 40 and 48, 80); 3 * 512, 5 * 256; 3 * 2048, 5 * 1024
@pytest.mark.parametrize("n", [17, 24, 33, 40, 41, 48, 65, 80, 640, 641, 768, 2049, 2560, 2561, 3072])
@pytest.mark.parametrize("cn", ["PHS", "REF"])
def test_filtered_rows_vs_oracle(n, cn):
    rows = 3
    g = np.random.default_rng(n)
    x = np.linspace(-1, 1, n)
    proj = (0.6 + 0.3 * np.exp(-(x / 0.3) ** 2) + 0.05 * g.standard_normal((rows, n))).astype(np.float32)
    res = g.standard_normal((rows, n)).astype(np.float32)
    contrast, fl = getattr(ct.Contrast, cn), ct.Filter("RAMP")
    want_p, want_r = O.ts_add(proj, res, fl.filter(), 0.0, 1.5, contrast, 0.3, 5)
    p, r = proj.copy(), res.copy()
    with ts.TS((rows, n), fl, contrast) as t:
        t.add(p, r, 1.5, 0.3, 5)
    tol = (1e-4 if cn == "REF" else 1e-5) * float(np.ptp(want_p))
    assert float(np.abs(p - want_p).max()) <= tol
    assert float(np.abs(r - want_r).max()) <= tol + 4 * float(np.spacing(np.abs(want_r).max()))
