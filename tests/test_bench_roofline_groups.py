"""The roofline term of bench.py for the four-slice kernel: bytes of the loads that the
sharing patterns leave, counted here from the patterns themselves, and a fraction that a
measured time cannot bring above 1."""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
sys.path.insert(0, HERE)

import bench  # noqa: E402
import oracle as O  # noqa: E402
from test_bp_quad_cover import SHARE, pattern_of  # noqa: E402


def test_group_roofline():
    f32 = np.float32
    tab = np.abs(O.angle_table(180.0, bench.N_ANGLES).reshape(-1, 2))
    m = f32(bench.WIDTH + 256) * f32(2.0 ** -19)
    loads = np.mean([sum(ab is None for ab in SHARE[pattern_of(min(p), max(p), m)])
                     for p in tab]) / 8
    assert abs(bench.quad_loads_per_update() - loads) < 1e-3
    bp_ms, S, sms, mhz = 105.6, 128, 148, 1965.0     # 1167 slices/s
    r = bench.roofline(bp_ms, S, 4.0, 36000.0, {"sm_mhz": mhz}, sms, 16000.0, -1)
    inmask = int(O.mask(bench.WIDTH, bench.CENTER).sum())
    assert np.isclose(r["algorithmic_bytes_per_launch"],
                      4.0 * bench.quad_loads_per_update() * bench.N_ANGLES * inmask * S)
    assert abs(r["frac"] - r["achieved"] / r["peak"]) < 1e-3
    assert 0.4 < r["frac"] < 1.0
    assert r["loads_per_update"] == round(bench.quad_loads_per_update(), 4)
    one = bench.roofline(200.0, S, 4.0, 36000.0, {"sm_mhz": mhz}, sms, 16000.0, 15)
    assert one["loads_per_update"] == 1.0
