"""Output geometries whose pixel coordinates round more coarsely than the four-slice
kernel's sharing patterns allow for (a disc at the far end of very many rows) keep the
one-slice kernel; up to the limit the patterns hold."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

import oracle as O  # noqa: E402
from test_bp_quad_cover import SHARE, pattern_of  # noqa: E402

f32 = np.float32


def _shift(W, p, rows):
    """Shift that puts the last of `rows` rows at coordinate W - 1."""
    return (W - 1) / (2 * p) - (rows - 1) / 2


def _violations(W, p, rows, angles):
    """Angles at which some pixel of the last 64-row tiles has another index than both
    pixels whose sample it may take."""
    C = max(64, int(W / p) // 64 * 64)
    oj, oi, p = O.geometry(W, rows, C, p, _shift(W, p, rows), 0.0)
    hp = W // 2
    gj = f32(oj) + f32(p) * np.arange((rows - C) // 64 * 64, (rows - C) // 64 * 64 + C, dtype=f32)
    gi = f32(oi) + f32(p) * np.arange(C, dtype=f32)
    disc = np.hypot(gj[:, None] - hp, gi[None] - hp) < hp
    tab, m, bad = O.angle_table_list(angles), f32(W + 256) * f32(2.0 ** -19), []
    for n in range(len(angles)):
        sx, cy = f32(tab[2 * n]), f32(tab[2 * n + 1])
        base = ((f32(1) - sx) - cy) * f32(hp)
        k = np.floor((base + sx * gj[:, None]) + cy * gi[None]).astype(np.int64)
        row = abs(sx) < abs(cy)
        us, fs = ((abs(sx), abs(cy)) if row else (abs(cy), abs(sx)))
        pat = pattern_of(us * f32(p), fs * f32(p), m)

        def blocks(a):
            b = np.moveaxis(a, 0 if row else 1, -1)
            b = b.reshape(b.shape[0] // 2, 2, b.shape[1] // 4, 4)
            return b[..., ::-1] if (sx < 0) != (cy < 0) else b
        px, live = blocks(k), blocks(disc)
        for i, ab in enumerate(SHARE[pat]):
            if ab:
                v, a, b = (px[:, j // 4, :, j % 4] for j in (i, *ab))
                if ((v != a) & (v != b) & live[:, i // 4, :, i % 4]).any():
                    bad.append(float(angles[n]))
    return sorted(set(bad))


DENSE = np.concatenate([np.linspace(0.70, 0.79, 900), np.linspace(2.1, 2.4, 300)])


@pytest.mark.parametrize("W,p", [(64, 0.9973), (100, 0.83), (128, 0.771), (300, 0.61)])
def test_patterns_hold_up_to_the_limit(W, p):
    assert _violations(W, p, int((4 * W + 1024) / p), DENSE) == []


@pytest.mark.skipif(not shutil.which("g++"), reason="g++ is missing")
def test_limit(tmp_path):
    exe = str(tmp_path / "quad_geometry")
    subprocess.run(["g++", "-std=c++17", os.path.join(HERE, "cpp", "quad_geometry.cpp"), "-o", exe],
                   check=True)
    cases = [(100, 65536, 64, 0.83, 0), (100, 64, 65536, 0.83, 0), (100, 1000, 1000, 0.83, 1),
             (2560, 2560, 2560, 1.0, 1), (4096, 40960, 40960, 0.1, 1), (64, 1285, 10, 0.9973, 0)]
    out = subprocess.run([exe], input="\n".join("%d %d %d %f" % c[:4] for c in cases), text=True,
                         capture_output=True, check=True).stdout.split()
    assert [int(v) for v in out] == [c[4] for c in cases]


@pytest.mark.gpu
def test_far_disc_bitexact():
    """A stack on 65536 rows, the disc in the last 120, at angles where the patterns fail."""
    from ctas_b200 import _lib, ct
    W, p, rows, cols, S = 100, 0.83, 65536, 64, 4
    th = _violations(W, p, rows, DENSE)
    assert len(th) >= 3
    q = np.random.default_rng(1).standard_normal((S, len(th), W)).astype(np.float32)
    shift = (_shift(W, p, rows), 0.0)
    with ct.CTrec((len(th), W), ct.Contrast.FLT, angles=np.array(th), out_shape=(rows, cols),
                  out_pixel=p, out_shift=shift, flags=_lib.FLAG_GROUPS) as rec:
        got = rec.reconstruct_stack(q.copy(), None, 0.0)
    oj, oi, pf = O.geometry(W, rows, cols, p, *shift)
    tab = O.angle_table_list(np.array(th))
    for s in range(S):
        want = O.bp_compat_geom(q[s], tab, 0.0, 1.0, rows, cols, oj, oi, pf)
        assert (want != 0).any()
        assert np.array_equal(got[s].view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), s
