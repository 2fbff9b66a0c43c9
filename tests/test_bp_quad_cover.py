"""CPU proof of the four-slice backprojector's index bounds (bp_quad.cu), with the
kernel's float32 arithmetic operation for operation: the window of every tile
that holds a reconstructed pixel covers the tile's pixels and stays within the
rows and their slack, and the pixels that take another pixel's sample have that
pixel's index."""
import numpy as np
import pytest

import oracle as O

f32 = np.float32
TILES = [(64, 64, 96), (32, 64, 80)]        # rows, columns, window samples
SLACK = 256                                 # kQuadSlack, fbp_kernels.hpp
# sharing patterns (share(), bp_quad.cu): for each pixel 4 r + k None (it loads its
# sample) or the two pixels one of whose indices it has
L = None
SHARE = [[L] * 8,
         [L, (0, 4), (4, 5), L, L, L, (3, 7), L],
         [L, (0, 4), (4, 3), L, L, (4, 3), (3, 7), L],
         [L, (0, 4), (0, 4), (4, 6), L, (4, 6), L, L],
         [L, (0, 4), (0, 4), (0, 4), L, (4, 7), (4, 7), L],
         [L, (0, 3), (0, 3), L, L, (4, 7), (4, 7), L]]


def pattern_of(u, s, m):
    one = f32(1) - m
    if s <= one and u + m <= s:
        if f32(3) * u <= one and f32(3) * u + m <= s:
            return 4
        if f32(2) * u <= one and f32(2) * u + m <= s and s + m <= f32(3) * u:
            return 3
        if s + m <= f32(2) * u:
            return 2 if f32(3) * u - s <= one else 1
    return 5 if f32(3) * u <= one else 0


def check_pattern(pat, k, slow_axis, mirrored):
    """k: indices of a grid of pixels, in whole 4 x 2 blocks."""
    b = np.moveaxis(k, slow_axis, -1)                       # (fast, slow)
    b = b.reshape(b.shape[0] // 2, 2, b.shape[1] // 4, 4)
    if mirrored:
        b = b[..., ::-1]
    px = [b[:, i // 4, :, i % 4] for i in range(8)]
    for i, ab in enumerate(SHARE[pat]):
        if ab:
            assert ((px[i] == px[ab[0]]) | (px[i] == px[ab[1]])).all(), (pat, i)


def _geo(o, p, n):
    return f32(o) + f32(p) * np.arange(n, dtype=f32)


@pytest.mark.parametrize("W,N,c,arc,p", [
    (256, 180, 0.0, 180.0, 1.0), (301, 61, -11.25, 180.0, 1.0), (256, 60, 3.5, 180.0, 0.61),
    (2560, 7, 3.5, 180.0, 1.0), (4096, 5, 12.25, 180.0, 1.0), (16000, 3, -8.0, 177.0, 1.0),
    (300, 60, -11.25, 360.0, 1.0), (200, 50, -90.25, 360.0, 1.0), (384, 30, 20.75, 270.0, 0.8),
    (67, 60, 1.5, 180.0, 1.0), (33, 40, 0.0, 360.0, 1.0), (5, 7, 0.5, 180.0, 1.0)])
def test_windows_and_patterns(W, N, c, arc, p):
    tab = O.angle_table(arc, N)
    wide = (tab[0::2] < 0).any()
    off = ((W + 16 + 7) // 8) * 8 if wide else 8
    Wp = off + ((2 * W + 16 + 7) // 8) * 8 if wide else ((W + 9 + 7) // 8) * 8 + 8
    hp = W // 2
    big = W > 4096
    R = W if p == 1.0 else int(W / p) + 3
    o = f32(0) if p == 1.0 else f32((W - 1) / 2 - p * (R - 1) / 2)
    pad = -(-R // 64) * 64
    g = _geo(o, p, pad)
    rows = np.arange(pad)
    if big:                                 # bands of tiles through the image
        rows = np.concatenate([np.arange(k, k + 64) for k in range(0, pad, 64 * 62)])
    jj, ii = g[rows][:, None], g[None, :]
    # the mask of the kernels at float coordinates
    ac = f32(abs(c))
    d = ((jj - f32(hp)) - f32(c)) ** 2 + (ii - f32(hp)) ** 2
    hpc, hmc = f32(hp) + f32(c), f32(hp) - f32(c)
    m = (ii > ac) & (ii < (f32(W) - ac) - f32(1))
    m = m & ~(((jj <= hpc) & (d >= hpc * hpc)) | ((jj >= hpc) & (d >= hmc * hmc)))
    m[rows >= R] = False
    m[:, R:] = False
    assert m.any()
    used = np.zeros(6, int)
    for n in range(N):
        sx, cy = f32(tab[2 * n]), f32(tab[2 * n + 1])
        base = f32(c) + ((f32(1) - sx) - cy) * f32(hp)
        jc = jj - f32(c)
        t = (base + sx * jc) + cy * ii
        fl = np.floor(t).astype(np.int64)
        tr = np.trunc(t).astype(np.int64)
        for TY, TX, BOX in TILES:
            for jb in range(0, len(rows), TY):
                for i0 in range(0, pad, TX):
                    mm = m[jb:jb + TY, i0:i0 + TX]
                    if not mm.any():
                        continue
                    b = base + sx * jc[[jb, jb + TY - 1], 0]
                    e = cy * ii[0, [i0, i0 + TX - 1]]
                    tmin = (b[:, None] + e[None, :]).min()
                    x0 = int(np.floor(tmin)) - 2
                    k = tr if wide and tmin < f32(1) else fl
                    k = k[jb:jb + TY, i0:i0 + TX]
                    assert k.min() >= x0 and k.max() < x0 + BOX
                    assert off + x0 >= -SLACK and off + x0 + BOX <= Wp + SLACK
                    want = tr[jb:jb + TY, i0:i0 + TX][mm]
                    got = k[mm]
                    if not wide:            # column -1 repeats sample 0
                        got = np.maximum(got, 0)
                    assert np.array_equal(got, want)
        # the pixels that take another one's sample, for the layout that suits the
        # projection and (runs along the slow axis alone) for the other ones
        m_ = f32(W + 256) * f32(2.0 ** -19)
        mirrored = (sx < 0) != (cy < 0)
        for row in (False, True):
            us, fs = (abs(sx), abs(cy)) if row else (abs(cy), abs(sx))
            us, fs = us * f32(p), fs * f32(p)
            for k in (fl, tr) if wide else (fl,):
                if row == (abs(sx) < abs(cy)):
                    pat = pattern_of(us, fs, m_)
                    used[pat] += 1
                    check_pattern(pat, k, 0 if row else 1, mirrored)
                check_pattern(5 if f32(3) * us <= f32(1) - m_ else 0, k, 0 if row else 1, False)
    if N >= 180 and p == 1.0:
        assert (used > 0).all()
