"""Rounding error of the tomosynthesis filter against 64 bits, where the transform
length is 3 times a power of two: no larger than that of the next power of two, which
such rows are transformed in elsewhere, for rows with and without a mean, derivatives,
steps, noise and combs.  The power of two's error is that of a float32 restatement of
its plan (radix 8, then 4 or 2; twiddles w and w^4 from a table, the others products)."""
import numpy as np
import pytest

import oracle as O

f32 = np.float32


def _fma(a, b, c):
    return (a.astype(np.float64) * b + c).astype(f32)


def _mul(a, b):                       # complex float32 product, one fused add each
    return _fma(a[0], b[0], -(a[1] * b[1])), _fma(a[0], b[1], a[1] * b[0])


def _bfly(x, d):
    """DFT of 2, 4 or 8 (re, im) pairs, direction d."""
    n = len(x)
    if n == 1:
        return x
    e, o = _bfly(x[0::2], d), _bfly(x[1::2], d)
    r, out = f32(np.sqrt(0.5)), [None] * n
    for k in range(n // 2):
        re, im = o[k]
        q = 8 * k // n                # eighths of a turn
        if q == 1:
            re, im = (re - d * im) * r, (im + d * re) * r
        elif q == 2:
            re, im = -d * im, d * re
        elif q == 3:
            re, im = (-re - d * im) * r, (-im + d * re) * r
        out[k] = e[k][0] + re, e[k][1] + im
        out[k + n // 2] = e[k][0] - re, e[k][1] - im
    return out


def _twiddles(P, R, h):
    def w(k):
        a = -2 * np.pi * (k % P) / P
        return np.cos(a).astype(f32), np.sin(a).astype(f32)
    m = np.arange(h) * (P // (R * h))
    t = [None, w(m)] + [None] * 6
    if R >= 4:
        t[2] = _mul(t[1], t[1])
        t[3] = _mul(t[2], t[1])
    if R == 8:
        t[4] = w(4 * m)
        t[5:8] = [_mul(t[4], t[k]) for k in (1, 2, 3)]
    return t


def _filter_pow2(x, fwin):
    """Rows (even number) filtered with the n-point window at the power of two."""
    n = x.shape[1]
    P = 1 << (2 * n - 2).bit_length()
    g = np.fft.ifft(fwin.astype(np.float64)).real
    h = np.zeros(P)
    for d in range(n // 2 + 1):
        v = g[d] * (0.5 if n % 2 == 0 and d == n // 2 else 1.0)
        h[d] += v
        if d:
            h[-d] += v
    lg = P.bit_length() - 1
    radices = [8] * (lg // 3) + [[], [2], [4]][lg % 3]
    order, mult = np.zeros(P, int), 1
    stages, L, p = [], P, np.arange(P)
    for R in radices:
        stages.append((R, L // R, L))
        L //= R
        order += (p // L) % R * mult
        mult *= R
    G = (np.fft.fft(h).real / P).astype(f32)[order]
    zs, m = n // 2, x.shape[0] // 2
    z = np.zeros((2, m, P), f32)
    idx = (np.arange(2 * n) - zs) % n
    z[0, :, :2 * n], z[1, :, :2 * n] = x[0::2][:, idx], x[1::2][:, idx]
    for R, s, L in stages:
        b = z.reshape(2, m, P // L, R, s)
        y = _bfly([(b[0, :, :, t], b[1, :, :, t]) for t in range(R)], f32(-1))
        if s > 1:
            w = _twiddles(P, R, s)
            y = y[:1] + [_mul(y[q], w[q]) for q in range(1, R)]
        z = np.stack([np.stack([v[c] for v in y], 2) for c in (0, 1)]).reshape(2, m, P)
    z = z * G
    for R, s, L in stages[::-1]:
        b = z.reshape(2, m, P // L, R, s)
        y = [(b[0, :, :, t], b[1, :, :, t]) for t in range(R)]
        if s > 1:
            w = _twiddles(P, R, s)
            y = y[:1] + [_mul(y[q], (w[q][0], -w[q][1])) for q in range(1, R)]
        y = _bfly(y, f32(1))
        z = np.stack([np.stack([v[c] for v in y], 2) for c in (0, 1)]).reshape(2, m, P)
    out = np.empty_like(x)
    out[0::2], out[1::2] = z[0, :, zs:zs + n], z[1, :, zs:zs + n]
    return out


def _rows(kind, n, m):
    g = np.random.default_rng(n)
    x, out = np.linspace(-1, 1, n), []
    for _ in range(m):
        c, s = g.uniform(-0.3, 0.3), g.uniform(0.1, 0.4)
        b = np.exp(-((x - c) / s) ** 2)
        noise = g.standard_normal(n)
        out.append({"mean": 0.6 + 0.3 * b + 0.05 * noise,
                    "smooth": b - b.mean(),
                    "derivative": np.gradient(b) * n / 50 + 0.003 * noise,
                    "noise": noise,
                    "comb": 1.0 * (np.arange(n) % max(1, n // 256) == 0) + 0.01 * noise,
                    "step": 1.0 * (x > c) - 0.5}[kind])
    return np.array(out).astype(f32)


KINDS = ["mean", "smooth", "derivative", "noise", "comb", "step"]


def _exact(x, fwin):
    return np.fft.ifft(np.fft.fft(x.astype(np.float64)) * fwin.astype(np.float64)).real


def _error(y, want):
    return float(np.linalg.norm(y - want) / np.linalg.norm(want))


def test_restatement_filters():
    """The restatement is a float32 filter: 1e-4 of 64 bits on rows of every kind."""
    for n in (600, 1025):
        fwin = O.filter_fill_plain(1, 0.0, n)
        for kind in KINDS:
            x = _rows(kind, n, 4)
            assert _error(_filter_pow2(x, fwin), _exact(x, fwin)) < 1e-4, (n, kind)


def _tall(n):
    """Rows of an image that takes the transform of 3 2^k (ts.cu, three_pays)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 2 * sms * (3 if n <= 4096 else 1) + 3


# 3072, 6144: the transform full; 2049, 4097: the shortest rows of each length
@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [2049, 2560, 3072, 4097, 6144])
def test_error_not_above_power_of_two(n, kind):
    """Over 64 rows of a tall image, whose errors scatter by a few per cent: at most 1.03
    times."""
    from ctas_b200 import ct, ts
    import torch
    fl = ct.Filter("RAMP")
    fwin = O.filter_fill_plain(fl.filter(), 0.0, n)
    x = _rows(kind, n, 64)
    d = torch.zeros((_tall(n), n), device="cuda")
    d[:64] = torch.from_numpy(x).cuda()
    with ts.TS(tuple(d.shape), fl, ct.Contrast.PHS) as t:
        t.add_batch_dev(d[None], np.zeros(1, f32), torch.zeros_like(d), 0.0, 0)
    want = _exact(x, fwin)
    assert _error(d[:64].cpu().numpy(), want) <= 1.03 * _error(_filter_pow2(x, fwin), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2049, 2560, 3072, 4098, 6144])
@pytest.mark.parametrize("cn", ["PHS", "ABS", "REF"])
def test_tall_images_vs_oracle(n, cn):
    """First and last rows of a tall image with an odd number of rows, filtered and added,
    against the oracle's exact circular convolution: the bounds of the other widths (1e-5
    of the filtered rows' range, 1e-4 with the running sum of refraction contrast); two
    calls and a batch of two give the same bits."""
    import torch
    from ctas_b200 import ct, ts
    rows, g, x = _tall(n), np.random.default_rng(n), np.linspace(-1, 1, n)
    pick = [0, 1, 2, rows - 2, rows - 1]
    proj = (0.6 + 0.3 * np.exp(-(x / 0.3) ** 2) + 0.02 * g.standard_normal((rows, n))).astype(f32)
    res = g.standard_normal((rows, n)).astype(f32)
    contrast, fl = getattr(ct.Contrast, cn), ct.Filter("RAMP")
    want_p, want_r = O.ts_add(proj[pick], res[pick], fl.filter(), 0.0, 1.5, contrast, 0.3, 5)
    with ts.TS((rows, n), fl, contrast) as t:
        p, r = proj.copy(), res.copy()
        t.add(p, r, 1.5, 0.3, 5)
        one, two = torch.from_numpy(res).cuda(), torch.from_numpy(res).cuda()
        d = torch.from_numpy(np.stack([proj, proj[::-1].copy()])).cuda()
        angles = np.array([0.3, -0.2], f32)
        for k in (0, 1):
            t.add_batch_dev(d[k:k + 1].clone(), angles[k:k + 1], one, 1.5, 5)
        t.add_batch_dev(d, angles, two, 1.5, 5)
        torch.cuda.synchronize()
    assert torch.equal(one.view(torch.int32), two.view(torch.int32))
    tol = (1e-4 if cn == "REF" else 1e-5) * float(np.ptp(want_p))
    assert float(np.abs(p[pick] - want_p).max()) <= tol
    assert float(np.abs(r[pick] - want_r).max()) <= tol + 4 * float(np.spacing(np.abs(want_r).max()))
