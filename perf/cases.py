"""Performance cases: the work a user of this package has it do, through its
public entry points, with the sizes, options and value distributions of real
use.

Kinds (the ``kind`` of a case):

* ``stack``  -- ``CTrec.reconstruct_stack_dev`` (``reconstruct_dev`` for one
  slice): filtered backprojection of sinograms held on the device;
* ``host``   -- ``CTrec.reconstruct_stack``: the same from and to pinned host
  memory, copies included;
* ``axis``   -- ``CTrec.sino_dev`` and ``repeat_multi_dev``: one sinogram
  filtered once and backprojected about several trial centres, the work of a
  rotation-axis search;
* ``batch``  -- ``Batch.run``: sinograms of mixed shapes in one graph launch;
* ``ts``     -- ``TS.add_batch_dev``: tomosynthesis of one plane;
* ``unet``   -- ``UNet.forward``: the learned sparse-angle stage, inference;
* ``conv``   -- one 3x3 convolution layer of that network forward and backward
  (activation, data gradient, weight gradient), the step its training repeats.

Inputs are seeded: exact projections of random ellipses with photon noise for
the reconstructions, unit-scale images and activations for the network.  The
64-bit values of ``exact`` keep the reconstruction's definition of which sample
a pixel reads (a float32 index expression, truncated) and do the rest in
float64.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from ctas_b200 import learned
from ctas_b200.ct import Batch, Contrast, CTrec, Filter
from ctas_b200.ts import TS

FILTERS = {"RAMP": Filter.RAMP, "HANN": Filter.HANN, "HAMMING": Filter.HAMMING,
           "SHEPP-LOGAN": Filter.SHEPP_LOGAN, "COSINE": Filter.COSINE}
CONTRASTS = {"ABS": Contrast.ABS, "PHS": Contrast.PHS}
STORES = {"f32": 0, "f16": 1, "bf16": 2}
PHOTONS = 1.0e4

# layers of the 4-level network in parameter order (cin, cout), 1x1 head
UNET = [(16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 256), (256, 256),
        (384, 128), (128, 128), (192, 64), (64, 64), (96, 32), (32, 32)]
HEAD = 32


def _stack(name, slices, angles, width, *, contrast="PHS", filt="RAMP", pad=0, store="f32",
           interp=0, arc=180.0, center=0.0, kind="stack"):
    case = {"kind": kind, "slices": slices, "angles": angles, "width": width,
            "contrast": contrast, "filter": filt, "pad": pad, "store": store, "interp": interp,
            "arc": arc, "center": center}
    return {"name": name, **case} if name else case


def listed():
    return [
        # one small slice, the call of an interactive preview: latency and an
        # almost empty chip
        _stack("slice_720x512", 1, 720, 512, pad=1024, center=-0.5),
        # a few odd-sized slices of raw absorption data (minus-log in the call)
        _stack("stack_abs_5x901x1023", 5, 901, 1023, contrast="ABS", center=2.25),
        # the main use: a stack of detector rows of a tomography scan
        _stack("stack_32x1800x2560", 32, 1800, 2560, filt="HANN", pad=4096, center=3.5),
        # the same scan with half-size filtered sinograms
        _stack("stack_f16_16x1800x2560", 16, 1800, 2560, filt="HANN", pad=4096, store="f16",
               center=3.5),
        # a full-turn scan (360 degrees)
        _stack("turn_6x1800x2560", 6, 1800, 2560, filt="HANN", pad=4096, arc=360.0, center=3.5),
        # linear detector interpolation
        _stack("linear_4x900x1536", 4, 900, 1536, filt="COSINE", interp=1, center=-1.75),
        # large detector rows from and to host memory, as a volume is streamed
        _stack("host_8x3600x4096", 8, 3600, 4096, filt="HAMMING", pad=8192, center=12.25,
               kind="host"),
        # rotation-axis search: one sinogram, a grid of trial centres
        {"name": "axis_9x1800x2560", "kind": "axis", "centers": 9, "angles": 1800, "width": 2560,
         "filter": "RAMP", "pad": 0, "span": 8.0},
        # sinograms of mixed widths and projection counts in one launch
        {"name": "batch_12", "kind": "batch", "jobs": 12, "shapes": 7, "filter": "SHEPP-LOGAN"},
        # tomosynthesis: one plane from 31 projection images
        {"name": "ts_31x1024x2560", "kind": "ts", "images": 31, "rows": 1024, "width": 2560,
         "filter": "RAMP", "center": 3.5, "plane": 500},
        # learned stage: inference on sparse-angle slices
        {"name": "unet_2x2048x2048", "kind": "unet", "batch": 2, "rows": 2048, "cols": 2048},
        # learned stage: one training layer, forward and backward
        {"name": "conv_64_2x1024x1024", "kind": "conv", "cin": 64, "cout": 64, "batch": 2,
         "rows": 1024, "cols": 1024},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stack"] * 6 + ["host", "host", "axis", "batch", "ts", "unet", "conv"])
    if kind in ("stack", "host"):
        while True:
            slices = _logint(rng, 1, 40) if kind == "stack" else _logint(rng, 2, 24)
            angles, width = _logint(rng, 180, 3600), _logint(rng, 180, 4096)
            if slices * angles * width * width <= 3.5e11:
                break
        option = rng.choice(["plain"] * 6 + ["f16", "f16", "bf16", "turn", "turn", "linear"])
        padded = 1 << (2 * width - 2).bit_length()
        return _stack(None, slices, angles, width, contrast=rng.choice(["PHS", "PHS", "ABS"]),
                      filt=rng.choice(sorted(FILTERS)),
                      pad=rng.choice([0, padded // 2]) if padded // 2 > width + 1 else 0,
                      store=option if option in STORES else "f32",
                      interp=1 if option == "linear" else 0,
                      arc=360.0 if option == "turn" else 180.0,
                      center=round(rng.uniform(-0.01, 0.01) * width, 2), kind=kind)
    if kind == "axis":
        return {"kind": kind, "centers": rng.randint(2, 17), "angles": _logint(rng, 300, 1800),
                "width": _logint(rng, 500, 2560), "filter": rng.choice(["RAMP", "HANN"]),
                "pad": 0, "span": round(rng.uniform(2.0, 12.0), 2)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(3, 16), "shapes": rng.randint(0, 1000),
                "filter": rng.choice(["SHEPP-LOGAN", "HANN"])}
    if kind == "ts":
        return {"kind": kind, "images": rng.randint(5, 61), "rows": _logint(rng, 64, 1500),
                "width": _logint(rng, 500, 3000), "filter": rng.choice(["RAMP", "HANN"]),
                "center": round(rng.uniform(-10, 10), 2), "plane": rng.randint(-200, 800)}
    if kind == "unet":
        return {"kind": kind, "batch": rng.randint(1, 4), "rows": 64 * rng.randint(4, 24),
                "cols": 128 * rng.randint(2, 12)}
    cin, cout = rng.choice([c for c in UNET if c[0] % 32 == 0])
    return {"kind": "conv", "cin": cin, "cout": cout, "batch": rng.randint(1, 4),
            "rows": 8 * rng.randint(8, 96), "cols": 16 * rng.randint(8, 48)}


# ------------------------------------------------------------------ inputs
def _projections(seed, slices, angles, width, arc, center):
    """Projections of random ellipses (line integrals of order 1) with photon
    noise: transmitted fractions (slices, angles, width), float32 on the GPU."""
    g = np.random.default_rng(seed)
    gpu = torch.Generator(device="cuda").manual_seed(seed)
    th = torch.arange(angles, device="cuda", dtype=torch.float64) * (math.radians(arc) / angles)
    cs, sn = th.cos().float()[:, None], th.sin().float()[:, None]
    u = (torch.arange(width, device="cuda", dtype=torch.float32) + 0.5 - width // 2 - center)[None]
    radius = 0.5 * width - abs(center) - 2.0
    out = torch.empty((slices, angles, width), device="cuda")
    for s in range(slices):
        p = torch.zeros((angles, width), device="cuda")
        for _ in range(8):
            a, b = g.uniform(0.05, 0.35, 2) * radius
            r, phi, turn = (radius - max(a, b)) * math.sqrt(g.uniform()), *g.uniform(0, 6.283, 2)
            rho = g.uniform(0.05, 0.5) * 4.0 / width
            na = cs * math.cos(phi) + sn * math.sin(phi)
            nb = sn * math.cos(phi) - cs * math.sin(phi)
            r2 = (a * na) ** 2 + (b * nb) ** 2
            d = u - r * (cs * math.cos(turn) + sn * math.sin(turn))
            p += (2.0 * rho * a * b / r2) * (r2 - d * d).clamp_min_(0.0).sqrt_()
        out[s] = torch.poisson(PHOTONS * torch.exp(-p), generator=gpu) / PHOTONS
    return out


def _phases(seed, slices, angles, width, arc, center):
    """The same as line integrals: -log of the transmitted fractions."""
    p = _projections(seed, slices, angles, width, arc, center)
    return p.clamp_min_(0.5 / PHOTONS).log_().neg_()


def _stack_input(case, seed):
    make = _projections if case["contrast"] == "ABS" else _phases
    return make(seed, case["slices"], case["angles"], case["width"], case["arc"], case["center"])


def _batch_jobs(case):
    g = np.random.default_rng(case["shapes"])
    return [(int(g.choice([900, 1200, 1800])), int(g.choice([1024, 1536, 2048, 2560])),
             round(float(g.uniform(-8, 8)), 3)) for _ in range(case["jobs"])]


def _axis_centers(case):
    return np.linspace(-case["span"], case["span"], case["centers"]).astype(np.float32)


def _ts_angles(case):
    return np.linspace(-0.5, 0.5, case["images"]).astype(np.float32)


def _unet_params(seed):
    g = np.random.default_rng(seed)
    parts = []
    for cin, cout in UNET:
        parts.append(g.standard_normal(cout * 9 * cin) * math.sqrt(2.0 / (9 * cin)))
        parts.append(0.01 * g.standard_normal(cout))
    parts += [0.1 * g.standard_normal(HEAD), np.array([0.02])]
    return np.concatenate(parts).astype(np.float32)


def _unet_input(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((case["batch"], case["rows"], case["cols"]), device="cuda", generator=g)


def _conv_input(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, W, ci, co = case["batch"], case["rows"], case["cols"], case["cin"], case["cout"]
    x = torch.randn((B, H, W, ci), device="cuda", generator=g).relu_().bfloat16()
    w = (torch.randn((co, 9, ci), device="cuda", generator=g) * math.sqrt(2.0 / (9 * ci))).bfloat16()
    b = 0.1 * torch.randn(co, device="cuda", generator=g)
    dy = torch.randn((B, H, W, co), device="cuda", generator=g).bfloat16()
    return x, w, b, dy


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("stack", "host"):
        S, N, W = case["slices"], case["angles"], case["width"]
        x = _stack_input(case, seed)
        state["rec"] = CTrec((N, W), CONTRASTS[case["contrast"]], case["arc"],
                             Filter(FILTERS[case["filter"]]), pad=case["pad"],
                             store=STORES[case["store"]], interp=case["interp"],
                             no_writeback=kind == "host")
        if kind == "stack":
            state["x"], state["y"] = x, torch.empty((S, W, W), device="cuda")
        else:
            state["keep"] = _pinned((S, N, W)), _pinned((S, W, W))
            state["keep"][0].copy_(x)
            state["x"], state["y"] = (t.numpy() for t in state["keep"])
    elif kind == "axis":
        N, W = case["angles"], case["width"]
        state["x"] = _phases(seed, 1, N, W, 180.0, 0.0)[0]
        state["rec"] = CTrec((N, W), Contrast.PHS, 180.0, Filter(FILTERS[case["filter"]]),
                             pad=case["pad"])
        state["y"] = torch.empty((case["centers"], W, W), device="cuda")
    elif kind == "batch":
        jobs = []
        for k, (N, W, c) in enumerate(_batch_jobs(case)):
            jobs.append((_phases(seed + 1000 * k, 1, N, W, 180.0, c)[0],
                         torch.empty((W, W), device="cuda"), c))
        torch.cuda.synchronize()  # the batch is tuned on its inputs when it is made
        state["jobs"] = jobs
        state["batch"] = Batch(jobs, Contrast.PHS, 180.0, Filter(FILTERS[case["filter"]]))
    elif kind == "ts":
        n, rows, W = case["images"], case["rows"], case["width"]
        state["x"] = _phases(seed, n, rows, W, 180.0, 0.0)
        state["y"] = torch.zeros((rows, W), device="cuda")
        state["ts"] = TS((rows, W), Filter(FILTERS[case["filter"]]), Contrast.PHS)
        state["angles"] = _ts_angles(case)
    elif kind == "unet":
        state["net"] = learned.UNet(0, 2.0)
        state["net"].set_params(_unet_params(seed))
        state["x"] = _unet_input(case, seed)
        state["y"] = torch.empty_like(state["x"])
    else:
        state["x"], state["w"], state["b"], state["dy"] = _conv_input(case, seed)
        state["y"] = torch.empty_like(state["dy"])
        state["dx"] = torch.empty_like(state["x"])
        state["dw"] = torch.empty(state["w"].shape, device="cuda")
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "stack":
        if case["slices"] == 1:
            state["rec"].reconstruct_dev(state["x"][0], state["y"][0], case["center"])
        else:
            state["rec"].reconstruct_stack_dev(state["x"], state["y"], case["center"])
        return state["y"]
    if kind == "host":
        return state["rec"].reconstruct_stack(state["x"], state["y"], case["center"])
    if kind == "axis":
        state["rec"].sino_dev(state["x"])
        return state["rec"].repeat_multi_dev(_axis_centers(case), state["y"])
    if kind == "batch":
        state["batch"].run()
        return [y for _, y, _ in state["jobs"]]
    if kind == "ts":
        state["y"].zero_()
        return state["ts"].add_batch_dev(state["x"], state["angles"], state["y"], case["center"],
                                         case["plane"], writeback=False)
    if kind == "unet":
        return state["net"].forward(state["x"], state["y"])
    x, w, dy = state["x"], state["w"], state["dy"]
    y = learned.conv3x3(x, w, state["b"], y=state["y"], relu=True)
    dx = learned.conv3x3(dy, learned.flip_weights(w), None, y=state["dx"], relu=False)
    dw = learned.conv3x3_wgrad(x, dy, state["dw"].zero_())
    return {"y": y, "dx": dx, "dw": dw}


# ------------------------------------------------------------------ work
def _pad(width, pad):
    return pad or 1 << (2 * width - 2).bit_length()


def _fbp_work(sinos, slices, angles, width, pad):
    """Rows read once, slices written once; a forward and an inverse real
    transform per row (5/2 P log2 P each); an index add and an accumulation per
    pixel of the disc and projection."""
    p = _pad(width, pad)
    return {"bytes": 4.0 * (sinos * angles * width + slices * width * width),
            "flops": sinos * angles * 5.0 * p * math.log2(p)
            + 2.0 * slices * angles * math.pi / 4 * width * width}


def work(case):
    kind = case["kind"]
    if kind in ("stack", "host"):
        return _fbp_work(case["slices"], case["slices"], case["angles"], case["width"],
                         case["pad"])
    if kind == "axis":
        return _fbp_work(1, case["centers"], case["angles"], case["width"], case["pad"])
    if kind == "batch":
        each = [_fbp_work(1, 1, n, w, 0) for n, w, _ in _batch_jobs(case)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if kind == "ts":
        n, rows, w = case["images"], case["rows"], case["width"]
        return {"bytes": 4.0 * (n + 1) * rows * w,
                "flops": n * rows * (5.0 * w * math.log2(w) + 2.0 * w)}
    px = float(case["batch"] * case["rows"] * case["cols"])
    if kind == "unet":
        scale = [1, 1, 4, 4, 16, 16, 64, 64, 16, 16, 4, 4, 1, 1]
        macs = sum(9.0 * ci * co / s for (ci, co), s in zip(UNET, scale)) + HEAD
        return {"bytes": 8.0 * px + 2.0 * sum(9 * ci * co for ci, co in UNET),
                "flops": 2.0 * macs * px}
    ci, co = case["cin"], case["cout"]
    return {"bytes": 2.0 * px * 2 * (ci + co) + 9.0 * ci * co * 8,
            "flops": 3 * 2.0 * 9 * ci * co * px}


# ------------------------------------------------------------------ 64-bit values
def _window(n, filt):
    """Ram-Lak response of n taps times the window, halved, frequencies 0 .. n/2."""
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    taps = torch.zeros(n, device="cuda", dtype=torch.float64)
    odd = torch.arange(1, (n + 1) // 2, 2, device="cuda")
    taps[0] = 0.25
    taps[odd] = -1.0 / (math.pi * k[odd]) ** 2
    taps[n - odd] = taps[odd]
    f = k[:n // 2 + 1] * (2.0 / n)
    win = {"RAMP": torch.ones_like(f), "HANN": 0.5 + 0.5 * torch.cos(math.pi * f),
           "HAMMING": 0.54 + 0.46 * torch.cos(math.pi * f),
           "SHEPP-LOGAN": torch.sinc(f / 2), "COSINE": torch.cos(math.pi * f / 2)}[filt]
    return torch.fft.rfft(taps).real * win / 2


def _filtered(x, case, contrast):
    """Filtered rows of one sinogram (angles, width) in float64.  The padded row
    carries the next row's first sample behind its own."""
    N, W = x.shape
    x = x.double()
    if contrast == "ABS":
        if float(x.min()) <= 0:
            x = x.clamp_min(float(x.max()) / 1e6)
        x = -x.log()
    P = _pad(W, case["pad"])
    z0 = (P - W) // 2
    g = _window(P, case["filter"]) * (P / W)
    out = torch.empty_like(x)
    for r in range(0, N, 512):
        n = min(512, N - r)
        z = torch.zeros((n, P), device="cuda", dtype=torch.float64)
        z[:, z0:z0 + W] = x[r:r + n]
        nxt = x[r + 1:r + n + 1, 0]
        z[:nxt.shape[0], z0 + W] = nxt
        out[r:r + n] = torch.fft.irfft(torch.fft.rfft(z) * g, n=P)[:, z0:z0 + W]
    return out


def _disc(W, c):
    """Pixels (row, column) that are reconstructed, as float32 coordinates."""
    hp, ac = W // 2, abs(c)
    j = torch.arange(W, device="cuda", dtype=torch.float32)[:, None]
    i = torch.arange(W, device="cuda", dtype=torch.float32)[None, :]
    cf = torch.tensor(c, device="cuda", dtype=torch.float32)
    d = ((j - hp) - cf) ** 2 + (i - hp) ** 2
    m = (i > ac) & (i < (W - cf.abs()) - 1.0)
    m = m & ~((j <= hp + cf) & (d >= (hp + cf) ** 2)) & ~((j >= hp + cf) & (d >= (hp - cf) ** 2))
    return m.nonzero(as_tuple=True)


# the C library's float32 sine and cosine: the angle table is defined by them
_libm = ctypes.CDLL("libm.so.6")
_sinf, _cosf = _libm.sinf, _libm.cosf
for _f in (_sinf, _cosf):
    _f.restype, _f.argtypes = ctypes.c_float, [ctypes.c_float]


def _table(arc, N):
    f32 = np.float32
    total = f32(float(f32(arc)) * (math.pi / 180))
    rad = [float(f32(i) * total / f32(N)) for i in range(N)]
    return [(f32(_sinf(t)), f32(_cosf(t))) for t in rad]


def _backproject(q, arc, c, interp=0):
    """q (slices, angles, width) float64 filtered rows -> (slices, W, W)."""
    S, N, W = q.shape
    hp = W // 2
    jj, ii = _disc(W, c)
    j, i = jj.float(), ii.float()
    acc = torch.zeros((j.numel(), S), device="cuda", dtype=torch.float64)
    if interp:
        rows = torch.zeros((N, W + 4, S), device="cuda", dtype=torch.float64)
        rows[:, 2:W + 2] = q.permute(1, 2, 0)
        jd, idd = jj.double(), ii.double()
        for n in range(N):
            th = n * math.radians(arc) / N
            s, co = math.sin(th), math.cos(th)
            u = ((hp + c) * (1.0 - s) - co * hp - 0.5) + s * jd + co * idd
            k = u.floor()
            f = (u - k)[:, None]
            k = (k.long() + 2).clamp(0, W + 2)
            acc += rows[n].index_select(0, k) * (1.0 - f)
            acc += rows[n].index_select(0, k + 1) * f
    else:
        # the flat array of all rows: a pixel near the rim may read the rows beside
        # its own, and 0 outside the sinogram
        flat = torch.zeros((N + 2, W, S), device="cuda", dtype=torch.float64)
        flat[1:N + 1] = q.permute(1, 2, 0)
        flat = flat.reshape((N + 2) * W, S)
        f32 = np.float32
        jc = j - float(f32(c))
        for n, (s, co) in enumerate(_table(arc, N)):
            base = f32(c) + ((f32(1) - s) - co) * f32(hp)
            t = (jc * float(s) + float(base)) + i * float(co)
            acc += flat.index_select(0, t.int().long() + (n + 1) * W)
    out = torch.zeros((S, W, W), device="cuda", dtype=torch.float64)
    out[:, jj, ii] = (acc / N).T
    return out


def _exact_fbp(x, case, contrast, arc, centers, interp=0):
    q = torch.stack([_filtered(s, case, contrast) for s in x])
    if len(centers) == 1:
        return _backproject(q, arc, float(np.float32(centers[0])), interp)
    return torch.cat([_backproject(q, arc, float(c), interp) for c in centers])


def _exact_ts(case, seed):
    n, rows, W = case["images"], case["rows"], case["width"]
    x = _phases(seed, n, rows, W, 180.0, 0.0)
    g = _window(W, case["filter"])
    f32 = np.float32
    rc = f32(W * 0.5 + float(f32(case["center"])))
    dx = torch.arange(W, device="cuda", dtype=torch.float32) - float(rc)
    out = torch.zeros((rows, W), device="cuda", dtype=torch.float64)
    for k, a in enumerate(_ts_angles(case)):
        sn, cs = f32(_sinf(a)), f32(_cosf(a))
        shift = (f32(case["plane"]) - f32(case["center"])) * sn
        di = (dx * float(cs) - float(shift)) + float(rc)
        di = torch.where(di < 0, torch.zeros_like(di),
                         torch.where(di >= W, torch.full_like(di, W - 1), di))
        y = torch.fft.irfft(torch.fft.rfft(x[k].double()) * g, n=W)
        out += y.index_select(1, di.int().long())
    return out


def _conv64(x, w, b):
    return torch.nn.functional.conv2d(x, w, b, padding=1)


def _exact_unet(case, seed, scale=2.0):
    p, o, ws = torch.from_numpy(_unet_params(seed)).cuda().double(), 0, []
    for ci, co in UNET:
        w = p[o:o + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous()
        o += co * 9 * ci
        ws.append((w, p[o:o + co]))
        o += co
    head, bias = p[o:o + HEAD], p[o + HEAD]
    pool = torch.nn.functional.max_pool2d

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3)

    def net(x):
        def c(t, k):
            return _conv64(t, *ws[k]).relu_()
        xs = torch.zeros((1, 16) + tuple(x.shape), device="cuda", dtype=torch.float64)
        xs[:, 0] = x * scale
        s1 = c(c(xs, 0), 1)
        s2 = c(c(pool(s1, 2), 2), 3)
        s3 = c(c(pool(s2, 2), 4), 5)
        t = c(c(pool(s3, 2), 6), 7)
        t = c(c(torch.cat([up(t), s3], 1), 8), 9)
        t = c(c(torch.cat([up(t), s2], 1), 10), 11)
        t = c(c(torch.cat([up(t), s1], 1), 12), 13)
        return x + (torch.einsum("bchw,c->hw", t, head) + bias) / scale

    with torch.no_grad():
        return torch.stack([net(x.double()) for x in _unet_input(case, seed)])


def _exact_conv(case, seed):
    x, w, b, dy = _conv_input(case, seed)
    B, H, W, ci = x.shape
    co = w.shape[0]
    w4 = w.double().reshape(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous()
    w4t = w4.flip(2, 3).transpose(0, 1).contiguous()
    y = torch.empty(dy.shape, device="cuda", dtype=torch.float64)
    dx = torch.empty(x.shape, device="cuda", dtype=torch.float64)
    dw = torch.zeros((co, 9, ci), device="cuda", dtype=torch.float64)
    for k in range(B):
        xk, dk = x[k].double(), dy[k].double()
        y[k] = _conv64(xk.permute(2, 0, 1)[None], w4, b.double())[0].relu_().permute(1, 2, 0)
        dx[k] = _conv64(dk.permute(2, 0, 1)[None], w4t, None)[0].permute(1, 2, 0)
        xp = torch.nn.functional.pad(xk, (0, 0, 1, 1, 1, 1))
        d2 = dk.reshape(-1, co)
        for t in range(9):
            dw[:, t] += d2.T @ xp[t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, ci)
    return {"y": y, "dx": dx, "dw": dw}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("stack", "host"):
        return _exact_fbp(_stack_input(case, seed), case, case["contrast"], case["arc"],
                          [case["center"]], case["interp"])
    if kind == "axis":
        x = _phases(seed, 1, case["angles"], case["width"], 180.0, 0.0)
        return _exact_fbp(x, case, "PHS", 180.0, _axis_centers(case))
    if kind == "batch":
        return [_exact_fbp(_phases(seed + 1000 * k, 1, N, W, 180.0, c),
                           {"pad": 0, "filter": case["filter"]}, "PHS", 180.0, [c])[0]
                for k, (N, W, c) in enumerate(_batch_jobs(case))]
    if kind == "ts":
        return _exact_ts(case, seed)
    if kind == "unet":
        return _exact_unet(case, seed)
    return _exact_conv(case, seed)
