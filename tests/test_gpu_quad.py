"""Stacks through the four-slice backprojection kernel: bit-identical to the
oracle's restatement of the reference arithmetic (backprojection of given rows)
and to the per-slice call (filtered rows included), over group remainders, odd
sizes, arcs, angle orders, output geometries and both index rules."""
import numpy as np
import pytest

import oracle as O
from ctas_b200 import _lib, ct

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _rows(S, N, W, seed):
    return np.random.default_rng(seed).standard_normal((S, N, W)).astype(np.float32)


@pytest.mark.parametrize("checked", [True, False])
@pytest.mark.parametrize("S,N,W,c,arc,rule", [
    (3, 37, 300, -4.25, 180.0, "ctcl"), (3, 32, 257, 0.0, 180.0, "shipped"),
    (4, 180, 64, 1.5, 180.0, "ctcl"), (5, 97, 96, -30.75, 180.0, "ctcl"),
    (4, 1, 33, 0.0, 180.0, "ctcl"), (7, 33, 5, 0.5, 180.0, "ctcl"), (3, 3, 2, 0.0, 180.0, "ctcl"),
    (6, 200, 300, -4.25, 360.0, "ctcl"), (3, 90, 200, -90.25, 360.0, "shipped"),
    (4, 61, 97, 2.0, 270.0, "ctcl"), (8, 48, 1290, 7.5, 180.0, "ctcl"),
    (4, 65, 1501, -3.25, 360.0, "ctcl")])
def test_stack_bitexact(S, N, W, c, arc, rule, checked):
    """Both tiles (the large one from 222 tiles of 64 x 64 on: 8 x 1290, 4 x 1501)."""
    q = _rows(S, N, W, 17 * S + W)
    tab = O.angle_table(arc, N)
    with ct.CTrec((N, W), ct.Contrast.FLT, arc, index_rule=rule, checked=checked,
                  flags=_lib.FLAG_GROUPS) as rec:
        got = rec.reconstruct_stack(q.copy(), None, c)
        assert rec.last_tile() == -1 or S % 4 in (1, 2)
    for s in range(S):
        assert np.array_equal(_bits(got[s]), _bits(O.bp_compat(q[s], tab, c, 1.0, rule=rule))), s


@pytest.mark.parametrize("S,W", [(11, 300), (12, 300), (3, 512), (4, 512), (10, 160)])
def test_size_rule(S, W):
    """Around the number of tiles from which groups are formed (four slices at 512 x 512,
    three groups at 300 x 300): the same bits on either side, in stacks whose chunks
    lie on both (device call: one chunk; host call: several)."""
    N, c = 40, 1.25
    q = _rows(S, N, W, S)
    tab = O.angle_table(180.0, N)
    want = [_bits(O.bp_compat(x, tab, c, 1.0)) for x in q]
    import torch
    with ct.CTrec((N, W), ct.Contrast.FLT, 180.0) as rec:
        d = torch.full((S, W, W), float("nan"), device="cuda")
        for n in (S, 2, S, 1, 3, S - 1):
            rec.reconstruct_stack_dev(torch.from_numpy(q[:n]).cuda(), d[:n], c)
            got = d.cpu().numpy()
            assert all(np.array_equal(_bits(got[s]), want[s]) for s in range(n)), n
        got = rec.reconstruct_stack(q.copy(), None, c)
    assert all(np.array_equal(_bits(got[s]), want[s]) for s in range(S))


@pytest.mark.parametrize("checked", [True, False])
@pytest.mark.parametrize("order", ["golden", "random", "reversed", "steps"])
def test_angle_orders_bitexact(order, checked):
    """Angle lists in which neighbouring projections differ: the pixel layout
    changes often, or fits only some projections of a chunk."""
    N, W, S, c = 150, 180, 4, 2.25
    th = {"golden": (np.arange(N) * 2.399963229728653) % np.pi,
          "random": np.random.default_rng(5).uniform(0, np.pi, N),
          "reversed": np.linspace(0, np.pi, N, endpoint=False)[::-1],
          "steps": np.where(np.arange(N) // 20 % 2 == 0, 0.05, 1.5)}[order]
    q = _rows(S, N, W, 3)
    with ct.CTrec((N, W), ct.Contrast.FLT, angles=th, checked=checked,
                  flags=_lib.FLAG_GROUPS) as rec:
        got = rec.reconstruct_stack(q.copy(), None, c)
    tab = O.angle_table_list(th)
    for s in range(S):
        assert np.array_equal(_bits(got[s]), _bits(O.bp_compat(q[s], tab, c, 1.0))), s


@pytest.mark.parametrize("rows,cols,pixel,shift", [(100, 77, 0.61, (3.5, -8.0)),
                                                   (65, 310, 1.0, (-40.0, 12.5))])
def test_output_geometry_bitexact(rows, cols, pixel, shift):
    N, W, S, c = 64, 220, 4, 1.25
    q = _rows(S, N, W, 9)
    with ct.CTrec((N, W), ct.Contrast.FLT, out_shape=(rows, cols), out_pixel=pixel,
                  out_shift=shift, checked=True, flags=_lib.FLAG_GROUPS) as rec:
        got = rec.reconstruct_stack(q.copy(), None, c)
    oj, oi, p = O.geometry(W, rows, cols, pixel, *shift)
    for s in range(S):
        want = O.bp_compat_geom(q[s], O.angle_table(180.0, N), c, 1.0, rows, cols, oj, oi, p)
        assert np.array_equal(_bits(got[s]), _bits(want)), s


@pytest.mark.parametrize("contrast,arc,ring", [("PHS", 180.0, 0), ("REF", 180.0, 3),
                                               ("ABS", 180.0, 2), ("PHS", 360.0, 0),
                                               ("FLT", 180.0, 4)])
def test_stack_equals_single_calls(contrast, arc, ring):
    """Filter and backprojection of a stack, both host and device forms, against
    one call per slice; the filtered rows written back included."""
    import torch
    S, N, W, c = 11, 91, 190, -2.5
    x = np.random.default_rng(2).uniform(0.2, 1.0, (S, N, W)).astype(np.float32)
    with ct.CTrec((N, W), getattr(ct.Contrast, contrast), arc, ct.Filter("HANN"),
                  ring_box=ring, flags=_lib.FLAG_GROUPS) as rec:
        rec.setPhysics(1e-6, 0.0)
        back = x.copy()
        single = np.stack([rec.reconstruct(back[s], None, c) for s in range(S)])
        for n in (2, 3, 4, 5, 11):
            y = x[:n].copy()
            got = rec.reconstruct_stack(y, None, c)
            assert np.array_equal(_bits(got), _bits(single[:n])), n
            assert np.array_equal(_bits(y), _bits(back[:n])), n
            d = torch.full((n, W, W), float("nan"), device="cuda")
            rec.reconstruct_stack_dev(torch.from_numpy(x[:n]).cuda(), d, c)
            assert np.array_equal(_bits(d.cpu().numpy()), _bits(single[:n])), n
        # a single slice afterwards still serves repeat()
        rec.sino(x[0].copy())
        assert np.array_equal(_bits(rec.repeat(None, c)), _bits(single[0]))


@pytest.mark.parametrize("store", [1, 2])
@pytest.mark.parametrize("S,N,W", [(3, 40, 300), (7, 33, 97), (6, 64, 260)])
def test_16bit_stack_equals_single_calls(S, N, W, store):
    """Groups expanded from 16-bit rows: the bits of one call per slice, which converts
    the same samples in the one-slice kernel."""
    x = _rows(S, N, W, 5 * S)
    x[1, ::3] *= 1e-3                       # rows of other scales
    x[0, 5] = 0.0
    with ct.CTrec((N, W), ct.Contrast.PHS, 180.0, ct.Filter("HANN"), store=store,
                  flags=_lib.FLAG_GROUPS) as rec:
        back = x.copy()
        single = np.stack([rec.reconstruct(back[s], None, 1.5) for s in range(S)])
        y = x.copy()
        got = rec.reconstruct_stack(y, None, 1.5)
    assert np.array_equal(_bits(got), _bits(single))
    assert np.array_equal(_bits(y), _bits(back))


@pytest.mark.parametrize("checked", [True, False])
@pytest.mark.parametrize("S,N,W,c,store", [(3, 180, 256, 2.5, 0), (7, 33, 97, -30.25, 0),
                                           (4, 61, 300, 0.0, 0), (8, 40, 1290, -7.5, 0),
                                           (4, 90, 260, 1.25, 1), (4, 5, 33, 0.0, 0)])
def test_linear_stack_vs_fp64_oracle(S, N, W, c, store, checked):
    """Linear interpolation of given rows (FLT): within the one-slice kernel's bounds
    against FP64 (relative RMSE 1e-5 float32, 2e-3 float16), and 0 outside the disc."""
    x = np.linspace(-1, 1, W)
    q = np.stack([np.exp(-(3 * x + 0.1 * s) ** 2)[None] * (1 + 0.3 * np.sin(np.arange(N) + s))[:, None]
                  for s in range(S)]).astype(np.float32)
    tab = O.angle_table_f64(180.0, N)
    m = O.mask(W, c)
    with ct.CTrec((N, W), ct.Contrast.FLT, 180.0, interp=1, store=store, checked=checked,
                  flags=_lib.FLAG_GROUPS) as rec:
        got = rec.reconstruct_stack(q.copy(), None, c)
    for s in range(S):
        want = O.bp_linear(q[s].astype(np.float64), tab, c, 1.0)
        err = np.sqrt(np.mean((got[s][m] - want[m]) ** 2)) / np.sqrt(np.mean(want[m] ** 2))
        assert err <= (1e-5 if store == 0 else 2e-3), s
        assert (got[s][~m] == 0).all()


def test_waits_run_out_and_context_survives():
    N, W = 120, 256
    q = _rows(4, N, W, 7)

    def run(flags):
        with ct.CTrec((N, W), ct.Contrast.FLT, flags=flags | _lib.FLAG_GROUPS) as rec:
            return rec.reconstruct_stack(q.copy(), None, 0.5)

    before = run(0)
    with pytest.raises(ct.CtasError) as e:
        run(_lib.FLAG_TEST_TIMEOUT)
    assert e.value.code == _lib.E_TIMEOUT
    assert np.array_equal(_bits(before), _bits(run(0)))
