"""The rule that sends slices of a stack through the four-slice kernel
(bp_quad_rule.hpp), compiled for the host: against measured times, and the bounds that
the work buffers are sized by."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# backprojection of slices of width x width at 720 projections on 148 SMs, us: one slice
# at a time; whole groups and the rest so; all in groups
MEASURED = [  # form, width, slices
    (0, 228, 4, 99, 158, 158),
    (0, 324, 9, 168, 257, 211),
    (0, 324, 10, 170, 256, 211),
    (0, 342, 9, 166, 258, 211),
    (0, 364, 8, 168, 160, 160),
    (0, 408, 4, 168, 158, 158),
    (0, 408, 9, 256, 310, 215),
    (0, 408, 10, 271, 310, 215),
    (0, 432, 9, 256, 310, 211),
    (0, 458, 8, 277, 215, 215),
    (0, 514, 6, 254, 320, 211),
    (0, 544, 6, 254, 339, 215),
    (0, 576, 3, 166, None, 211),
    (0, 576, 5, 258, 312, 219),
    (0, 576, 6, 283, 377, 219),
    (0, 612, 3, 168, None, 212),
    (0, 612, 6, 299, 380, 381),
    (0, 612, 10, 469, 549, 343),
    (0, 648, 3, 252, None, 211),
    (0, 866, 3, 299, None, 381),
    (0, 866, 12, 1043, 668, 668),
    (0, 1636, 5, 1411, 998, 1350),
    (1, 204, 9, 127, 320, 193),
    (1, 306, 3, 127, None, 191),
    (1, 324, 9, 195, 316, 248),
    (1, 342, 9, 193, 318, 252),
    (1, 408, 9, 330, 374, 252),
    (1, 514, 6, 328, 379, 250),
    (1, 544, 6, 328, 396, 250),
    (1, 576, 3, 191, None, 246),
    (1, 576, 6, 332, 433, 255),
    (1, 576, 11, 553, 445, 396),
    (1, 612, 3, 189, None, 248),
    (1, 612, 5, 330, 374, 451),
    (1, 612, 6, 365, 437, 451),
    (1, 612, 10, 560, 640, 441),
    (1, 866, 3, 345, None, 447),
    (1, 866, 5, 529, 634, 689),
    (1, 866, 6, 643, 773, 689),
    (1, 1024, 3, 449, None, 386),
    (1, 1224, 3, 617, None, 699),
    (1, 1376, 9, 2063, 1570, 1903),
    (1, 1536, 7, 1948, 1635, 1582),
    (1, 2600, 3, 2354, None, 2272),
    (2, 192, 3, 240, None, 238),
    (2, 192, 4, 240, 238, 238),
    (2, 192, 5, 240, 478, 240),
    (2, 204, 7, 240, 484, 244),
    (2, 288, 7, 406, 480, 240),
    (2, 408, 8, 668, 363, 363),
    (2, 484, 11, 1114, 836, 653),
    (2, 514, 3, 473, None, 240),
    (2, 544, 6, 707, 507, 365),
    (2, 1024, 8, 2912, 1170, 1170),
    (2, 2062, 7, 9692, 6182, 4463),
]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ is missing")
    exe = str(tmp_path_factory.mktemp("rule") / "quad_rule")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(ROOT, "tests", "cpp", "quad_rule.cpp"),
                    "-o", exe], check=True)

    def ask(cases):
        out = subprocess.run([exe], input="\n".join("%d %d %d %d" % c for c in cases), text=True,
                             capture_output=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return ask


def test_no_choice_slower_than_single_slices(rule):
    """The chosen way's measured time is at most 2 % above one slice at a time."""
    for (f, W, S, single, part, whole), (n, *_) in zip(
            MEASURED, rule([(f, W, S, 148) for f, W, S, *_ in MEASURED])):
        us = single if n == 0 else whole if n == S else part
        assert us <= 1.02 * single, (f, W, S, n)


def test_main_stacks_are_grouped(rule):
    """The stacks the kernel was made for keep their groups."""
    want = {(0, 2560, 32): 32, (0, 2560, 16): 16, (0, 1023, 5): 4, (1, 2560, 6): 4,
            (2, 1536, 4): 4, (0, 4096, 8): 8, (0, 2560, 256): 256, (0, 2560, 4): 4}
    for n, got in zip(want.values(), rule([k + (148,) for k in want])):
        assert got[0] == n


def test_tiles_hold_the_disc(rule):
    for W in (2, 5, 63, 64, 65, 200, 1023):
        (_, all64, in64, in32, _), = rule([(0, W, 1, 148)])
        hp = W // 2
        y, x = np.mgrid[:W, :W] - hp
        disc = y * y + x * x < hp * hp
        assert all64 == (-(-W // 64)) ** 2
        for ty, got in ((64, in64), (32, in32)):
            n = sum(disc[j:j + ty, i:i + 64].any() for j in range(0, W, ty) for i in range(0, W, 64))
            assert got == n, (W, ty)


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("sms", [148, 132, 16])
def test_rest_stays_below_four_where_groups_always_pay(rule, form, sms):
    """Counts are 0, all or all but a rest below four, and not 0 beyond the count up to
    which buffers are sized one by one."""
    for W in (2, 64, 300, 700, 1500, 4000):
        always = rule([(form, W, 1, sms)])[0][4]
        counts = list(range(1, min(always, 400))) + list(range(always + 1, always + 40))
        for S, (n, *_) in zip(counts, rule([(form, W, S, sms) for S in counts])):
            assert n in (0, S, S - S % 4) and (n == 0 or n >= 3)
            assert n > 0 or S <= max(always, 2)
