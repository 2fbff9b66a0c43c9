"""The autotuner's choice is shared by launches of one kernel form and fill only."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(not shutil.which("g++") or
                    not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                    reason="g++ or the CUDA headers are missing")
def test_tune_key_separates_forms(tmp_path):
    exe = str(tmp_path / "tune_key")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "cpp", "tune_key.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("S,arc", [(4, 180.0), (4, 360.0), (1, 180.0)])
def test_untuned_launch_under_capture(S, arc):
    """A graph capture of single slices on a handle whose only earlier call was a stack
    in four-slice groups, which tunes no tile: captured and replayed, not refused."""
    import numpy as np
    import torch

    from ctas_b200 import _lib, ct
    N, W, c = 67, 331, 1.25                 # a shape no other test tunes
    x = torch.from_numpy(np.random.default_rng(4).standard_normal((S, N, W)).astype(np.float32)).cuda()
    y = torch.empty((S, W, W), device="cuda")
    one = torch.full((W, W), float("nan"), device="cuda")
    with ct.CTrec((N, W), ct.Contrast.PHS, arc, flags=_lib.FLAG_GROUPS) as rec:
        rec.reconstruct_stack_dev(x, y, c)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            rec.reconstruct_dev(x[0], one, c)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(one.view(torch.int32), y[0].view(torch.int32))
        rec.synchronize()
