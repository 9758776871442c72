"""The quotients that stand for divisions must be the divisions' results bit for
bit: a small CUDA program built with the library's flags compares them on 2^28
operands. (That they are follows from Markstein's theorem; this checks the code.)"""
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


def test_quotients_equal_division(cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "quotient_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-fmad=false", "-std=c++17",
                    "-I", str(HERE.parent / "crossstage_stitch_b200" / "csrc"), str(HERE / "gpu_quotient_check.cu"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=120).stdout
    assert out.split() == ["operands", str(1 << 28), "quotient", "0", "over255", "0"], out


@pytest.mark.parametrize("snap", [0.0, 1e-15, 1e-10, 0.4])
@pytest.mark.parametrize("h", [[1, 0, 3.25, 0, 1, -2.5, 0, 0, 1], [0.9, 0.1, 4, -0.1, 1.1, 3, 2e-4, -1e-4, 1],
                               [1, 0, 1e-140, 0, 1, 1e-200, 0, 0, 1], [1, 0, 2, 0, 1, 1, 0, 0, 1]])
def test_render_snap_and_range(cuda, snap, h):
    """The render where the snap tolerance is, and is not, the larger bound, and
    where a projection leaves the range of the corrected quotients."""
    import numpy as np
    import torch

    from crossstage_stitch_b200 import render
    from oracle import c_oracle
    rng = np.random.default_rng(3)
    a, b = (rng.integers(0, 256, (37, 53, 3), dtype=np.uint8) for _ in range(2))
    p = render.default_policy()
    p.snap_tolerance = snap
    g = render.prepare_geometry(53, 37, 53, 37, h, p)
    pano, mask = render.render(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), g)
    op = c_oracle.s6_policy()
    op.snap_tol = snap
    st, og = c_oracle.s6_geometry(53, 37, 53, 37, h, op)
    opano, omask, _ = c_oracle.s6_feather(a, b, og)
    assert st == 0 and np.array_equal(pano.cpu().numpy(), opano) and np.array_equal(mask.cpu().numpy(), omask)
