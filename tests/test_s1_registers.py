"""The kernels that run S1's float filter, which lives on resident warps, take at most 32
(per-image and per-pair) and 40 registers (batched): the runs of the integer modes,
which take 64, have a kernel of their own."""
import re
import subprocess
import tempfile
from pathlib import Path

import pytest

from crossstage_stitch_b200 import build as native


def test_float_filter_keeps_its_warps():
    try:
        nvcc = native.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    with tempfile.TemporaryDirectory() as d:
        out = subprocess.run([nvcc, *native.ARCH, *native.NVCC_FLAGS, "-Xptxas", "-v", "-c", str(native.CSRC / "s1.cu"),
                              "-o", str(Path(d) / "s1.o")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-4000:]
    used = {m[1]: int(m[2]) for m in re.finditer(r"entry function '(\w+)'.*?Used (\d+) registers", out.stderr, re.S)}
    per_call = [n for name, n in used.items() if "s1_kernel" in name]
    batched = [n for name, n in used.items() if "s1_batch_kernel" in name]
    assert min(per_call) <= 32 and max(batched) <= 40, used
