"""The kernels that a batch plan chooses by sizes alone. The check is a small host
program (tests/plan_choices_check.cu) compiled against the package's headers and
linked to the built library; it runs on the CPU."""
import os
import shutil
import subprocess
import tempfile
from pathlib import Path

import pytest

from crossstage_stitch_b200 import build as native

ROOT = Path(__file__).resolve().parents[1]


def test_plan_choices():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    lib = native.build()
    with tempfile.TemporaryDirectory() as d:
        exe = Path(d) / "plan_choices_check"
        cmd = [nvcc, *native.ARCH, "-std=c++17", "-O1", "-I", str(native.CSRC), "-I", str(native.INCLUDE),
               str(ROOT / "tests" / "plan_choices_check.cu"), str(lib), "-o", str(exe), "-Xlinker", f"-rpath={lib.parent}"]
        built = subprocess.run(cmd, capture_output=True, text=True)
        assert built.returncode == 0, built.stderr[-4000:]
        out = subprocess.run([str(exe)], capture_output=True, text=True, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
        assert out.returncode == 0 and "plan choices ok" in out.stdout, (out.returncode, out.stdout, out.stderr)
