"""Every call works on each GPU of one process, and after a device reset: the
kernels that need more shared memory than a launch may have by default are opted in
in every context, whether the driver gives contexts an id or not. The check (tests/multi_device_check.cpp) links the built objects to a CUDA
runtime of its own and runs on the CPU."""
import shutil
import subprocess
import tempfile
from pathlib import Path

import pytest

from crossstage_stitch_b200 import build as native

ROOT = Path(__file__).resolve().parents[1]


def test_calls_on_every_device_of_a_process():
    nvcc, gxx = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", shutil.which("g++")
    if not Path(nvcc).exists() or not gxx:
        pytest.skip("compilers not available")
    native.build()
    with tempfile.TemporaryDirectory() as d:
        exe = Path(d) / "multi_device_check"
        cmd = [gxx, "-std=c++17", "-O1", "-I", str(native.INCLUDE), "-I", str(Path(nvcc).resolve().parents[1] / "include"),
               str(ROOT / "tests" / "multi_device_check.cpp"), *[str(native.BUILD / (s.stem + ".o")) for s in native.sources()],
               "-pthread", "-o", str(exe)]
        built = subprocess.run(cmd, capture_output=True, text=True)
        assert built.returncode == 0, built.stderr[-4000:]
        for ids in ([], ["ids"]):
            out = subprocess.run([str(exe), *ids], capture_output=True, text=True, timeout=120)
            assert out.returncode == 0, (out.returncode, out.stdout, out.stderr)
            assert "devices ok" in out.stdout
