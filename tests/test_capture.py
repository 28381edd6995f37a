"""A launch that is refused while a graph is captured (csrc/capture.hpp): its error is
the capture's result, so no graph without the steps is run.  On the CPU, with a fake
of the failing call; and no capture elsewhere in the engine goes without it."""
import shutil
import subprocess
from pathlib import Path

import pytest

from mipx_b200 import build

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "mipx_b200" / "csrc"


def test_errors_of_a_capture(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    cuda = Path(build.nvcc()).resolve().parents[1] / "include"
    exe = tmp_path / "capture_test"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", f"-I{cuda}",
                    str(ROOT / "tests" / "cpp" / "capture_test.cpp"), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout


def test_every_capture_keeps_its_errors():
    users = [f.name for f in CSRC.iterdir() if f.is_file() and "cudaStreamBeginCapture" in f.read_text()]
    assert users == ["capture.hpp"]
