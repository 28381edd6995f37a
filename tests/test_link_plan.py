"""The rule that takes an LP's steps to the linked restart cycle (csrc/link_plan.hpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_rule(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "link_plan_test"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'mipx_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "link_plan_test.cpp"), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout
