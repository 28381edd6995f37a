"""bench.py where the reference library is not built: the reference arm says so in its
one line and exits 0, on every machine and without touching a device."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif((ROOT / "oracle" / "_ref" / "libmipx_pdlp_ref.so").exists(), reason="the reference library is built")
def test_reference_arm_says_unavailable():
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "1"],
                         capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
    assert "value" not in line
