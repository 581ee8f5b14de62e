"""bench.py where the reference renderer is not built: the reference arm says so
in one line and succeeds, and the GPU arm's CPU baseline says so in its place
instead of losing the finished line."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

from oracle import oracle as O

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture
def no_reference(monkeypatch):
    monkeypatch.setattr(O, "TIMING_LIB_PATH", ROOT / "oracle" / "no_such_library.so")


def test_reference_arm_says_why():
    if O.TIMING_LIB_PATH.is_file():
        pytest.skip("the reference renderer is built here")
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "3"], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "not built" in line["unavailable"]


def test_cpu_baseline_says_why(no_reference):
    import bench
    assert "not built" in bench.cpu_baseline(None, 1)["unavailable"]
