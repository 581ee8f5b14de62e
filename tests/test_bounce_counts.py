"""The host's wait for the sizes of a wave's bounces, on the host against a
scripted CUDA runtime: which counts it takes, that the cause of a refused launch
is what it returns and that no error stays pending, that a stream which has run
dry ends it, and that there is none on devices whose waiting threads sleep."""
import shutil
import subprocess
from pathlib import Path

import pytest

from slr_gb300 import build

ROOT = Path(__file__).resolve().parents[1]


def test_wait_for_a_bounce(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "bounce_counts"
    subprocess.run([cxx, "-std=c++17", "-O2", f"-I{build._cuda_home() / 'include'}", "-o", str(exe),
                    str(ROOT / "tests" / "bounce_counts.cpp"), str(ROOT / "slr_gb300" / "csrc" / "bounce_counts.cpp")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
