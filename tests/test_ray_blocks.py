"""The arithmetic by which a ray query's blocks and warps take their rays, on the
host: a cursor that counted in ray numbers went past 2^32 for query sizes
within 256 of it, and its block then took other blocks' rays."""
import shutil
import subprocess
from pathlib import Path

import pytest


def test_every_ray_is_taken_once_up_to_the_largest_query(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "ray_blocks"
    subprocess.run([cxx, "-std=c++17", "-O2", "-o", str(exe), str(Path(__file__).with_name("ray_blocks.cpp"))], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout
