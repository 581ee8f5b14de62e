"""The film's byte of a colour value takes the gamma's power in single precision
and asks the double-precision one near the steps only.  For every float from
below the gamma's linear part's end to 1 the byte equals the double-precision
one, and without the second look a few would not."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from slr_gb300 import build

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.gpu
def test_every_value_has_the_double_precision_byte(tmp_path):
    so = tmp_path / "film_gamma.so"
    subprocess.run([str(build._cuda_home() / "bin" / "nvcc"), "-std=c++17", "-O3", *build.ARCH, "-shared", "-Xcompiler",
                    "-fPIC", "-o", str(so), str(ROOT / "tests" / "film_gamma.cu")], check=True, timeout=300)
    lib = C.CDLL(str(so))
    bits = lambda v: int(np.float32(v).view(np.uint32))  # noqa: E731
    counts = (C.c_ulonglong * 2)()
    assert lib.film_gamma_compare(C.c_uint32(bits(0.003)), C.c_uint32(bits(1.0)), counts) == 0
    assert counts[0] == 0
    assert counts[1] > 0      # the values around the steps are among those tried
