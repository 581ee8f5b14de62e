"""BMP rows into arrays whose pages nobody has touched: the same rows as into an
array in use, at sizes around one page and many, and from any offset in a
page; the bytes on either side of the array stay as they were."""
import ctypes as C
import mmap

import numpy as np
import pytest

from slr_gb300 import api


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1, 4095])
@pytest.mark.parametrize("w,h", [(1, 1), (36, 37), (44, 31), (148, 148), (333, 217)])
def test_rows_in_untouched_pages(w, h, offset):
    rng = np.random.default_rng(w)
    film = np.exp(rng.normal(-1.0, 1.0, (h, w, 16))).astype(np.float32)
    n = (3 * w + w % 4) * h
    want = api.film_to_bmp(film, 0.5).ravel()
    with_guard = np.frombuffer(mmap.mmap(-1, offset + n + 4096), np.uint8)
    px = with_guard[offset:offset + n]
    api.check(api.lib().slrgpu_film_to_bmp(film.ctypes.data_as(C.POINTER(C.c_float)), w, h, 0, 0.5, 1.0,
                                           px.ctypes.data_as(C.POINTER(C.c_uint8)), None))
    assert np.array_equal(px, want)
    assert not with_guard[:offset].any() and not with_guard[offset + n:].any()
