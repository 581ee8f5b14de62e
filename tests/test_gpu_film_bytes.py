"""BMP rows of films at the edges of the kernel's groups of 32 pixels, from
aligned and unaligned host arrays and from device memory, against the
same steps in numpy: single precision to the colour values, double precision
for the gamma.  Bytes agree except where the two libraries' exponentials
differ in the last bit at an 8-bit step (at most 1 apart on at most 0.1 % of
the bytes, or one byte of a small film); the gamma's steps themselves are covered by a film that
sweeps every byte value."""
import ctypes as C

import numpy as np
import pytest

from slr_gb300 import api

M = np.array([[3.2404542, -1.5371385, -0.4985314], [-0.9692660, 1.8760108, 0.0415560],
              [0.0556434, -0.2040259, 1.0572252]])


def _rows(film, scale):
    bins, integral = api.film_cmf()
    h, w = film.shape[:2]
    xyz = np.zeros((h, w, 3), np.float32)
    for b in range(16):
        v = film[..., b] * np.float32(scale)
        for c in range(3):
            xyz[..., c] += bins[c, b] * v
    xyz /= np.float32(integral)
    rgb = np.maximum((xyz.astype(np.float64) @ M.T).astype(np.float32), 0)
    v = np.float32(1) - np.exp(-rgb)
    g = np.where(v <= 0.0031308, 12.92 * v.astype(np.float64),
                 1.055 * np.power(v.astype(np.float64), 1 / 2.4) - 0.055).astype(np.float32)
    px = np.minimum(255, (np.float32(256) * g).astype(np.uint32)).astype(np.uint8)
    out = np.zeros((h, 3 * w + w % 4), np.uint8)
    out[:, :3 * w] = px[::-1, :, ::-1].reshape(h, 3 * w)
    return out


def _check(got, want):
    d = np.abs(got.astype(int) - want.astype(int))
    assert d.max() <= 1 and (d > 0).sum() <= max(1, 1e-3 * d.size)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (32, 1), (33, 1), (5, 13), (64, 9), (203, 77)])
def test_rows_of_host_and_device_films(w, h):
    import torch
    rng = np.random.default_rng(w + h)
    film = np.exp(rng.normal(-1.0, 1.5, (h, w, 16))).astype(np.float32)
    want = _rows(film, 0.3)
    got = api.film_to_bmp(film, 0.3)
    _check(got, want)
    store = np.zeros(film.size + 1, np.float32)     # a film 4 bytes past an aligned address
    store[1:] = film.ravel()
    off = store[1:].reshape(film.shape)
    assert off.ctypes.data % 16 != film.ctypes.data % 16 or film.ctypes.data % 16 != 0
    assert np.array_equal(api.film_to_bmp(off, 0.3), got)
    dev = torch.from_numpy(film).cuda()
    px = np.full_like(got, 7)
    api.check(api.lib().slrgpu_film_to_bmp(C.cast(dev.data_ptr(), C.POINTER(C.c_float)), w, h, 1, 0.3, 1.0,
                                           px.ctypes.data_as(C.POINTER(C.c_uint8)), None))
    assert np.array_equal(px, got)


@pytest.mark.gpu
def test_every_byte_value():
    """A grey ramp through all 256 steps in both branches of the gamma."""
    ramp = np.linspace(0.0, 24.0, 512 * 64, dtype=np.float32) ** 2 / 64
    film = np.repeat(ramp[:, None], 16, 1).reshape(64, 512, 16)
    got, want = api.film_to_bmp(film, 1.0), _rows(film, 1.0)
    _check(got, want)
    assert len(np.unique(got)) >= 250
