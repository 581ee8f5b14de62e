"""BMP rows of films that just fit the library's array for small images and that
just do not, and from several threads at once, one of which has the array: the
rows of each film are its own."""
import threading

import numpy as np
import pytest

from slr_gb300 import api

SCRATCH = (2 << 20) + (256 << 10)


def _need(w, h):
    return (w * h * 64 + 255) // 256 * 256 + (3 * w + w % 4) * h


def _film(w, h, seed):
    return np.exp(np.random.default_rng(seed).normal(-1.0, 1.0, (h, w, 16))).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("w", [1, 36, 127, 736])
def test_films_around_the_array_size(w):
    """Each film's rows against those of its halves, which are small."""
    h = next(h for h in range(1, 1 << 16) if _need(w, h + 1) > SCRATCH)
    assert _need(w, h) <= SCRATCH
    for k in (h, h + 1):
        film = _film(w, k, k)
        rows = api.film_to_bmp(film, 0.5)
        assert np.array_equal(rows[k - k // 2:], api.film_to_bmp(film[:k // 2], 0.5))     # bottom up
        assert np.array_equal(rows[:k - k // 2], api.film_to_bmp(film[k // 2:], 0.5))


@pytest.mark.gpu
def test_threads_do_not_share_the_array():
    sizes = [(33, 33), (200, 150), (736, 44), (64, 300), (400, 300), (101, 77)]
    films = [_film(w, h, w) for w, h in sizes]
    want = [api.film_to_bmp(f, 0.5) for f in films]
    bad = []

    def work(k):
        for _ in range(40):
            if not np.array_equal(api.film_to_bmp(films[k], 0.5), want[k]):
                bad.append(sizes[k])
                return

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
