"""The film kernel and the path order of a wave: a frame is the same bits
whatever its split into waves (one sample of the whole grid at a time, some,
or all), on images that end inside a sensor tile, are smaller than one, or
fill whole tiles, and in a resumed render."""
import numpy as np
import pytest

from slr_gb300 import api, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,spp", [(1, 1, 5), (7, 9, 4), (8, 8, 33), (9, 17, 6), (40, 24, 3)])
def test_film_is_the_same_for_every_wave_split(width, height, spp):
    scene = api.Scene(scenes.glossy_box_scene(width, height))
    whole, st = scene.render(width, height, spp, 6, seed=3)
    assert st.path_samples == (width + 7) // 8 * 8 * ((height + 7) // 8 * 8) * spp
    assert np.isfinite(whole).all() and whole.sum() > 0
    for per_wave in (1, 2, spp - 1):
        film, other = scene.render(width, height, spp, 6, seed=3, samples_per_wave=per_wave)
        assert np.array_equal(film, whole)
        assert other.dropped_samples == st.dropped_samples
    c = api.FilmCheckpoint(width, height, 6, seed=3)
    for n in (1, spp - 1):
        film, _ = scene.render_continue(c, n)
    assert np.array_equal(film, whole) and np.array_equal(c.film(), whole)
