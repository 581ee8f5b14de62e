"""The bidirectional tracer's kernels for scenes of Lambert materials alone
against the ones for any material: the same box, once as it is and once with a
mirror among its materials that no mesh uses, gives the same paths and the same
film to rounding."""
import numpy as np
import pytest

from slr_gb300 import api, scenes
from slr_gb300.scene_desc import REFLECTANCE


def _desc(medium, unused, w, h):
    d = scenes.medium_box_scene(w, h, grid=16) if medium else scenes.box_scene(w, h)
    if unused:
        d.material("specular_reflection", (d.spectrum_rgb(REFLECTANCE, 0.9, 0.9, 0.9), d.spectrum_regular([0.2, 0.2]),
                                           d.spectrum_regular([3.0, 3.0])))
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("medium", [False, True])
@pytest.mark.parametrize("width,height,spp,depth", [(1, 1, 1, 1), (8, 8, 3, 2), (33, 17, 4, 9), (96, 64, 2, 16)])
def test_lambert_scenes_take_the_same_paths(medium, width, height, spp, depth):
    """Contributions are summed by atomics: a bin's sum is reproducible to a few
    units in the last place, and the two instances' expressions may round apart
    once per vertex (bar 2e-5 of the larger of the value and the film's root
    mean square)."""
    films, stats = [], []
    for unused in (False, True):
        film, st = api.Scene(_desc(medium, unused, width, height)).render(width, height, spp, depth, seed=4,
                                                                          volumetric=medium, bpt=True)
        films.append(film.astype(np.float64))
        stats.append((st.extension_rays, st.shadow_rays, st.dropped_samples))
    assert stats[0] == stats[1] and np.isfinite(films[0]).all()
    # vertices in one plane connect with an invalid weight, which is no dropped sample
    assert medium or stats[0][2] == 0
    rms = np.sqrt((films[1] ** 2).mean())
    assert np.all(np.abs(films[0] - films[1]) <= 2e-5 * np.maximum(np.abs(films[1]), rms))
