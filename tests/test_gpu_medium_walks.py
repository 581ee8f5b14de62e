"""Transmittance walks at the edges of their work distribution: a frame of a
medium is the same bits whether its shadow rays reach the kernel as one queue or
in waves of one sample (queues of a few rays, below a warp's refill, up to
many chunks), on the smallest grids and on sizes that are no multiple of a
super voxel."""
import numpy as np
import pytest

from slr_gb300 import api, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [2, 5, 16, 67])
@pytest.mark.parametrize("width,height,spp", [(1, 1, 3), (8, 8, 2), (33, 17, 5)])
def test_volumetric_film_is_the_same_for_every_queue_length(grid, width, height, spp):
    desc = scenes.medium_box_scene(width, height, grid=8)
    rng = np.random.default_rng(grid)
    desc.medium.density = rng.random((grid, grid, grid), np.float32)
    scene = api.Scene(desc)
    whole, st = scene.render(width, height, spp, 20, seed=5, volumetric=True)
    assert np.isfinite(whole).all() and st.shadow_rays > 0
    film, other = scene.render(width, height, spp, 20, seed=5, volumetric=True, samples_per_wave=1)
    assert np.array_equal(film, whole)
    assert (other.extension_rays, other.shadow_rays) == (st.extension_rays, st.shadow_rays)
