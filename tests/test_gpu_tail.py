"""Waves at and around the line below which the tail kernel takes the paths:
the film of a frame traced by bounce kernels (all samples in one wave) and by
the tail kernel alone (one sample of the grid per wave) agree, and the queue
counters account for every ray on both sides."""
import numpy as np
import pytest

from slr_gb300 import api, scenes


def _scene(name, w, h):
    if name == "box":
        return scenes.box_scene(w, h)
    return scenes.heightfield_scene(grid=24, spheres=4, sphere_freq=3, env_size=(64, 32), width=w, height=h, seed=2)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["box", "terrain"])
@pytest.mark.parametrize("width,height,spp", [(8, 8, 1), (64, 64, 1), (64, 64, 2), (72, 64, 1), (40, 48, 12)])
def test_tail_and_bounce_kernels_trace_the_same_paths(name, width, height, spp):
    """Waves of 64, 4096 (the line), 4608 and up to 23040 paths.  The two sides
    evaluate the same expressions, compiled twice: a throughput may differ by a
    few units in the last place per vertex (bar 2e-5 of the larger of the value
    and the film's root mean square, 300 roundings)."""
    ctx = api.Context(0)
    scene = api.Scene(_scene(name, width, height), context=ctx)
    try:
        film, st = scene.render(width, height, spp, 9, seed=11)
        q = ctx.queue_counts().astype(np.int64)
        assert q[0, 7] == width * height * spp
        assert q[:, 7].sum() == st.extension_rays and q[:, 8].sum() == st.shadow_rays
        assert q[0, 0:6].sum() == q[0, 7] and q[10:, :].sum() == 0
        for b in range(1, 10):
            assert q[b, 0:6].sum() <= q[b, 7] <= q[b - 1, 0:5].sum() and q[b, 8] <= q[b, 0:5].sum()
        split, st1 = scene.render(width, height, spp, 9, seed=11, samples_per_wave=1)
        assert st1.extension_rays == st.extension_rays and st1.shadow_rays == st.shadow_rays
        rms = float(np.sqrt((film.astype(np.float64) ** 2).mean()))
        assert np.all(np.abs(split - film) <= 2e-5 * np.maximum(np.abs(film), rms))
    finally:
        scene.close()
        ctx.close()
