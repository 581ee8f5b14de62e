"""A film's bits do not depend on how its samples are split into waves, also
where the split decides which kernels shade a bounce (waves of few paths are
taken to their end by one kernel): every material kind alone among matte
walls, rough glass whose indices vary with the wavelength, and height fields of
rough conductors and dielectrics under an environment, rendered whole, in waves of 4096 paths, of three samples and as
a resumed film, and served beside larger requests."""
import numpy as np
import pytest

from slr_gb300 import api, scenes
from slr_gb300.scene_desc import REFLECTANCE

KINDS = ["matte", "specular_reflection", "specular_scattering", "microfacet_reflection", "microfacet_scattering"]
W, H, SPP, DEPTH = 64, 64, 16, 10


def _desc(name):
    if name == "dispersive":
        d = _desc("microfacet_scattering")
        outside = d.spectrum_regular(np.linspace(1.0, 1.02, 5).astype(np.float32), 360.0, 830.0)
        inside = d.spectrum_regular(np.linspace(1.7, 1.45, 5).astype(np.float32), 360.0, 830.0)
        glass = d.material("microfacet_scattering", (outside, inside), 0.1, 0.3)
        d.materials = [d.materials[glass] if m.kind == "microfacet_scattering" else m for m in d.materials]
        return d
    if name in KINDS:
        d = scenes.glossy_box_scene(W, H)
        d.materials = [m if m.kind in ("matte", "emitter", name) else d.materials[0] for m in d.materials]
        return d
    d = scenes.heightfield_scene(grid=64, spheres=8, sphere_freq=6, env_size=(128, 64), width=W, height=H,
                                 seed=int(name[7:] or 1) if name.startswith("terrain") else 1)
    if name == "conductors":
        matte = d.material("matte", (d.spectrum_rgb(REFLECTANCE, 0.7, 0.5, 0.3),))
        d.materials = [m if m.kind != "microfacet_scattering" else d.materials[matte] for m in d.materials]
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("name", KINDS + ["dispersive", "conductors", "terrain0", "terrain1", "terrain2", "terrain3"])
def test_film_does_not_depend_on_the_wave_split(name):
    scene = api.Scene(_desc(name))
    whole, st = scene.render(W, H, SPP, DEPTH, seed=5)
    assert np.isfinite(whole).all() and whole.sum() > 0
    for per_wave in (1, 3):      # 4096 paths a wave, all in the last kernel where the scene allows it; 12288
        film, other = scene.render(W, H, SPP, DEPTH, seed=5, samples_per_wave=per_wave)
        assert (other.extension_rays, other.shadow_rays) == (st.extension_rays, st.shadow_rays)
        assert np.array_equal(film, whole)
    c = api.FilmCheckpoint(W, H, DEPTH, seed=5)
    for n in (1, 2, SPP - 3):
        scene.render_continue(c, n)
    assert np.array_equal(c.film(), whole)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["microfacet_reflection", "terrain"])
def test_served_film_does_not_depend_on_its_company(name):
    """A request of 3072 paths that shares its waves with larger ones equals
    the standalone render, whose one wave is small enough for the last kernel."""
    scene = api.Scene(_desc(name))
    alone = [scene.render(48, 32, 2, DEPTH, seed=9 + k)[0] for k in range(4)]
    srv = api.Server(mode=api.SERVER_BATCHED, slots=1, paths_per_slot=1 << 16, max_depth=DEPTH)
    try:
        ids = [srv.submit(scene, 64, 64, 40, DEPTH, seed=1)]
        for k in range(4):
            ids += [srv.submit(scene, 48, 32, 2, DEPTH, seed=9 + k), srv.submit(scene, 64, 48, 8, DEPTH, seed=20 + k)]
        films = [srv.wait(i, timeout=120)[0] for i in ids]
        for k in range(4):
            assert np.array_equal(films[1 + 2 * k], alone[k])
    finally:
        srv.close()
