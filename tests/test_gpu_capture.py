"""The allocation-free render inside a stream capture: its kernels, which
overlap their neighbours, keep their order in a CUDA graph, whose replays give
slrgpu_render's film bit for bit.  Waves below and above the line of the tail
kernel, every material kind, and the volumetric tracer."""
import ctypes as C

import numpy as np
import pytest

from slr_gb300 import api, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("name,width,height,spp,depth", [("box", 40, 24, 2, 8), ("glossy", 96, 64, 4, 9),
                                                         ("medium", 64, 40, 3, 12), ("terrain", 96, 96, 3, 6)])
def test_captured_render_replays_the_film(name, width, height, spp, depth):
    import torch
    desc = {"box": lambda: scenes.box_scene(width, height),
            "glossy": lambda: scenes.glossy_box_scene(width, height),
            "medium": lambda: scenes.medium_box_scene(width, height, grid=24),
            "terrain": lambda: scenes.heightfield_scene(grid=24, spheres=4, sphere_freq=3, env_size=(64, 32),
                                                        width=width, height=height, seed=2)}[name]()
    scene = api.Scene(desc)
    vol = name == "medium"
    film = torch.zeros((height, width, 16), device="cuda")
    s = api.Settings(width, height, spp, depth, 9, int(vol), 0, 0)

    def call(stream):
        api.check(api.lib().slrgpu_render_noalloc(scene.handle, C.byref(s), C.c_void_p(film.data_ptr()),
                                                  C.c_void_p(stream.cuda_stream)))

    call(torch.cuda.current_stream())
    torch.cuda.synchronize()
    plain = film.cpu().numpy()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(torch.cuda.current_stream())
    for _ in range(3):
        film.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(film.cpu().numpy(), plain)
    want, _ = scene.render(width, height, spp, depth, seed=9, volumetric=vol, samples_per_wave=65536 // (
        (width + 7) // 8 * 8 * ((height + 7) // 8 * 8)))
    assert np.array_equal(plain, want)
