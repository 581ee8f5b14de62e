"""Performance cases: the calls a user of this renderer makes, at the sizes they make them.

A case is a dict of plain values; ``listed()`` returns the fixed ones,
``draw(rng)`` one more of the same ranges, ``prepare(case, seed)`` what a
program holds before the call (a committed scene, a film buffer, rays on the
GPU, a server), ``run(state)`` one pass through the public entry points and
``work(case)`` the bytes and operations such a pass cannot do without.

Kinds of case:

* ``render``: one frame with one of the four integrators, into host memory
  (a renderer object, as code written against the reference's
  ``Renderer::render`` does it) or into a CUDA tensor (``Scene.render``);
* ``trace``: closest-hit or any-hit ray queries on device rays;
* ``serve``: a burst of requests through the batching server;
* ``bmp``: a film to 8-bit BMP rows.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from slr_gb300 import api, raysets, scenes

# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # An interactive preview: one sample per pixel of a thumbnail, where
        # the launches of the bounces count and not the rays.
        dict(name="preview_box", kind="render", integrator="pt", scene="box", film="host", width=64, height=64, spp=1,
             depth=8),
        # The closed-box frame of the benchmark, host film through the
        # renderer object.
        dict(name="box_frame", kind="render", integrator="pt", scene="box", film="host", width=256, height=256, spp=16,
             depth=8),
        # Every BSDF kind under a thin lens, an image that is not a multiple
        # of the sensor's 8 x 8 tiles.
        dict(name="glossy_ragged", kind="render", integrator="pt", scene="glossy", film="device", width=333,
             height=187, spp=24, depth=12),
        # A draft of a 176k-triangle GGX terrain under an environment.
        dict(name="terrain_draft", kind="render", integrator="pt", scene="terrain", grid=256, spheres=16, freq=12,
             film="device", width=512, height=512, spp=4, depth=10),
        # The headline benchmark's frame: 1,034,242 triangles, 64 samples per
        # pixel of a 1024 x 1024 image.
        dict(name="terrain_1m", kind="render", integrator="pt", scene="terrain", grid=512, spheres=64, freq=20,
             film="device", width=1024, height=1024, spp=64, depth=10),
        # The volumetric path tracer in a 256^3 density grid.
        dict(name="cloud_frame", kind="render", integrator="volpt", scene="cloud", voxels=256, film="device",
             width=512, height=512, spp=8, depth=32),
        # The bidirectional tracer on the box.
        dict(name="bpt_box", kind="render", integrator="bpt", scene="box", film="device", width=512, height=512, spp=4,
             depth=16),
        # The volumetric bidirectional tracer, the costliest sample of all.
        dict(name="bpt_cloud", kind="render", integrator="vbpt", scene="cloud", voxels=128, film="device", width=200,
             height=152, spp=4, depth=12),
        # Ray queries: closest hits of incoherent rays (baking, sensors) ...
        dict(name="closest_incoherent", kind="trace", scene="terrain", grid=96, spheres=8, freq=6, rays=1000003,
             coherent=False, any_hit=False),
        # ... and a large batch of visibility tests.
        dict(name="any_incoherent", kind="trace", scene="terrain", grid=256, spheres=16, freq=12, rays=1 << 22,
             coherent=False, any_hit=True),
        # A burst of 24 requests of three scenes (one with a medium) through
        # the batching server.
        dict(name="serve_burst", kind="serve", requests=24, max_side=256, max_spp=16, depth=8),
        # The finished film of a full-HD frame to BMP rows.
        dict(name="film_bmp", kind="bmp", width=1920, height=1080),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pt", "pt", "pt", "volpt", "bpt", "vbpt", "trace", "trace", "serve", "bmp"])
    if kind == "pt":
        scene = rng.choice(["box", "glossy", "terrain"])
        w, h = _log_int(rng, 24, 900), _log_int(rng, 24, 900)
        c = dict(kind="render", integrator="pt", scene=scene, film=rng.choice(["host", "device"]), width=w, height=h,
                 spp=min(_log_int(rng, 1, 64), max(1, (16 << 20) // (w * h))), depth=rng.randint(3, 16))
        if scene == "terrain":
            c.update(grid=_log_int(rng, 32, 400), spheres=rng.randint(2, 24), freq=rng.randint(2, 14))
        return c
    if kind == "volpt":
        w, h = _log_int(rng, 24, 512), _log_int(rng, 24, 512)
        return dict(kind="render", integrator="volpt", scene="cloud", voxels=_log_int(rng, 20, 256), film="device",
                    width=w, height=h, spp=min(_log_int(rng, 1, 16), max(1, (2 << 20) // (w * h))),
                    depth=rng.randint(6, 32))
    if kind == "bpt":
        w, h = _log_int(rng, 24, 512), _log_int(rng, 24, 512)
        return dict(kind="render", integrator="bpt", scene=rng.choice(["box", "glossy"]), film="device", width=w,
                    height=h, spp=min(_log_int(rng, 1, 8), max(1, (1 << 20) // (w * h))), depth=rng.randint(4, 16))
    if kind == "vbpt":
        w, h = _log_int(rng, 24, 200), _log_int(rng, 24, 152)
        return dict(kind="render", integrator="vbpt", scene="cloud", voxels=_log_int(rng, 20, 128), film="device",
                    width=w, height=h, spp=_log_int(rng, 1, 4), depth=rng.randint(4, 12))
    if kind == "trace":
        return dict(kind="trace", scene="terrain", grid=_log_int(rng, 24, 256), spheres=rng.randint(2, 16),
                    freq=rng.randint(2, 12), rays=_log_int(rng, 1000, 1 << 22), coherent=rng.random() < 0.4,
                    any_hit=rng.random() < 0.5)
    if kind == "serve":
        return dict(kind="serve", requests=rng.randint(2, 24), max_side=_log_int(rng, 32, 256),
                    max_spp=_log_int(rng, 1, 16), depth=rng.randint(3, 8))
    return dict(kind="bmp", width=_log_int(rng, 33, 1920), height=_log_int(rng, 33, 1080))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _cloud_grid(n, seed):
    """n^3 density [z][y][x], max(0, 5 octaves of interpolated noise), largest value 1."""
    g = torch.Generator().manual_seed(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    total = torch.zeros((n, n, n), device=dev)
    for o in range(5):
        k = min(n, 4 << o)
        noise = (torch.rand((1, 1, k, k, k), generator=g) - 0.5).to(dev)
        total += 0.5 ** o * torch.nn.functional.interpolate(noise, size=(n, n, n), mode="trilinear",
                                                            align_corners=True)[0, 0]
    total.clamp_(min=0.0)
    return (total / total.max()).float().cpu().numpy()


def _scene_desc(case, seed):
    """The scene of a case; the seed varies its content and its camera."""
    w, h = case.get("width", 512), case.get("height", 512)
    if case["scene"] == "terrain":
        return scenes.heightfield_scene(grid=case["grid"], spheres=case["spheres"], sphere_freq=case["freq"],
                                        env_size=(512, 256) if case["grid"] > 256 else (256, 128), width=w, height=h,
                                        seed=seed)
    rng = np.random.default_rng(seed)
    eye = np.array([0.5, 0.5, 2.3]) + rng.uniform(-0.05, 0.05, 3)
    if case["scene"] == "glossy":
        d = scenes.glossy_box_scene(w, h)
        d.camera.lens_radius = 0.02
    elif case["scene"] == "cloud":
        d = scenes.medium_box_scene(w, h, grid=8)
        d.medium.density = _cloud_grid(case["voxels"], seed)
    else:
        d = scenes.box_scene(w, h)
    d.camera.cam_to_world = scenes.look_at(eye, (0.5, 0.5, 0.0))
    return d


def _rays(case, desc, seed):
    if not case["coherent"]:
        # drawn on the host, whose generator and sums repeat bit for bit
        rays = raysets.incoherent_rays(desc, case["rays"], device="cpu", seed=seed)
    else:
        side = int(math.ceil(math.sqrt(case["rays"])))
        rays = raysets.coherent_rays(desc, side, device="cpu")[:case["rays"]].contiguous()
    return rays.cuda()


def _film(width, height, seed):
    """A film as a 64-sample render leaves it: smooth exposure with noise, mostly below clipping."""
    rng = np.random.default_rng(seed)
    y, x = np.meshgrid(np.linspace(0, 3, height, dtype=np.float32), np.linspace(0, 5, width, dtype=np.float32),
                       indexing="ij")
    base = (0.02 + 0.01 * (np.sin(x + rng.uniform(0, 6)) + np.cos(y * x))).astype(np.float32)
    spread = rng.uniform(0.2, 1.8, 16).astype(np.float32)
    grain = rng.random((height, width), np.float32) + 0.5
    return np.maximum(base * grain, 0.0)[..., None] * spread * 64.0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "bmp":
        return dict(kind=kind, film=_film(case["width"], case["height"], seed))
    if kind == "serve":
        rng = np.random.default_rng(case["requests"])   # the sizes belong to the case, the content to the seed
        descs = [scenes.box_scene(128, 128),
                 scenes.heightfield_scene(grid=64, spheres=8, sphere_freq=6, env_size=(256, 128), seed=seed),
                 _scene_desc(dict(scene="cloud", voxels=64), seed)]
        scs = [api.Scene(d) for d in descs]
        reqs = []
        for i in range(case["requests"]):
            k = int(rng.integers(0, 3))
            side = int(rng.integers(max(8, case["max_side"] // 4), case["max_side"] + 1))
            reqs.append(dict(scene=k, side=side, spp=int(rng.integers(1, case["max_spp"] + 1)), seed=seed * 100 + i))
        return dict(kind=kind, server=api.Server(max_depth=case["depth"]), scenes=scs, requests=reqs,
                    depth=case["depth"], volumetric=[d.medium is not None for d in descs])
    desc = _scene_desc(case, seed)
    scene = api.Scene(desc)
    if kind == "trace":
        return dict(kind=kind, scene=scene, rays=_rays(case, desc, seed), any_hit=case["any_hit"])
    cls = {"pt": api.PathTracingRenderer, "volpt": api.VolumetricPathTracingRenderer,
           "bpt": api.BidirectionalPathTracingRenderer,
           "vbpt": api.VolumetricBidirectionalPathTracingRenderer}[case["integrator"]]
    st = dict(kind=kind, scene=scene, integrator=case["integrator"], film=None, width=case["width"],
              height=case["height"], spp=case["spp"], depth=case["depth"], seed=seed)
    if case["film"] == "device":
        st["film"] = torch.empty((case["height"], case["width"], 16), dtype=torch.float32, device="cuda")
    else:
        st["renderer"] = cls(case["spp"], case["depth"])
        st["settings"] = api.RenderSettings(ImageWidth=case["width"], ImageHeight=case["height"], RNGSeed=seed)
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "bmp":
        return api.film_to_bmp(state["film"], scale=1.0 / 64.0)
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(state["scenes"][r["scene"]], r["side"], r["side"], r["spp"], state["depth"], seed=r["seed"],
                          volumetric=state["volumetric"][r["scene"]]) for r in state["requests"]]
        return [srv.wait(i)[0] for i in ids]
    if kind == "trace":
        prim, t, b1, b2 = state["scene"].trace(state["rays"], any_hit=state["any_hit"])
        return dict(prim=prim) if state["any_hit"] else dict(prim=prim, t=t, b1=b1, b2=b2)
    if state["film"] is None:
        return state["renderer"].render(state["scene"], state["settings"])
    it = state["integrator"]
    film, _ = state["scene"].render(state["width"], state["height"], state["spp"], state["depth"], seed=state["seed"],
                                    volumetric=it in ("volpt", "vbpt"), bpt=it in ("bpt", "vbpt"), film=state["film"])
    return film


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

# Arithmetic of one closest-hit query (about 20 nodes of four box tests and 6
# triangle tests), of one any-hit query, and of one shaded vertex (16
# wavelengths of light, BSDF and throughput), in operations.
_OPS_CLOSEST, _OPS_ANY, _OPS_VERTEX = 20 * 4 * 18 + 6 * 45, 12 * 4 * 18 + 4 * 45, 1200
# Vertices of a path that ends by roulette, per integrator (both subpaths of
# the bidirectional ones), and extra operations of a vertex in a medium (free
# flight and 16 transmittance estimates).
_VERTICES = {"pt": 3.0, "volpt": 6.0, "bpt": 8.0, "vbpt": 12.0}
_OPS_MEDIUM = 16 * 12 * 120


def _triangles(case):
    if case.get("scene") == "terrain":
        return 2 * (case["grid"] - 1) ** 2 + case["spheres"] * 20 * case["freq"] ** 2
    return 34


def _render_work(integrator, triangles, voxels, width, height, spp, depth):
    vertices = min(_VERTICES[integrator], depth) * width * height * spp
    flops = vertices * (_OPS_CLOSEST + _OPS_ANY + _OPS_VERTEX)
    if integrator in ("volpt", "vbpt"):
        flops += vertices * _OPS_MEDIUM
    # triangles (three positions and normals) and density read once, film written once
    return triangles * 72 + voxels ** 3 * 4 + width * height * 64, flops


def work(case):
    kind = case["kind"]
    if kind == "bmp":
        px = case["width"] * case["height"]
        return {"bytes": px * (64 + 3), "flops": px * (16 * 7 + 3 * 60)}
    if kind == "trace":
        out = 4 if case["any_hit"] else 16
        return {"bytes": case["rays"] * (32 + out) + _triangles(case) * 36,
                "flops": case["rays"] * (_OPS_ANY if case["any_hit"] else _OPS_CLOSEST)}
    if kind == "serve":
        side, spp = case["max_side"] * 5 / 8, (1 + case["max_spp"]) / 2
        n = case["requests"]
        surf = _render_work("pt", 13000, 0, side, side, spp, case["depth"])
        vol = _render_work("volpt", 34, 64, side, side, spp, case["depth"])
        return {"bytes": n * (2 * surf[0] + vol[0]) / 3, "flops": n * (2 * surf[1] + vol[1]) / 3}
    b, f = _render_work(case["integrator"], _triangles(case), case.get("voxels", 0), case["width"], case["height"],
                        case["spp"], case["depth"])
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------


def exact(case, seed):
    """Closest hits by testing every triangle in 64 bits, where that is a few
    seconds' work.  A film has no such value (each sample is a chain of
    random decisions) and BMP rows and any-hit answers are whole numbers."""
    if case["kind"] != "trace" or case["any_hit"] or case["rays"] * _triangles(case) > 3e10:
        return None
    desc = _scene_desc(case, seed)
    rays = _rays(case, desc, seed).double()
    tris = torch.tensor(desc.triangle_arrays(), dtype=torch.float32, device=rays.device).double()
    v0, e1, e2 = tris[:, 0], tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]
    n = torch.linalg.cross(e1, e2)
    out = {k: torch.full((len(rays),), v, dtype=torch.float64, device=rays.device)
           for k, v in (("t", math.inf), ("b1", 0.0), ("b2", 0.0))}
    # with s = o - v0: t = -n.s / n.d, b1 = -d.(e2 x s) / n.d, b2 = d.(e1 x s) / n.d, each split
    # into products of per-triangle and per-ray rows
    c1, c2, nv0 = torch.linalg.cross(e1, v0), torch.linalg.cross(e2, v0), (n * v0).sum(1)
    step = max(1, int(1.5e8) // len(tris))
    for i in range(0, len(rays), step):
        r = rays[i:i + step]
        o, d = r[:, 0:3], r[:, 4:7]
        od = torch.linalg.cross(o, d)
        det = d @ n.T
        t = (nv0 - o @ n.T) / det
        b1 = (d @ c2.T - od @ e2.T) / det
        b2 = (od @ e1.T - d @ c1.T) / det
        hit = (det != 0) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= r[:, 3:4]) & (t <= r[:, 7:8])
        t = torch.where(hit, t, math.inf)
        best, k = t.min(1)
        found = torch.isfinite(best)
        rows = torch.arange(len(r), device=r.device)
        out["t"][i:i + step] = best
        out["b1"][i:i + step] = torch.where(found, b1[rows, k], 0.0)
        out["b2"][i:i + step] = torch.where(found, b2[rows, k], 0.0)
    return dict(prim=None, **out)
