"""Performance cases of the rasterizer, through its public entry points.

Each case is a plain dict; ``prepare`` makes what a program has in hand before
the call (scene buffers on the GPU, surfaces, an initialised CudaRaster with
its default tuning), ``run`` is one pass (a frame, a batch, a vertex-shader or
resolve call, a predictor pass) and returns every word that it wrote. Scenes
are seeded synthetic ones of the shapes that bench.py and the tests use,
generated on the GPU.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

PKG = "cudaraster-linux_gb300"
CLEAR = ((0.1, 0.2, 0.3, 1.0), 1.0)
RESOLUTIONS = [(256, 256), (512, 512), (1024, 768), (1920, 1080)]
# Pipe, samples per pixel: every blend, sample count and render mode that a scene of Gouraud records can ask for.
GOURAUD_PIPES = [("PixelPipe_gouraud", 1), ("PixelPipe_gouraud_srcover", 1), ("PixelPipe_gouraud_additive", 1),
                 ("PixelPipe_gouraud_nodepth", 1), ("PixelPipe_gouraud_depthonly", 1), ("PixelPipe_gouraud_flat", 1),
                 ("PixelPipe_gouraud_msaa2", 2), ("PixelPipe_gouraud_msaa4", 4), ("PixelPipe_gouraud_msaa8", 8),
                 ("PixelPipe_gouraud_srcover_msaa4", 4)]


def _mod(name=""):
    return importlib.import_module(PKG + ("." + name if name else ""))


def listed():
    return [
        # The demo cube, one blocking draw: the smallest call, launches and latency only.
        {"name": "cube_1024x768", "kind": "cube", "width": 1024, "height": 768, "timing": True},
        # A small translucent mesh on an odd viewport (an interactive viewer's frame).
        {"name": "soup_5k_blend_641x479", "kind": "soup", "tris": 5003, "width": 641, "height": 479, "median_px": 6.0,
         "pipe": "PixelPipe_gouraud_srcover", "samples": 1, "queued": False, "timing": True},
        # The headline: one million small opaque triangles at 1080p, blocking draw.
        {"name": "soup_1m_1080p", "kind": "soup", "tris": 1000000, "width": 1920, "height": 1080, "median_px": 4.0,
         "pipe": "PixelPipe_gouraud", "samples": 1, "queued": False, "timing": False},
        # Order-dependent blending at 1080p, draws queued without waiting (a render loop that runs ahead).
        {"name": "soup_300k_blend_1080p", "kind": "soup", "tris": 300000, "width": 1920, "height": 1080,
         "median_px": 6.0, "pipe": "PixelPipe_gouraud_srcover", "samples": 1, "queued": True, "timing": False},
        # Few large triangles (architecture, CAD, user interfaces): every triangle covers many tiles.
        {"name": "large_20k_1440p", "kind": "soup", "tris": 20000, "width": 2560, "height": 1440, "median_px": 60.0,
         "pipe": "PixelPipe_gouraud", "samples": 1, "queued": False, "timing": False},
        # The subpixel stress: 8.4M triangles, 3840x2160, 4x MSAA.
        {"name": "grid_2048_msaa4_4k", "kind": "grid", "n": 2048, "width": 3840, "height": 2160,
         "pipe": "PixelPipe_gouraud_msaa4", "samples": 4, "queued": False, "timing": False},
        # A fly-through frame: 33.5M terrain triangles and a blended water layer, the vertex transform fused into setup.
        {"name": "fly_4096_4k", "kind": "fly", "n": 4096, "width": 3840, "height": 2160, "timing": False},
        # Many independent scenes of uneven sizes, half of them blended, replayed as one CUDA graph.
        {"name": "batch_32_graph", "kind": "batch", "scenes": 32, "lo": 1000, "hi": 500000, "graph": True},
        # Textured, lit, alpha-tested terrain at 4K: the vertex shader and the draw.
        {"name": "textured_2048_4k", "kind": "textured", "n": 2048, "width": 3840, "height": 2160,
         "pipe": "PixelPipe_texPhong", "samples": 1, "timing": False},
        # The lit vertex shader alone, over more vertices than the L2 holds.
        {"name": "vertex_gouraud_8m", "kind": "vertex", "shader": "gouraud", "n": 8388608},
        # A 4x MSAA frame resolved to an image, on a size that is no multiple of the 8x8 tiles.
        {"name": "resolve_msaa4_3839x2159", "kind": "resolve", "width": 3839, "height": 2159, "samples": 4},
        # One backward and one forward pass of the queue predictor at its fly-through shape (510 bins).
        {"name": "predictor_b32", "kind": "predictor", "batch": 32, "outputs": 1022},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["soup", "soup", "soup", "soup", "grid", "grid", "fly", "batch", "textured", "vertex",
                       "resolve", "predictor"])
    width, height = _log(rng, 200, 3840), _log(rng, 150, 2160)
    timing = rng.random() < 0.3
    if kind == "soup":
        pipe, samples = rng.choice(GOURAUD_PIPES)
        tris = _log(rng, 500, 1500000)
        # Larger triangles come in smaller numbers: at most about 40 layers over the viewport.
        median = max(2.0, min(100.0, math.exp(rng.uniform(math.log(2.0), math.log(100.0))),
                              math.sqrt(40.0 * width * height / tris)))
        return {"kind": kind, "tris": tris, "width": width, "height": height, "median_px": round(median, 2),
                "pipe": pipe, "samples": samples, "queued": rng.random() < 0.4, "timing": timing}
    if kind == "grid":
        pipe, samples = rng.choice(GOURAUD_PIPES)
        return {"kind": kind, "n": _log(rng, 64, 2048), "width": width, "height": height, "pipe": pipe,
                "samples": samples, "queued": rng.random() < 0.4, "timing": timing}
    if kind == "fly":
        return {"kind": kind, "n": _log(rng, 256, 4000), "width": width, "height": height, "timing": timing}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 32), "lo": 500, "hi": _log(rng, 5000, 500000),
                "graph": rng.random() < 0.5}
    if kind == "textured":
        pipe, samples = rng.choice([("PixelPipe_texPhong", 1), ("PixelPipe_texPhong_quads", 1),
                                    ("PixelPipe_texPhong_srcover", 1), ("PixelPipe_texPhong_msaa4", 4)])
        return {"kind": kind, "n": _log(rng, 64, 2048), "width": width, "height": height, "pipe": pipe,
                "samples": samples, "timing": timing}
    if kind == "vertex":
        return {"kind": kind, "shader": rng.choice(["passthrough", "gouraud", "tex_phong"]),
                "n": _log(rng, 1000, 8388608)}
    if kind == "resolve":
        return {"kind": kind, "width": width, "height": height, "samples": rng.choice([1, 2, 4, 8])}
    return {"kind": kind, "batch": rng.randint(1, 64), "outputs": 2 * rng.randint(16, 600) + 2}


# ------------------------------------------------------------------ scenes
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _soup(g, n, width, height, median_px, blended):
    """scenes.soup on the GPU: random triangles, lognormal edge length, half of them back-facing."""
    w = _uniform(g, (n, 1), 1.0, 10.0)
    c = _uniform(g, (n, 3), -1.0, 1.0)
    r = median_px * torch.exp(torch.randn((n, 1), generator=g, device="cuda", dtype=torch.float64)) / math.sqrt(3.0)
    k = torch.arange(3, device="cuda", dtype=torch.float64)
    ang = _uniform(g, (n, 1), 0.0, 2.0 * math.pi) + 2.0 * math.pi / 3.0 * k + _uniform(g, (n, 3), -0.35, 0.35)
    back = torch.rand((n, 1), generator=g, device="cuda") < 0.5
    ang = torch.where(back, ang.flip(1), ang)
    v = torch.empty((n, 3, 8), dtype=torch.float32, device="cuda")
    v[..., 0] = (c[:, 0:1] + r * torch.cos(ang) * (2.0 / width)) * w
    v[..., 1] = (c[:, 1:2] + r * torch.sin(ang) * (2.0 / height)) * w
    v[..., 2] = torch.clamp(c[:, 2:3] + _uniform(g, (n, 3), -0.01, 0.01), -1.0, 1.0) * w
    v[..., 3] = w
    v[..., 4:8] = torch.randint(0, 256, (n, 3, 4), generator=g, device="cuda").float() / 255.0
    if blended:
        v[..., 7] = (torch.round(_uniform(g, (n, 1), 0.2, 1.0) * 255.0) / 255.0).float()
    return v.reshape(3 * n, 8), torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(n, 3)


def _heights(g, n):
    """scenes.value_noise on the GPU: six octaves of smoothed lattice noise, times the heightfield's 0.4."""
    out = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for o in range(6):
        cells = 4 << o
        lat = _uniform(g, (cells + 2, cells + 2), -1.0, 1.0)
        x = torch.arange(n, dtype=torch.float64, device="cuda") * (cells / n)
        i = x.long()
        f = x - i
        f = f * f * (3.0 - 2.0 * f)
        rows = lat[i] * (1.0 - f)[:, None] + lat[i + 1] * f[:, None]
        out += (rows[:, i] * (1.0 - f) + rows[:, i + 1] * f) * 0.5 ** o
    return out / sum(0.5 ** o for o in range(6)) * 0.4


def _grid_indices(n):
    i = torch.arange(n - 1, device="cuda", dtype=torch.int32)
    v00 = (i[:, None] * n + i[None, :]).reshape(-1)
    return torch.stack([v00, v00 + n, v00 + 1, v00 + 1, v00 + n, v00 + n + 1], dim=1).reshape(-1, 3).contiguous()


def _plane(n):
    x = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda")
    return x[None, :].expand(n, n), x[:, None].expand(n, n)


def _heightfield(g, n):
    """Model positions [n * n, 3], colours [n * n, 4] and indices of the heightfield, and its heights."""
    h = _heights(g, n)
    X, Z = _plane(n)
    t = (h / 0.4 + 1.0) * 0.5
    rgba = torch.stack([0.2 + 0.6 * t, 0.5 + 0.3 * (1.0 - t), 0.25 + 0.2 * t, torch.full_like(t, 0.8)], dim=-1)
    rgba = (torch.round(rgba * 255.0) / 255.0).float().reshape(-1, 4)
    return torch.stack([X, h, Z], dim=-1).float().reshape(-1, 3), rgba, _grid_indices(n), h


def _surfaces(width, height, samples):
    p = _mod()
    return (p.CudaSurface((width, height), p.CudaSurface.FORMAT_RGBA8, samples),
            p.CudaSurface((width, height), p.CudaSurface.FORMAT_DEPTH32, samples))


def _raster(surfaces, pipe, vertices, indices, timing):
    cr = _mod().CudaRaster()
    cr.init()
    cr.setSurfaces(*surfaces)
    cr.setPixelPipe(None, pipe)
    cr.setVertexBuffer(vertices, 0)
    cr.setIndexBuffer(indices, 0, indices.shape[0])
    cr.setStageTiming(timing)
    return cr


def _camera(seed, width, height, elevation=15.0):
    scenes = _mod("scenes")
    eye, target = scenes.terrain_eye_target(float(seed * 37 % 300), elevation)
    view = scenes.look_at(eye, target).astype(np.float32)
    proj = scenes.perspective(60.0, width / height, 0.05, 10.0).astype(np.float32)
    return (proj @ view).astype(np.float32), view


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    g = _gen(seed * 1000003 + 17)
    return {"case": dict(case), **globals()["_prepare_" + case["kind"]](case, seed, g)}


def _prepare_cube(case, seed, g):
    sc = _mod("scenes").cube(case["width"], case["height"], distance=2.5 + (seed % 64) / 64.0)
    s = _surfaces(case["width"], case["height"], 1)
    v, i = torch.from_numpy(sc["vertices"]).cuda(), torch.from_numpy(sc["indices"]).cuda()
    return {"cr": _raster(s, "PixelPipe_gouraud", v, i, case["timing"]), "surfaces": s, "queued": False}


def _prepare_soup(case, seed, g):
    blended = "srcover" in case["pipe"] or "nodepth" in case["pipe"]
    v, i = _soup(g, case["tris"], case["width"], case["height"], case["median_px"], blended)
    return _prepare_single(case, v, i)


def _prepare_grid(case, seed, g):
    pos, rgba, idx, _ = _heightfield(g, case["n"])
    mvp, _ = _camera(seed, case["width"], case["height"])
    return _prepare_single(case, _mod("raster").vertex_shader_passthrough(pos, mvp, rgba), idx)


def _prepare_single(case, vertices, indices):
    s = _surfaces(case["width"], case["height"], case["samples"])
    cr = _raster(s, case["pipe"], vertices, indices, case["timing"])
    if case["queued"]:   # a program that queues draws sizes its queues with a blocking one first
        cr.deferredClear(*CLEAR)
        cr.drawTriangles()
    return {"cr": cr, "surfaces": s, "queued": case["queued"]}


def _prepare_fly(case, seed, g):
    n = case["n"]
    m = max(2, int(round((n - 1) * math.sqrt(0.1))) + 1)
    pos, rgba, idx, _ = _heightfield(g, n)
    X, Z = _plane(m)
    ripple = 0.5 + 0.5 * torch.sin(X * 37.0) * torch.cos(Z * 29.0)
    wpos = torch.stack([X, torch.full_like(X, -0.02), Z], dim=-1).float().reshape(-1, 3)
    wrgba = torch.stack([0.1 + 0.1 * ripple, 0.3 + 0.2 * ripple, 0.6 + 0.2 * ripple, torch.full_like(X, 0.35)], dim=-1)
    wrgba = (torch.round(wrgba * 255.0) / 255.0).float().reshape(-1, 4)
    s = _surfaces(case["width"], case["height"], 1)
    layers = []
    for p, c, i, pipe in ((pos, rgba, idx, "PixelPipe_gouraud"),
                          (wpos, wrgba, _grid_indices(m), "PixelPipe_gouraud_srcover")):
        records = torch.zeros((p.shape[0], 8), dtype=torch.float32, device="cuda")
        records[:, 4:8] = c
        model = torch.ones((p.shape[0], 4), dtype=torch.float32, device="cuda")
        model[:, 0:3] = p
        layers.append((_raster(s, pipe, records, i, case["timing"]), model))
    return {"layers": layers, "surfaces": s, "mvp": _camera(seed, case["width"], case["height"])[0]}


def _prepare_batch(case, seed, g):
    r = np.random.default_rng(case["scenes"])   # the batch's sizes are the case's, its scenes are the seed's
    p = _mod()
    items = []
    for k in range(case["scenes"]):
        n = int(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        w, h = RESOLUTIONS[int(r.integers(0, len(RESOLUTIONS)))]
        blended = k % 2 == 1
        v, i = _soup(g, n, w, h, 4.0, blended)
        c, d = _surfaces(w, h, 1)
        items.append({"pipe": "PixelPipe_gouraud_srcover" if blended else "PixelPipe_gouraud", "color": c, "depth": d,
                      "vertices": v, "indices": i, "numTris": n, "clear": (*CLEAR[0], CLEAR[1])})
    cr = p.CudaRaster()
    cr.init()
    cr.setStageTiming(False)
    state = {"cr": cr, "items": items, "graph": None}
    if case["graph"]:
        cr.drawBatch(items)   # sizes the queues that the capture fixes
        state["graph"] = cr.createBatchGraph(items)
    return state


def _prepare_textured(case, seed, g):
    scenes, raster = _mod("scenes"), _mod("raster")
    n = case["n"]
    pos, _, idx, h = _heightfield(g, n)
    gz, gx = torch.gradient(h, spacing=2.0 / (n - 1))
    nrm = torch.stack([-gx, torch.ones_like(gx), -gz], dim=-1)
    nrm = (nrm / nrm.norm(dim=-1, keepdim=True)).float().reshape(-1, 3)
    X, Z = _plane(n)
    uv = torch.stack([X * 3.0, (Z + 1.0) * 3.0], dim=-1).float().reshape(-1, 2)
    r = np.random.default_rng(seed + 9)
    texs = [(np.clip(np.stack([scenes.value_noise(64, 64, 4, seed + 10 * t + c) for c in range(4)], axis=-1) * 0.6 + 0.5
                     + r.uniform(-0.08, 0.08, (64, 64, 4)), 0.0, 1.0) * 255.0).round().astype(np.uint8)
            for t in range(3)]
    atlas, specs = scenes.texture_atlas(texs, 256, 128)
    materials = raster.material_records(
        diffuse=[[0.7, 0.6, 0.5, 1.0], [1.0, 1.0, 1.0, 1.0], [1.0, 1.0, 1.0, 1.0], [1.0, 1.0, 1.0, 0.8]],
        specular=[[0.3, 0.3, 0.3], [0.5, 0.5, 0.4], [0.2, 0.2, 0.2], [0.8, 0.8, 0.8]],
        glossiness=[8.0, 32.0, 4.0, 96.0], diffuse_texture=[None, specs[0], specs[2], specs[2]],
        alpha_texture=[None, None, specs[1], None])
    clip, view = _camera(seed, case["width"], case["height"], 25.0)
    shaded = torch.empty((n * n, 16), dtype=torch.float32, device="cuda")
    s = _surfaces(case["width"], case["height"], case["samples"])
    return {"input": torch.cat([pos, nrm, uv], dim=1).contiguous(), "shaded": shaded, "surfaces": s,
            "matrices": (clip, view, view[:3, :3].copy()),
            "materials": torch.from_numpy(materials).cuda(), "atlas": torch.from_numpy(atlas.view(np.int32)).cuda(),
            "tri_material": torch.randint(0, 4, (idx.shape[0],), generator=g, device="cuda", dtype=torch.int32),
            "cr": _raster(s, case["pipe"], shaded, idx, case["timing"])}


def _prepare_vertex(case, seed, g):
    n = case["n"]
    records = torch.rand((n, 8), generator=g, device="cuda", dtype=torch.float32) * 2.0 - 1.0
    scenes = _mod("scenes")
    view = scenes.look_at((1.5, 2.0, 3.0 + (seed % 16) / 16.0), (0.0, 0.0, 0.0)).astype(np.float32)
    clip = (scenes.perspective(60.0, 16 / 9, 0.1, 100.0) @ view).astype(np.float32)
    st = {"matrices": (clip, view, view[:3, :3].copy()),
          "out": torch.empty((n, 16 if case["shader"] == "tex_phong" else 8), dtype=torch.float32, device="cuda")}
    if case["shader"] == "passthrough":
        return {**st, "model": records[:, 0:3].contiguous(), "colors": (records[:, 4:8] * 0.5 + 0.5).contiguous()}
    if case["shader"] == "gouraud":
        mats = _mod("raster").material_records([[0.7, 0.6, 0.5, 1.0], [0.2, 0.9, 0.4, 0.5]] * 2, [[0.3, 0.3, 0.3]] * 4,
                                               [8.0, 16.0, 32.0, 64.0])
        st.update(materials=torch.from_numpy(mats).cuda(),
                  material_idx=torch.randint(0, 4, (n,), generator=g, device="cuda", dtype=torch.int32))
    return {**st, "records": records}


def _prepare_resolve(case, seed, g):
    color, _ = _surfaces(case["width"], case["height"], case["samples"])
    color.tensor.copy_(torch.randint(-2**31, 2**31 - 1, color.tensor.shape, generator=g, device="cuda",
                                     dtype=torch.int32))
    return {"color": color}


def _predictor_data(case, seed):
    """Host data of a predictor pass: parameters, samples, targets and the batch's rows."""
    r = np.random.default_rng(seed + 3)
    dims = (262, 64, 64, case["outputs"])
    sizes = [(64 * 262, 262), (64, 262), (64 * 64, 64), (64, 64), (64 * dims[3], 64), (dims[3], 64)]
    params = np.concatenate([r.uniform(-1.0, 1.0, n) / math.sqrt(fan) for n, fan in sizes]).astype(np.float32)
    x = r.normal(0.5, 0.5, (64, dims[0])).astype(np.float32)
    t = r.normal(0.0, 0.05, (64, dims[3])).astype(np.float32)
    return dims, params, x, t, r.integers(0, 64, case["batch"]).astype(np.int32)


def _prepare_predictor(case, seed, g):
    dims, params, x, t, rows = _predictor_data(case, seed)
    net = _mod("predictor").Network(*dims, max_batch=64, params=params)
    return {"net": net, "x": torch.from_numpy(x).cuda(), "t": torch.from_numpy(t).cuda(),
            "rows": torch.from_numpy(rows).cuda()}


# --------------------------------------------------------------------- run
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state, state["case"])


def _run_single(st, case):
    cr = st["cr"]
    cr.deferredClear(*CLEAR)
    if st["queued"]:
        cr.drawTrianglesAsync()
    else:
        cr.drawTriangles()
    return [s.tensor for s in st["surfaces"]]


_run_cube = _run_soup = _run_grid = _run_single


def _run_fly(st, case):
    for k, (cr, model) in enumerate(st["layers"]):
        cr.setVertexTransform(model, st["mvp"])
        if k == 0:
            cr.deferredClear(*CLEAR)
        cr.drawTriangles()
    return [s.tensor for s in st["surfaces"]]


def _run_batch(st, case):
    if st["graph"] is not None:
        st["graph"].launch()
    else:
        st["cr"].drawBatch(st["items"])
    return [s.tensor for it in st["items"] for s in (it["color"], it["depth"])]


def _run_textured(st, case):
    raster = _mod("raster")
    raster.set_tex_phong_constants(st["materials"], st["tri_material"], st["atlas"])
    raster.vertex_shader_tex_phong(st["input"], *st["matrices"], out=st["shaded"])
    st["cr"].deferredClear(*CLEAR)
    st["cr"].drawTriangles()
    return [s.tensor for s in st["surfaces"]]


def _run_vertex(st, case):
    raster = _mod("raster")
    if case["shader"] == "passthrough":
        return raster.vertex_shader_passthrough(st["model"], st["matrices"][0], st["colors"], out=st["out"])
    if case["shader"] == "gouraud":
        return raster.vertex_shader_gouraud(st["records"], *st["matrices"], st["materials"], st["material_idx"],
                                            out=st["out"])
    return raster.vertex_shader_tex_phong(st["records"], *st["matrices"], out=st["out"])


def _run_resolve(st, case):
    return st["color"].resolve()


def _run_predictor(st, case):
    grad, loss = st["net"].gradients(st["x"], st["t"], st["rows"])
    return {"grad": grad, "loss": loss, "y": st["net"].forward(st["x"])}


# -------------------------------------------------------------------- work
def _draw_work(tris, verts, stride, width, height, samples, surface_passes):
    pixels = ((width + 7) & ~7) * ((height + 7) & ~7) * samples
    return 12.0 * tris + stride * verts + 8.0 * pixels * surface_passes, 150.0 * tris + 30.0 * pixels


def work(case):
    kind = case["kind"]
    if kind in ("cube", "soup"):
        t = 12 if kind == "cube" else case["tris"]
        b, f = _draw_work(t, 8 if kind == "cube" else 3 * t, 32, case["width"], case["height"], case.get("samples", 1), 1)
    elif kind == "grid":
        n = case["n"]
        b, f = _draw_work(2 * (n - 1) ** 2, n * n, 32, case["width"], case["height"], case["samples"], 1)
    elif kind == "fly":
        n = case["n"]
        m = max(2, int(round((n - 1) * math.sqrt(0.1))) + 1)
        b, f = (x + y for x, y in zip(_draw_work(2 * (n - 1) ** 2, n * n, 32, case["width"], case["height"], 1, 1),
                                      _draw_work(2 * (m - 1) ** 2, m * m, 32, case["width"], case["height"], 1, 2)))
    elif kind == "batch":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        pixels = sum(w * h for w, h in RESOLUTIONS) / len(RESOLUTIONS)
        b, f = (case["scenes"] * x for x in _draw_work(mean, 3 * mean, 32, 8 * round(pixels / 64), 8, 1, 1))
    elif kind == "textured":
        n = case["n"]
        b, f = _draw_work(2 * (n - 1) ** 2, n * n, 64 + 96, case["width"], case["height"], case["samples"], 1)
        b, f = b + 8.0 * (n - 1) ** 2, f + 60.0 * n * n
    elif kind == "vertex":
        per = {"passthrough": (60, 28), "gouraud": (68, 130), "tex_phong": (96, 71)}[case["shader"]]
        b, f = per[0] * case["n"], per[1] * case["n"]
    elif kind == "resolve":
        pixels = case["width"] * case["height"]
        b, f = 4.0 * pixels * (case["samples"] + 1), 4.0 * pixels * case["samples"]
    else:
        params = 262 * 64 + 64 + 64 * 64 + 64 + 64 * case["outputs"] + case["outputs"]
        b = 2.0 * params + 4.0 * params + 4.0 * (64 + case["batch"]) * (262 + case["outputs"])
        f = 2.0 * params * (3 * case["batch"] + 64)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """64-bit values of the floating-point outputs; framebuffers and images are whole words."""
    if case["kind"] == "vertex":
        st = prepare(case, seed)
        clip, view, normal = (torch.from_numpy(m.astype(np.float64)).cuda() for m in st["matrices"])
        src = (st["model"] if case["shader"] == "passthrough" else st["records"]).double()
        pos = torch.cat([src[:, 0:3], torch.ones_like(src[:, 0:1])], dim=1)
        out = [pos @ clip.T]
        if case["shader"] == "passthrough":
            out.append(st["colors"].double())
        elif case["shader"] == "tex_phong":
            zero = torch.zeros_like(src[:, 0:1])
            out += [pos @ view.T, src[:, 3:6] @ normal.T, zero, src[:, 6:8], zero, zero + 1.0]
        else:
            mat = st["materials"][st["material_idx"].long()].double()
            unit = lambda a: a / a.norm(dim=1, keepdim=True)  # noqa: E731
            I, N = unit((pos @ view.T)[:, 0:3]), unit(src[:, 3:6] @ normal.T)
            cos = (I * N).sum(1, keepdim=True)
            spec = (-(I * (I - 2.0 * cos * N)).sum(1, keepdim=True)).clamp(min=0.0) ** mat[:, 7:8]
            out += [((-cos).clamp(min=0.0) * 0.75 + 0.25) * mat[:, 0:3] + spec * mat[:, 4:7], mat[:, 3:4]]
        return torch.cat(out, dim=1)
    if case["kind"] == "predictor":
        dims, params, x, t, rows = _predictor_data(case, seed)
        shapes = [(64, 262), (64,), (64, 64), (64,), (dims[3], 64), (dims[3],)]
        flat = torch.from_numpy(params).to(torch.bfloat16).double().split([math.prod(s) for s in shapes])
        w = [v.reshape(s).clone().requires_grad_(True) for v, s in zip(flat, shapes)]

        def net(a):
            a = torch.nn.functional.gelu(a @ w[0].T + w[1])
            return torch.nn.functional.gelu(a @ w[2].T + w[3]) @ w[4].T + w[5]

        xd, td, r = torch.from_numpy(x).double(), torch.from_numpy(t).double(), torch.from_numpy(rows).long()
        loss = ((net(xd[r]) - td[r]) ** 2).mean()
        loss.backward()
        return {"grad": torch.cat([v.grad.reshape(-1) for v in w]), "loss": loss.detach().reshape(1),
                "y": net(xd).detach()}
    return None
