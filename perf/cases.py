"""The renders that users of ymrt_b200 make, as timed cases.

Every case goes through the package's public calls: `Scene.render` (one frame
into a host array or a CUDA tensor), `render_batch` (many renders in one
call) and `render_batch` with path records followed by
`render_backward_ex` (gradients). Scenes, resolutions, sample counts, depths
and estimator options are those of the repository's benchmark and tests; the
drawn cases spread over the same ranges, odd resolutions among them.

What a program has in hand before the call (`prepare`): a context, the
uploaded scene with its sampler's permutation table, the output buffers, and
for gradients the path-record buffers and the target images. The seed chooses
the scene's random layout and materials and the permutation table, so two
seeds share no sample.
"""
from __future__ import annotations

import functools
import os
import tempfile

import numpy as np
import torch

import ymrt_b200 as Y
from ymrt_b200 import scenes

DEPTH = {"cornell": 8, "spheres": 8, "imaged": 12, "glossy": 8, "instanced": 12, "instanced_fog": 12,
         "volumetric": 16, "textured": 12}
GRID = 64   # the fog's density grid (per axis) of the differentiable media workload
SMOKE = 128  # the smoke box's density grid of the grid workload
PCG, HALTON = 0, 1


def _frame(name, scene, width, height, spp, **more):
    c = {"name": name, "kind": "frame", "scene": scene, "width": width, "height": height, "spp": spp,
         "sampler": HALTON, "media": False, "sun": False, "env": False, "roulette": False, "grid": False,
         "host": False}
    c.update(more)
    return c


def listed():
    return [
        # a thumbnail into a host array, the library's smallest render: launch and synchronisation latency
        _frame("thumbnail", "cornell", 64, 64, 1, host=True),
        # an ordinary still of a small scene
        _frame("cornell_still", "cornell", 256, 256, 16),
        # one frame of a progressive view of the analytic shapes, odd size, the other sampler, environment light
        # and Russian roulette
        _frame("spheres_view", "spheres", 637, 479, 4, sampler=PCG, env=True, roulette=True),
        # one frame of a progressive view of the 1.2 M-triangle scene, a ragged resolution
        _frame("instanced_view", "instanced", 1277, 717, 1),
        # the headline render: 1080p, 64 samples
        _frame("instanced_1080p", "instanced", 1920, 1080, 64),
        # fog and procedural smoke, delta tracking, with the sun
        _frame("volumetric_720p", "volumetric", 1280, 720, 16, media=True, sun=True),
        # the smoke as a 128^3 float16 density grid, odd size
        _frame("smoke_grid", "volumetric", 957, 541, 8, media=True, grid=True),
        # every solid texture node, bump and normal maps, a noise-density medium
        _frame("textured_720p", "textured", 1280, 720, 8, media=True),
        # image textures on surfaces alone, environment light
        _frame("images_vga", "imaged", 640, 480, 16, env=True),
        # many small previews in one call
        {"name": "previews", "kind": "batch", "count": 48, "smallest": 64, "spp": 8},
        # gradients for albedo and roughness: several views, forward with records and backward
        {"name": "gradients", "kind": "gradient", "scene": "instanced", "views": 4, "size": 512, "spp": 16},
        # the same in a fog whose density grid is differentiated too
        {"name": "gradients_fog", "kind": "gradient", "scene": "instanced_fog", "views": 4, "size": 256, "spp": 8},
    ]


# Most paths (pixels times samples) a drawn render of each scene has: as many as the listed one of its kind.
MOST_PATHS = {"cornell": 1 << 25, "spheres": 1 << 24, "imaged": 1 << 23, "glossy": 1 << 25, "instanced": 1920 * 1080 * 64,
              "volumetric": 1280 * 720 * 16, "textured": 1280 * 720 * 8}


def draw(rng):
    def spread(lo, hi):
        return int(round(float(lo) * (float(hi) / float(lo)) ** rng.random()))

    kind = rng.choice(["frame", "frame", "frame", "frame", "frame", "batch", "gradient"])
    if kind == "batch":
        return {"kind": "batch", "count": spread(4, 48), "smallest": rng.choice([48, 64, 100]), "spp": spread(1, 8)}
    if kind == "gradient":
        scene = rng.choice(["instanced", "instanced_fog"])
        return {"kind": "gradient", "scene": scene, "views": rng.randint(1, 4), "size": spread(63, 256),
                "spp": spread(1, 8)}
    scene = rng.choice(["cornell", "spheres", "imaged", "glossy", "instanced", "instanced", "volumetric", "volumetric",
                        "textured"])
    most = MOST_PATHS[scene]
    width = spread(64, 1920)
    height = max(48, min(1080, int(width * rng.choice([0.5625, 0.75, 1.0, 0.617]))))
    spp = max(1, min(spread(1, 64), most // (width * height)))
    media = scene in ("volumetric", "textured", "spheres") and rng.random() < 0.8
    return {"kind": "frame", "scene": scene, "width": width, "height": height, "spp": spp,
            "sampler": rng.choice([HALTON, HALTON, HALTON, PCG]), "media": media,
            "sun": scene == "volumetric" and rng.random() < 0.5,
            "env": rng.random() < 0.3, "roulette": rng.random() < 0.2,
            "grid": media and scene == "volumetric" and rng.random() < 0.4, "host": rng.random() < 0.2}


# ------------------------------------------------------------------ states ---

_folder = None


@functools.lru_cache(maxsize=None)
def _scene_file(scene: str, layout: int) -> str:
    """The generated scene file, as a user has it on disk (written once per process)."""
    global _folder
    if _folder is None:
        _folder = tempfile.TemporaryDirectory(prefix="ymrt_cases_")
    return scenes.scene_path(scene, layout, os.path.join(_folder.name, scene))


def _layout(scene: str, seed: int) -> int:
    # the 1.2 M-triangle scenes take a second to write: four layouts of them, and the permutations differ anyway
    return seed % 4 if scene.startswith("instanced") else seed % 1000


def _upload(ctx, scene, seed, width, height, perm, camera=None):
    return Y.Scene(ctx, Y.HostScene(_scene_file(scene, _layout(scene, seed)), width, height, camera=camera), perm)


def _image(width, height):
    return torch.zeros((height, width, 4), dtype=torch.float32, device="cuda")


def _density_node(host) -> int:
    """The texture node the scene's smoke reads its density from (word 6 of a volume's record)."""
    return next(int(v[6]) for v in host.records("volumes") if int(v[6]) != 0xFFFFFFFF)


def _previews(case):
    """Resolutions and samples of a batch's renders (the same for every seed)."""
    rng = np.random.default_rng(case["count"] * 1000 + case["smallest"])
    s = case["smallest"]
    sizes = [(s, s), (2 * s, 2 * s), (5 * s // 2, 15 * s // 8), (4 * s, 4 * s)]
    out = []
    for k in range(case["count"]):
        w, h = sizes[int(rng.integers(0, len(sizes)))]
        kind = "instanced" if k % 24 == 23 else "cornell"
        out.append((kind, w, h, int(rng.integers(1, case["spp"] + 1))))
    return out


def prepare(case, seed):
    perm = scenes.halton_permutations(seed)
    ctx = Y.Context(0)
    if case["kind"] == "frame":
        w, h = case["width"], case["height"]
        sc = _upload(ctx, case["scene"], seed, w, h, perm)
        if case["grid"]:
            tex = _density_node(sc.host)
            sc.set_density_grid(tex, scenes.fbm_grid(sc, tex, SMOKE), half=True)
        setting = Y.default_setting(spp=case["spp"], ray_depth=DEPTH[case["scene"]], volume=case["media"],
                                    distant_light=case["sun"], env_light=case["env"],
                                    russian_roulette=case["roulette"], sampler_type=case["sampler"])
        return {"kind": "frame", "ctx": ctx, "scene": sc, "setting": setting, "frame": 1 + seed % 3,
                "out": None if case["host"] else _image(w, h)}
    if case["kind"] == "batch":
        renders = []
        for k, (scene, w, h, spp) in enumerate(_previews(case)):
            sc = _upload(ctx, scene, seed + (0 if scene == "instanced" else k), w, h, perm)
            renders.append([sc, Y.default_setting(spp=spp, ray_depth=DEPTH[scene]), 1 + seed % 3, _image(w, h)])
        return {"kind": "batch", "ctx": ctx, "renders": renders}
    # gradients: several cameras on an arc around the scene, one shared material table
    scene, n, size = case["scene"], case["views"], case["size"]
    fog = scene == "instanced_fog"
    layout = _layout(scene, seed)
    views = [_upload(ctx, scene, seed, size, size, perm, camera=scenes.orbit_view(scene, layout, v, n))
             for v in range(n)]
    grid = scenes.smooth_grid(GRID, seed) if fog else None
    if fog:
        for v in views:
            v.set_density_grid(0, grid)
    setting = Y.default_setting(spp=case["spp"], ray_depth=DEPTH[scene], volume=fog)
    renders = [[v, setting, 1 + seed % 3, _image(size, size)] for v in views]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return {"kind": "gradient", "ctx": ctx, "renders": renders,
            "records": [torch.zeros((Y.path_count(r), 4), dtype=torch.float32, device="cuda") for r in renders],
            "targets": [0.5 * torch.rand((size, size, 4), device="cuda", generator=gen) for _ in renders],
            "grads": torch.zeros((views[0].material_params().shape[0], 4), dtype=torch.float32, device="cuda"),
            "grid_grads": torch.zeros(GRID ** 3, dtype=torch.float32, device="cuda") if fog else None}


# --------------------------------------------------------------------- run ---

def run(state):
    if state["kind"] == "frame":
        image, _ = state["scene"].render(state["setting"], state["frame"], out=state["out"])
        return image
    if state["kind"] == "batch":
        Y.render_batch(state["ctx"], state["renders"])
        return [r[3] for r in state["renders"]]
    # a step of an optimisation: forward with records, the L2 loss's gradient, backward
    Y.render_batch(state["ctx"], state["renders"], state["records"])
    dloss = [2.0 * (r[3] - t) for r, t in zip(state["renders"], state["targets"])]
    # the library renders on a stream of its own: dLoss/dImage has to be there before the call
    torch.cuda.current_stream().synchronize()
    Y.render_backward_ex(state["ctx"], state["renders"], state["records"], dloss, material_grads=state["grads"],
                         grid_texture=0 if state["grid_grads"] is not None else None, grid_grads=state["grid_grads"])
    out = {"images": [r[3] for r in state["renders"]], "grads": state["grads"]}
    if state["grid_grads"] is not None:
        out["grid_grads"] = state["grid_grads"]
    return out


# -------------------------------------------------------------------- work ---

# Unique triangles and instances of each scene, and closest-hit and shadow queries per camera path (typical: many
# camera rays of the instanced scene see the background).
TRIANGLES = {"cornell": 14, "glossy": 14, "spheres": 26, "imaged": 28, "textured": 28, "volumetric": 14,
             "instanced": 155662, "instanced_fog": 155674}
QUERIES = {"cornell": 9.0, "glossy": 9.0, "spheres": 9.0, "imaged": 9.0, "textured": 12.0, "volumetric": 16.0,
           "instanced": 1.7, "instanced_fog": 8.0}
NODE_FLOPS = 8 * 20      # one visit of an 8-wide node: three slabs of eight boxes
TRIANGLE_FLOPS = 60      # one watertight triangle test
VERTEX_FLOPS = 400       # one path vertex: frame, lobes, light and direction samples


def _render_work(scene, pixels, spp):
    tris = TRIANGLES[scene]
    visits = 2.0 + np.log(max(tris, 8)) / np.log(8.0)
    per_query = visits * NODE_FLOPS + 2 * TRIANGLE_FLOPS + VERTEX_FLOPS / 3
    # each triangle's corners once (positions, normals), the image once
    return 72.0 * tris + 16.0 * pixels, float(pixels * spp * QUERIES[scene] * per_query)


def work(case):
    if case["kind"] == "frame":
        b, f = _render_work(case["scene"], case["width"] * case["height"], case["spp"])
        return {"bytes": b + (2.0 * SMOKE ** 3 if case["grid"] else 0.0), "flops": f}
    if case["kind"] == "batch":
        parts = [_render_work(s, w * h, spp) for s, w, h, spp in _previews(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    pixels = case["size"] ** 2
    b, f = _render_work(case["scene"], pixels, case["spp"])
    fog = 2 * 4.0 * GRID ** 3 if case["scene"] == "instanced_fog" else 0.0
    # views share the scene's geometry; each path's record is written and read once, dLoss/dImage read once
    n = case["views"]
    tris = 72.0 * TRIANGLES[case["scene"]]
    return {"bytes": tris + n * (b - tris + 2 * 16.0 * pixels * case["spp"] + 16.0 * pixels) + fog, "flops": 2 * n * f}


def exact(case, seed):
    """No value: each pixel is a sum over random paths whose branches (which lobe, which collision, hit or miss at a
    silhouette) hang on the float32 samples and positions, so the same render in 64 bits is another set of paths, and
    a whole renderer in plain torch would take minutes for the smallest of these."""
    return None
