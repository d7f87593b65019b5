"""The workloads this library's speed is measured on.

Each case is one call (or one frame's calls) that a program makes through the
public entry points, over the range the library is used in: a single picking
ray up to a 1080p path-traced frame and a 16-million-triangle scene rebuilt
for every frame. The scenes are the benchmark's own seeded ones
(meercadraytracer_b200.scenes); a case's seed moves the camera, the rays or
the instances, as a viewer's program does over a scene that stays resident.

  listed()            the fixed cases
  draw(rng)           another case of the same ranges
  prepare(case, seed) what the program holds before the call
  run(state)          the call, and everything it returns
  work(case)          the bytes and operations the call cannot do without
  exact(case, seed)   ray queries answered in 64 bits by brute force
"""
from __future__ import annotations

import functools
import math
from typing import Any, Dict, List, Optional, Tuple

import numpy as np
import torch

from meercadraytracer_b200 import scenes
from meercadraytracer_b200.batch import BatchRenderer, RenderRequest
from meercadraytracer_b200.compile import compile_camera, compile_scene
from meercadraytracer_b200.executors import GpuExecutor
from meercadraytracer_b200.progressive import ProgressiveOptions, ProgressiveRenderer
from meercadraytracer_b200.raytrace import output_srgb, raytrace_compiled, sample_count, trace_settings
from meercadraytracer_b200.types import Tile

Case = Dict[str, Any]

# Triangles of the resident scenes, and the orbits their viewers' cameras are on
# (radius, height), as in the serving loop.
TRIANGLES = {"small": 22_530, "mid": 1_310_720, "soup": 500_000}
ORBIT = {"small": (17.0, 6.0), "mid": (70.0, 32.0), "soup": (34.0, 12.0)}
INSTANCE_TRIANGLES = 20_480
# Queries a path makes on average: camera ray, bounce rays and shadow rays.
QUERIES = {("small", False): 2.3, ("small", True): 3.5, ("mid", False): 2.0, ("mid", True): 2.1,
           ("soup", False): 2.2, ("soup", True): 3.5}


def listed() -> List[Case]:
    return [
        # A mouse click: what is under the cursor.
        {"name": "pick_mid", "kind": "rays", "scene": "mid", "rays": 1, "any": False},
        # Distance measuring or ambient visibility from a program's own rays.
        {"name": "rays_small_40k", "kind": "rays", "scene": "small", "rays": 40_007, "any": False},
        # One pass of one tile, the unit of work of the tile executor protocol.
        {"name": "tile_small_64", "kind": "tile", "scene": "small", "width": 640, "height": 480, "tile_w": 64,
         "tile_h": 64, "pass": 3, "block": 1, "gi": False},
        # The plain still image: raytrace() at its default sample count.
        {"name": "still_small", "kind": "still", "scene": "small", "width": 320, "height": 240, "samples": 16,
         "gi": False, "shadows": "all"},
        # A path-traced draft at an odd window size.
        {"name": "draft_mid_odd", "kind": "still", "scene": "mid", "width": 633, "height": 471, "samples": 7,
         "gi": True, "shadows": "all"},
        # The headline: a path-traced 1080p frame of 1.3 M triangles.
        {"name": "frame_mid_1080p", "kind": "still", "scene": "mid", "width": 1920, "height": 1080, "samples": 64,
         "gi": True, "shadows": "all"},
        # Unstructured geometry with vertex colours: incoherent rays throughout.
        {"name": "frame_soup_720p", "kind": "still", "scene": "soup", "width": 1280, "height": 720, "samples": 4,
         "gi": True, "shadows": "all"},
        # Several viewers' images in one batch, sizes and sample counts mixed.
        {"name": "batch_mixed_12", "kind": "batch", "requests": 12, "gi": True},
        # A viewer after a camera move: preview, then every pass shown.
        {"name": "progressive_small", "kind": "progressive", "scene": "small", "width": 640, "height": 480,
         "samples": 8, "block": 4, "gi": True},
        # Loading a model: the hierarchy over its triangles.
        {"name": "bvh_100k", "kind": "bvh", "triangles": 100_003},
        # An animation frame: instances moved, geometry rebuilt on the device, image traced.
        {"name": "rebuild_1m", "kind": "rebuild", "instances": 64, "width": 512, "height": 512, "samples": 4,
         "bins": 32},
        # The same with 16.4 M triangles.
        {"name": "rebuild_16m", "kind": "rebuild", "instances": 800, "width": 1024, "height": 1024, "samples": 4,
         "bins": 32},
    ]


def _log(rng: Any, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: Any) -> Case:
    kind = rng.choice(["rays", "tile", "still", "still", "still", "still", "batch", "progressive", "bvh", "rebuild",
                       "rebuild"])
    gi = rng.random() < 0.6
    if kind == "rays":
        return {"kind": kind, "scene": rng.choice(["small", "mid"]), "rays": _log(rng, 1, 300_000),
                "any": rng.random() < 0.3}
    if kind == "tile":
        return {"kind": kind, "scene": rng.choice(["small", "mid"]), "width": rng.randint(128, 1920),
                "height": rng.randint(128, 1080), "tile_w": rng.randint(8, 128), "tile_h": rng.randint(8, 128),
                "pass": rng.randint(0, 63), "block": rng.choice([1, 1, 1, 4]), "gi": gi}
    if kind == "still":
        scene = rng.choice(["small", "mid", "mid", "soup"])
        width = _log(rng, 64, 1920)
        height = max(36, min(1080, int(width * rng.uniform(0.5, 1.1))))
        most = (1920 * 1080 * 64 if scene != "soup" else 1280 * 720 * 16) // (width * height)
        return {"kind": kind, "scene": scene, "width": width, "height": height,
                "samples": _log(rng, 1, max(1, min(64, most))), "gi": gi,
                "shadows": rng.choice(["all", "all", "all", "mesh", "none"])}
    if kind == "batch":
        return {"kind": kind, "requests": rng.randint(2, 24), "gi": gi}
    if kind == "progressive":
        return {"kind": kind, "scene": rng.choice(["small", "mid"]), "width": _log(rng, 160, 1280),
                "height": _log(rng, 120, 720), "samples": rng.randint(1, 16), "block": rng.choice([0, 4, 8]), "gi": gi}
    if kind == "bvh":
        return {"kind": kind, "triangles": _log(rng, 1, 300_000)}
    size = _log(rng, 256, 1024)
    return {"kind": kind, "instances": _log(rng, 4, 800), "width": size, "height": max(64, size - rng.randint(0, 99)),
            "samples": rng.randint(1, 4), "bins": rng.choice([16, 32])}


# ------------------------------------------------------------ resident scenes
@functools.lru_cache(maxsize=None)
def _bench(name: str) -> Any:
    if name == "small":
        return scenes.small_scene()
    if name == "mid":
        return scenes.mid_scene()
    return scenes.soup_scene(count=TRIANGLES["soup"])


@functools.lru_cache(maxsize=None)
def _compiled(name: str) -> Any:
    return compile_scene(_bench(name).scene)


@functools.lru_cache(maxsize=None)
def _executor(name: str) -> GpuExecutor:
    """The program's executor for a scene, the scene already resident."""
    ex = GpuExecutor(0)
    ex.load_scene(_compiled(name))
    return ex


@functools.lru_cache(maxsize=None)
def _batch_renderer() -> BatchRenderer:
    r = BatchRenderer(0, capacity=1 << 24, memory_budget=2 << 30)
    for name in ("small", "mid"):
        r.adopt(_compiled(name), _executor(name))
    return r


@functools.lru_cache(maxsize=None)
def _progressive(name: str) -> ProgressiveRenderer:
    return ProgressiveRenderer([GpuExecutor(0)])


@functools.lru_cache(maxsize=None)
def _rebuilder(count: int) -> Tuple[GpuExecutor, Any, int]:
    scene = scenes.large_scene(count=count, box=200.0 * (count / 4096.0) ** (1.0 / 3.0))
    ex = _rebuild_executor()
    ex.upload_meshes([scene.mesh])
    return ex, scene, ex.send_shading_only(scene.shading)


@functools.lru_cache(maxsize=None)
def _rebuild_executor() -> GpuExecutor:
    return GpuExecutor(0)


def _camera(name: str, rng: np.random.Generator, aspect: float) -> Any:
    radius, height = ORBIT[name]
    return scenes.orbit_camera(radius * rng.uniform(0.9, 1.1), height, rng.uniform(0.0, 360.0), aspect=aspect)


def _options(name: str, gi: bool, samples: int, seed: int, shadows: str = "all") -> Dict[str, Any]:
    return dict(_bench(name).options, samples=samples, global_illumination=gi, seed=seed % 65536, shadows=shadows)


def _rays(case: Case, seed: int) -> np.ndarray:
    """[n, 8] floats: camera rays through random points of the view for a few rays, else rays
    from random points around the scene's centre in random directions."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    radius, height = ORBIT[case["scene"]]
    out = np.zeros((n, 8), np.float32)
    if n <= 64:
        angle = rng.uniform(0.0, 2.0 * math.pi)
        origin = np.array([radius * math.sin(angle), height, radius * math.cos(angle)])
        target = rng.uniform(-0.25, 0.25, (n, 3)) * radius
        target[:, 1] = np.abs(target[:, 1]) * 0.2
        d = target - origin
        out[:, 0:3] = origin
    else:
        out[:, 0] = rng.uniform(-0.5, 0.5, n) * radius
        out[:, 1] = rng.uniform(0.1, 0.5, n) * height
        out[:, 2] = rng.uniform(-0.5, 0.5, n) * radius
        d = rng.normal(size=(n, 3))
    out[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return out


def _model_triangles(n: int, seed: int) -> np.ndarray:
    """n triangles as buildBvh takes them (v0, e1, e2): facets scattered over spheres of varying
    size. The seed shuffles them and scales the model by a power of two, so every seed's tree
    has as many nodes."""
    rng = np.random.default_rng(n)
    centre = rng.uniform(-40, 40, (max(1, n // 2000), 3))
    radius = rng.uniform(0.5, 4.0, centre.shape[0])
    k = np.arange(n) % centre.shape[0]
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tri = np.empty((n, 9), np.float32)
    tri[:, 0:3] = centre[k] + d * radius[k, None]
    tri[:, 3:9] = rng.normal(size=(n, 6)) * (0.05 * radius[k, None])
    rng = np.random.default_rng(seed)
    return (rng.permutation(tri) * np.float32(2.0 ** int(rng.integers(-3, 4)))).reshape(-1)


def _batch_requests(case: Case, seed: int) -> List[RenderRequest]:
    rng = np.random.default_rng(seed)
    sizes = [(256, 256), (512, 512), (640, 480), (333, 217)]
    spp = [4, 16, 5]
    out = []
    for i in range(case["requests"]):
        # Sizes and sample counts go round, so every seed's batch is the same amount of work.
        name = "mid" if i % 2 else "small"
        w, h = sizes[(i // 2) % len(sizes)]
        s = spp[i % len(spp)]
        st = trace_settings(_options(name, case["gi"], s, seed + i))
        out.append(RenderRequest(_compiled(name), compile_camera(_camera(name, rng, w / h)), w, h, st, s))
    return out


def prepare(case: Case, seed: int) -> Dict[str, Any]:
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "rays":
        ex = _executor(case["scene"])
        return {"case": case, "ex": ex, "version": ex.load_scene(_compiled(case["scene"]))[0],
                "rays": _rays(case, seed)}
    if kind == "tile":
        name, w, h = case["scene"], case["width"], case["height"]
        ex = _executor(name)
        gv, sv = ex.load_scene(_compiled(name))
        tw, th = min(case["tile_w"], w), min(case["tile_h"], h)
        tile = Tile((w - tw) // 2, (h - th) // 2, tw, th)
        return {"case": case, "ex": ex, "message": {
            "type": "tile", "job": 1, "geometry_version": gv, "shading_version": sv,
            "camera": compile_camera(_camera(name, rng, w / h)),
            "settings": trace_settings(_options(name, case["gi"], 1, seed)), "tile": tile, "width": w, "height": h,
            "pass": case["pass"], "block": case["block"]}}
    if kind == "still":
        name, w, h = case["scene"], case["width"], case["height"]
        return {"case": case, "ex": _executor(name), "scene": _compiled(name),
                "camera": compile_camera(_camera(name, rng, w / h)),
                "options": _options(name, case["gi"], case["samples"], seed, case["shadows"])}
    if kind == "batch":
        return {"case": case, "renderer": _batch_renderer(), "requests": _batch_requests(case, seed)}
    if kind == "progressive":
        name, w, h = case["scene"], case["width"], case["height"]
        opts = _options(name, case["gi"], case["samples"], seed)
        return {"case": case, "renderer": _progressive(name), "scene": _bench(name).scene,
                "camera": _camera(name, rng, w / h),
                "options": ProgressiveOptions(w, h, trace_settings(opts), samples=case["samples"],
                                              preview_block=case["block"])}
    if kind == "bvh":
        return {"case": case, "ex": _executor("small"), "triangles": _model_triangles(case["triangles"], seed)}
    ex, scene, shading = _rebuilder(case["instances"])
    camera = scenes.orbit_camera(scene.box * 1.6, scene.box * 0.35, float(rng.uniform(0.0, 360.0)),
                                 aspect=case["width"] / case["height"])
    options = dict(scene.options, samples=case["samples"], seed=seed % 65536)
    return {"case": case, "ex": ex, "mesh": scene.mesh, "instances": scene.frame(seed), "shading": shading,
            "camera": compile_camera(camera), "options": options, "settings": trace_settings(options)}


def run(state: Dict[str, Any]) -> Any:
    case = state["case"]
    kind = case["kind"]
    if kind == "rays":
        if case["any"]:
            return state["ex"].intersect_any_count(state["version"], state["rays"])
        return state["ex"].intersect_closest(state["version"], state["rays"])
    if kind == "tile":
        return state["ex"].render(state["message"]).result()
    if kind == "still":
        return raytrace_compiled(state["scene"], state["camera"], case["width"], case["height"], state["options"],
                                 executor=state["ex"]).data
    if kind == "batch":
        return state["renderer"].render(state["requests"])
    if kind == "progressive":
        frames = []
        state["renderer"].render(state["scene"], state["camera"], state["options"], frames.append)
        return frames[-1].image
    if kind == "bvh":
        bvh, order = state["ex"].build_bvh(state["triangles"], case["triangles"])
        return {"bounds": bvh.bounds, "nodes": bvh.nodes, "order": order.astype(np.int64)}
    ex = state["ex"]
    info, _ = ex.compile_instances(state["instances"], bins=case["bins"])
    image = ex.raytrace_resident((info["version"], state["shading"]), state["camera"], case["width"], case["height"],
                                 state["settings"], sample_count(state["options"]), output_srgb(state["options"]))
    return {"image": image, "triangles": info["triangle_count"], "nodes": info["node_count"]}


# ------------------------------------------------------------------- the work
def _query_flops(triangles: int) -> float:
    """One query in a binary hierarchy over leaves of two or three triangles: two box tests of 24
    operations per level of a balanced tree and two triangle tests of 60."""
    return 48.0 * max(1.0, math.log2(max(2.0, triangles / 2.5))) + 120.0


def _scene_bytes(triangles: int) -> float:
    """Vertices, normals, uvs and flags of every triangle and a node per leaf."""
    return triangles * (36.0 + 36.0 + 24.0 + 6.0 + 64.0 / 2.5)


def _render_work(triangles: int, samples: float, queries: float, image_bytes: float) -> Dict[str, float]:
    """samples paths: their queries, and 300 operations per path for the camera and shading."""
    return {"bytes": _scene_bytes(triangles) + image_bytes,
            "flops": samples * (queries * _query_flops(triangles) + 300.0)}


def _build_work(triangles: int, out_bytes: float) -> Dict[str, float]:
    """Every triangle read once and every output written once; per triangle and level of the
    tree its bin on three axes and its box joined to the bin's (40 operations)."""
    levels = max(1.0, math.log2(max(2.0, triangles / 2.5)))
    return {"bytes": triangles * (36.0 + out_bytes), "flops": 40.0 * triangles * levels}


def work(case: Case) -> Dict[str, float]:
    kind = case["kind"]
    if kind == "rays":
        n, t = case["rays"], TRIANGLES[case["scene"]]
        # A few rays read a path through the hierarchy, many rays all of it.
        return {"bytes": n * 48.0 + min(_scene_bytes(t), n * 1200.0), "flops": n * _query_flops(t)}
    if kind == "tile":
        w, h = min(case["tile_w"], case["width"]), min(case["tile_h"], case["height"])
        paths = math.ceil(w / case["block"]) * math.ceil(h / case["block"])
        q = QUERIES[(case["scene"], case["gi"])]
        t = TRIANGLES[case["scene"]]
        d = _render_work(t, paths, q, 0.0)
        return {"bytes": min(_scene_bytes(t), paths * q * 1200.0) + w * h * 16.0, "flops": d["flops"]}
    if kind in ("still", "progressive"):
        px = case["width"] * case["height"]
        return _render_work(TRIANGLES[case["scene"]], px * case["samples"], QUERIES[(case["scene"], case["gi"])],
                            px * 4.0)
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        sizes, spp = [256 * 256, 512 * 512, 640 * 480, 333 * 217], [4, 16, 5]
        for i in range(case["requests"]):
            name = "mid" if i % 2 else "small"
            px = sizes[(i // 2) % 4]
            d = _render_work(TRIANGLES[name], px * spp[i % 3], QUERIES[(name, case["gi"])], px * 4.0)
            total["flops"] += d["flops"]
            total["bytes"] += px * 4.0
        total["bytes"] += _scene_bytes(TRIANGLES["small"]) + _scene_bytes(TRIANGLES["mid"])
        return total
    if kind == "bvh":
        return _build_work(case["triangles"], 40.0)
    t = case["instances"] * INSTANCE_TRIANGLES
    px = case["width"] * case["height"]
    b = _build_work(t, 102.0 + 64.0 / 2.5)
    d = _render_work(t, px * case["samples"], 2.0, px * 4.0)
    return {"bytes": b["bytes"] + d["bytes"], "flops": b["flops"] + d["flops"]}


# ------------------------------------------------------------- 64-bit answers
def exact(case: Case, seed: int) -> Optional[Dict[str, Any]]:
    """The nearest hit of every ray by testing every triangle in double (Moller-Trumbore), where
    that is quick; images and trees have no such value."""
    if case["kind"] != "rays" or case["any"]:
        return None
    t_count = TRIANGLES[case["scene"]]
    if case["rays"] * t_count > 2_000_000_000:
        return None
    g = _compiled(case["scene"]).geometry
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tri = torch.from_numpy(np.asarray(g.triangles, np.float64).reshape(-1, 9)).to(dev)
    side = torch.from_numpy(np.asarray(g.sides, np.int64)).to(dev)
    rays = torch.from_numpy(_rays(case, seed).astype(np.float64)).to(dev)
    v0 = tri[:, 0:3]
    # The vertices are what a hit is tested against: float32, as the scene holds them.
    e1 = (v0 + tri[:, 3:6]).float().double() - v0
    e2 = (v0 + tri[:, 6:9]).float().double() - v0
    best_t = torch.zeros(case["rays"], dtype=torch.float64, device=dev)
    best_u = torch.zeros_like(best_t)
    step = max(1, 40_000_000 // t_count)
    normal = torch.linalg.cross(e1, e2)
    for a in range(0, case["rays"], step):
        o, d = rays[a:a + step, 0:3], rays[a:a + step, 4:7]
        # With n = e1 x e2 and s = o - v0: det = -d.n, t = s.n / det, and the weights of v1 and v2
        # from the ray's moment m = o x d, all as matrix products over [rays, triangles].
        det = -(d @ normal.T)
        s_n = o @ normal.T - (v0 * normal).sum(1)
        m = torch.linalg.cross(o, d)
        u = (m @ e2.T + d @ torch.linalg.cross(v0, e2).T) / det
        v = -(m @ e1.T + d @ torch.linalg.cross(v0, e1).T) / det
        t = s_n / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (det != 0)
        ok &= ~((side == 0)[None, :] & (det < 0)) & ~((side == 1)[None, :] & (det > 0))
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        tm, k = t.min(1)
        hit = torch.isfinite(tm)
        best_t[a:a + step] = torch.where(hit, tm, torch.zeros_like(tm))
        uu = u.gather(1, k[:, None])[:, 0]
        best_u[a:a + step] = torch.where(hit, uu, torch.zeros_like(uu))
    return {"tri": None, "t": best_t.cpu().numpy(), "u": best_u.cpu().numpy(), "front": None}
