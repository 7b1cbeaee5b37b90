"""The work that users of luce_render_b200 have it do, as measured cases: probes and ray
queries, moved and rebuilt geometry, and renders, each through the package's public entry
points and over the range of sizes it is used at.

``listed()`` names the standing cases, ``draw(rng)`` gives others of the same ranges,
``prepare`` makes what a program holds before the call, ``run`` is one pass, ``work`` the
bytes and operations a pass cannot do without, and ``exact`` the answer of plain 64-bit
arithmetic where there is one (a brute force over all triangles for probes and closest
hits; a Monte Carlo image has none)."""
from __future__ import annotations

import math

import numpy as np
import torch

import luce_render_b200 as lr
from luce_render_b200 import scenes

# The most ray-triangle tests exact() takes on.
EXACT_TESTS = 4.0e10
# Rays a moved or rebuilt scene is asked after the change.
QUERY_RAYS = 32768
# The largest scene: the incoherent generator's 1,048,576 triangles.
LARGEST = 1 << 20

_context = None


def context() -> "lr.Context":
    global _context
    if _context is None:
        _context = lr.Context(0)
    return _context


# ---- the cases ---------------------------------------------------------------------------


def listed() -> list[dict]:
    return [
        # A click in a viewport: one pixel's polygon and distance.
        dict(name="probe_pick", kind="probe", triangles=20000, width=1, height=1, reference=False),
        # A depth and polygon picture of a large scene, as a viewer's selection buffer.
        dict(name="probe_view", kind="probe", triangles=LARGEST, width=640, height=359, reference=False),
        # A tool's few thousand rays (snapping, baking a patch) in host memory, there and back.
        dict(name="rays_host_4k", kind="rays", triangles=LARGEST, rays=4099, any=False, device=False, aim="box"),
        # The incoherent closest-hit workload, resident in device memory.
        dict(name="rays_closest_4m", kind="rays", triangles=LARGEST, rays=1 << 22, any=False, device=True, aim="box"),
        # Visibility of lights from points of a scene (a bake): any-hit rays of finite reach.
        dict(name="rays_occlusion_1m", kind="rays", triangles=200000, rays=1000003, any=True, device=True, aim="lights"),
        # A deforming mesh: every point moved on the device, the trees refit, the scene queried.
        dict(name="refit_1m", kind="refit", triangles=LARGEST),
        # Edited geometry queried without the host's tree: a BVH2 built on the device.
        dict(name="build_200k", kind="build", triangles=200000),
        # A thumbnail or a tuning loop: a small box, a few samples, started over each time.
        dict(name="render_cornell_256", kind="render", scene="cornell", triangles=34, width=256, height=256, samples=4,
             bounces=6, spectral=False, light_tracing=0.0),
        # The glossy Cornell box at its own settings: 12 bounces, light tracing at its default.
        dict(name="render_glossy_512", kind="render", scene="glossy", triangles=15000, width=512, height=500, samples=2,
             bounces=12, spectral=True, light_tracing=0.5),
        # One sample after a camera move in an interactive view of a medium scene.
        dict(name="render_view_720p", kind="render", scene="incoherent", triangles=100000, width=1280, height=719,
             samples=1, bounces=6, spectral=False, light_tracing=0.0),
        # The headline: 1080p, depth 6, spectral, 1,048,576 triangles.
        dict(name="render_incoherent_1080p", kind="render", scene="incoherent", triangles=LARGEST, width=1920,
             height=1080, samples=4, bounces=6, spectral=True, light_tracing=0.0),
        # Many users' scenes in one wavefront: sizes and films as the batched workload draws them.
        dict(name="batch_12", kind="batch", plan=0xBA7C4, members=12, samples=8, bounces=6, pool=1 << 21),
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["probe", "rays", "rays", "refit", "build", "render", "render", "render", "batch"])
    triangles = _log(rng, 1000, LARGEST)
    if kind == "probe":
        pixels = _log(rng, 1, 1 << 20)
        width = max(1, int(math.sqrt(pixels * 16.0 / 9.0)))
        return dict(kind=kind, triangles=triangles, width=width, height=max(1, pixels // width),
                    reference=rng.random() < 0.25)
    if kind == "rays":
        device = rng.random() < 0.75
        return dict(kind=kind, triangles=triangles, rays=_log(rng, 1000, (1 << 22) if device else (1 << 18)),
                    any=rng.random() < 0.4, device=device, aim=rng.choice(["box", "lights", "camera"]))
    if kind in ("refit", "build"):
        return dict(kind=kind, triangles=triangles)
    if kind == "render":
        scene = rng.choice(["cornell", "glossy", "incoherent", "incoherent"])
        pixels = _log(rng, 64 * 64, 1920 * 1080 if scene == "incoherent" else 1024 * 1024)
        aspect = rng.choice([1.0, 4.0 / 3.0, 16.0 / 9.0])
        width = max(16, int(math.sqrt(pixels * aspect)))
        return dict(kind=kind, scene=scene, triangles={"cornell": 34, "glossy": 15000}.get(scene, triangles), width=width,
                    height=max(16, pixels // width), samples=rng.randint(1, 4 if scene != "glossy" else 2),
                    bounces=rng.randint(3, 6 if scene == "incoherent" else 12), spectral=rng.random() < 0.5,
                    light_tracing=0.5 if scene != "incoherent" and rng.random() < 0.5 else 0.0)
    return dict(kind=kind, plan=rng.randint(1, 1 << 20), members=rng.randint(4, 12), samples=rng.randint(1, 8), bounces=rng.randint(4, 6),
                pool=1 << rng.randint(20, 21))


# ---- inputs ------------------------------------------------------------------------------


def _extent(triangles: int) -> float:
    """Half the side of scenes.scene_of_size's box."""
    objects = max(1, int(round(triangles / 1024)))
    return max(50.0 * (objects / 1024.0) ** (1.0 / 3.0), 4.0)


def _geometry(case: dict, seed: int):
    """Meshes, cameras, lights and materials of the case's scene."""
    name = case.get("scene", "incoherent")
    if name == "cornell":
        return (scenes.cornell_meshes(materials=True), [scenes.cornell_camera()], [scenes.cornell_light()],
                scenes.cornell_materials())
    if name == "glossy":
        return scenes.glossy_cornell(4)
    meshes, materials, lights, cam = scenes.scene_of_size(case["triangles"], seed)
    return meshes, [cam], lights, materials


def _view(case: dict, seed: int) -> dict:
    """A view of the case's scene, a little different for every seed."""
    rng = np.random.default_rng(seed + 17)
    jitter = rng.uniform(-1.0, 1.0, 3)
    name = case.get("scene", "incoherent")
    if name == "cornell":
        return dict(position=np.array([0.0, 0.0, 3.0]) + 0.05 * jitter, forward=np.array([0.0, 0.0, -1.0]),
                    tan=math.tan(math.radians(20.0)))
    if name == "glossy":
        return dict(position=np.array([0.0, 1.0, 3.9]) + 0.05 * jitter, forward=np.array([0.0, 0.0, -1.0]), tan=0.3565)
    e = _extent(case["triangles"])
    return dict(position=np.array([0.0, 0.0, 2.6 * e]) + 0.1 * e * jitter, forward=np.array([0.02, -0.01, -1.0]),
                tan=0.3375)


def _frame(case: dict, seed: int) -> "lr.Frame":
    v = _view(case, seed)
    return lr.look_frame(v["position"], v["forward"], (0.0, 1.0, 0.0), v["tan"], case["width"], case["height"])


def _rays(case: dict, seed: int, count: int, device: str) -> torch.Tensor:
    """count x 8 floats: origin, t_min 0, direction, t_max (finite: a tool's reach). `aim`:
    "box" incoherent directions, "lights" toward points on the scene's overhead lights, "camera"
    a pinhole's pixel centres in scanline order."""
    g = torch.Generator(device="cpu").manual_seed(int(seed) * 7 + 5)
    e = _extent(case["triangles"])
    rays = torch.zeros((count, 8), dtype=torch.float32)
    aim = case.get("aim", "box")
    u = torch.rand((count, 5), generator=g, dtype=torch.float32)
    if aim == "camera":
        side = max(1, int(math.isqrt(count)))
        i = torch.arange(count)
        x, y = (i % side).float(), (i // side).float()
        rays[:, 2] = 2.6 * e
        rays[:, 4] = ((x + 0.5) / side - 0.5) * 0.9
        rays[:, 5] = (0.5 - (y + 0.5) / side) * 0.9
        rays[:, 6] = -1.0
        rays[:, 7] = 8.0 * e
    else:
        rays[:, 0:3] = (u[:, 0:3] * 2.0 - 1.0) * e
        if aim == "lights":
            k = torch.randint(0, 4, (count,), generator=g).float() * (0.5 * math.pi)
            target = torch.stack([30.0 * torch.cos(k) + (u[:, 3] - 0.5) * 20.0, torch.full((count,), 70.0),
                                  30.0 * torch.sin(k) + (u[:, 4] - 0.5) * 20.0], 1)
            d = target - rays[:, 0:3]
            length = d.norm(dim=1, keepdim=True)
            rays[:, 4:7] = d / length
            rays[:, 7] = length[:, 0] * 0.999
        else:
            z = 1.0 - 2.0 * u[:, 3]
            r = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
            phi = 2.0 * math.pi * u[:, 4]
            rays[:, 4], rays[:, 5], rays[:, 6] = r * torch.cos(phi), r * torch.sin(phi), z
            rays[:, 7] = 4.0 * e
    return rays.to(device)


def _moved(positions: np.ndarray) -> np.ndarray:
    base = positions.astype(np.float64)
    return np.ascontiguousarray(base + 0.1 * np.sin(0.7 * base[:, [1, 2, 0]]), np.float32)


def _settings(case: dict, seed: int, width: int, height: int, spectral: bool) -> "lr.RenderSettings":
    s = lr.RenderSettings.of(width, height, case["samples"])
    s.max_bounces = case["bounces"]
    s.spectral = 1 if spectral else 0
    s.light_tracing = case.get("light_tracing", 0.0)
    s.seed = seed & 0x7FFFFFFF
    s.c.material = lr.OpenPbr.lambert()
    return s


def _pinned(height: int, width: int) -> np.ndarray:
    """A page-locked image buffer that lives as long as any view of it."""
    return torch.empty((height, width, 4), dtype=torch.float32, pin_memory=True).numpy()


class Queried:
    """Rays in device memory and room for their hits."""

    def __init__(self, case: dict, seed: int, count: int):
        self.rays = _rays(case, seed, count, "cuda")
        self.hits = torch.empty((count, 4), dtype=torch.float32, device="cuda")

    def trace(self, ctx, scene, any_hit: bool) -> dict:
        lr._check(lr.lib.lr_trace_rays_device(ctx.handle, scene.handle, self.rays.data_ptr(), len(self.rays),
                                              self.hits.data_ptr(), lr.TRACE_ANY if any_hit else 0))
        return {"t": self.hits[:, 0], "id": self.hits.view(torch.int32)[:, 1], "uv": self.hits[:, 2:]}


def prepare(case: dict, seed: int) -> dict:
    ctx = context()
    kind = case["kind"]
    state = dict(case=case, ctx=ctx)
    if kind == "batch":
        plan = scenes.batch_plan(case["members"], case["plan"])
        state["batch"] = lr.Batch(ctx, lr.BatchSettings.default(pool=case["pool"], max_bounces=case["bounces"],
                                                                capacity=case["members"]))
        state["members"], state["images"] = [], []
        for i, p in enumerate(plan):
            meshes, materials, lights, cam = scenes.scene_of_size(min(p["triangles"], 100000), seed + i)
            scene = lr.compile_scene(meshes, [cam], lights, materials)
            state["members"].append((lr.GpuScene.upload(ctx, scene), scene,
                                     _settings(case, seed + i, p["side"], p["side"], p["spectral"])))
            state["images"].append(_pinned(p["side"], p["side"]))
        return state
    meshes, cameras, lights, materials = _geometry(case, seed)
    scene = lr.compile_scene(meshes, cameras, lights, materials, trees=kind != "build")
    state["scene"] = scene
    if kind == "render":
        settings = _settings(case, seed, case["width"], case["height"], case["spectral"])
        state["frame"] = _frame(case, seed)
        state["renderer"] = lr.Renderer.create(ctx, scene, settings, state["frame"])
        state["image"] = _pinned(case["height"], case["width"])
        return state
    if kind != "build":
        state["gpu"] = lr.GpuScene.upload(ctx, scene)
    if kind == "probe":
        state["frame"] = _frame(case, seed)
    elif kind == "rays" and not case["device"]:
        state["rays"] = _rays(case, seed, case["rays"], "cpu").numpy()
    else:
        state["query"] = Queried(case, seed, case.get("rays", QUERY_RAYS))
    if kind == "refit":
        state["points"] = torch.from_numpy(_moved(scene.arrays()["positions"])).cuda()
    torch.cuda.synchronize()
    return state


# ---- one pass ----------------------------------------------------------------------------


def run(state: dict):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "probe":
        faces, distances = lr.probe(ctx, state["gpu"], state["frame"], reference=case["reference"])
        return {"faces": faces, "distances": distances}
    if kind == "rays":
        if case["device"]:
            return state["query"].trace(ctx, state["gpu"], case["any"])
        hits = lr.trace_rays(ctx, state["gpu"], state["rays"], any_hit=case["any"])
        return {"t": hits[:, 0], "id": lr.hit_ids(hits), "uv": hits[:, 2:]}
    if kind == "refit":
        state["gpu"].refit(ctx, (state["points"].data_ptr(), len(state["points"])), device=True)
        return state["query"].trace(ctx, state["gpu"], False)
    if kind == "build":
        built = lr.GpuScene.build(ctx, state["scene"])
        out = state["query"].trace(ctx, built, False)
        built.destroy()
        return out
    if kind == "render":
        r = state["renderer"]
        r.restart(state["frame"])
        r.finish()
        return {"image": r.read_into(state["image"])}
    batch = state["batch"]
    members = [batch.add(gpu, scene, settings) for gpu, scene, settings in state["members"]]
    batch.finish()
    images = [batch.read_into(m, image) for m, image in zip(members, state["images"])]
    for m in members:
        batch.remove(m)
    return {"images": images}


# ---- what a pass cannot do without -------------------------------------------------------


def _query_work(rays: int, triangles: int, answer_bytes: int, ray_bytes: int) -> tuple[float, float]:
    """Rays in, answers out, and of the scene at most every triangle once; a descent to one
    leaf a ray: two boxes (24 operations) a level and four triangle tests (50 each)."""
    scene = 48.0 * min(triangles, 4 * rays)
    return rays * float(ray_bytes + answer_bytes) + scene, rays * (24.0 * math.log2(max(2, triangles)) + 200.0)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "probe":
        b, f = _query_work(case["width"] * case["height"], case["triangles"], 8, 0)
    elif kind == "rays":
        b, f = _query_work(case["rays"], case["triangles"], 16, 32)
    elif kind in ("refit", "build"):
        b, f = _query_work(QUERY_RAYS, case["triangles"], 16, 32)
        # Points and indices read; triangle records and (a refit: half a node a triangle, two
        # 48-byte copies; a build: one node a triangle) boxes written.
        t = float(case["triangles"])
        b += 6.0 * t + 12.0 * t + 48.0 * t + 48.0 * t
        f += 60.0 * t
    else:
        if kind == "batch":
            films = [(p["side"] * p["side"], min(p["triangles"], 100000)) for p in scenes.batch_plan(case["members"], case["plan"])]
        else:
            films = [(case["width"] * case["height"], case["triangles"])]
        b = f = 0.0
        for pixels, triangles in films:
            # Half the bounces survive on average; a closest and a shadow ray and some 500
            # operations of shading each; the image out, the scene read once.
            vertices = pixels * case["samples"] * (1.0 + 0.5 * case["bounces"])
            b += 16.0 * pixels + 48.0 * triangles
            f += vertices * (2.0 * (24.0 * math.log2(max(2, triangles)) + 200.0) + 500.0)
    return {"bytes": b, "flops": f}


# ---- the answer in 64 bits ---------------------------------------------------------------


def _triangles(case: dict, seed: int) -> torch.Tensor:
    """The scene's corners in world space, triangles x 3 x 3, moved for a refit."""
    meshes = _geometry(case, seed)[0]
    out = []
    for m in meshes:
        p = m.positions.astype(np.float64)
        if m.transform is not None:
            t = np.asarray(m.transform, np.float64).reshape(4, 3)
            p = p @ t[:3] + t[3]
        p = p.astype(np.float32)
        if case["kind"] == "refit":
            p = _moved(p)
        out.append(p.astype(np.float64)[m.indices])
    return torch.from_numpy(np.concatenate(out)).cuda()


def _closest(o: torch.Tensor, d: torch.Tensor, limit: torch.Tensor, tri: torch.Tensor) -> tuple:
    """The nearest hit of every ray over every triangle (Moller and Trumbore 1997), in 64 bits:
    t (the ray's limit when none), u and v."""
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    chunk = max(1, (1 << 24) // len(tri))
    ts, us, vs = [], [], []
    for i in range(0, len(o), chunk):
        O, D, L = o[i:i + chunk], d[i:i + chunk], limit[i:i + chunk]
        # With s = O - a and det = -(D . n): t = s . n / det, u = (s x D) . e2 / det and
        # v = -(s x D) . e1 / det, where (s x D) . e = (O x D) . e - D . (e x a): products of
        # matrices over (rays x triangles).
        det = -(D @ n.T)
        oxd = torch.linalg.cross(O, D)
        inv = 1.0 / det
        u = (oxd @ e2.T - D @ torch.linalg.cross(e2, a).T) * inv
        v = (oxd @ e1.T - D @ torch.linalg.cross(e1, a).T) * -inv
        t = (O @ n.T - (a * n).sum(1)) * inv
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (t < L[:, None])
        t = torch.where(ok, t, torch.inf)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        ts.append(torch.where(hit, best, L))
        us.append(torch.where(hit, u.gather(1, k[:, None])[:, 0], 0.0))
        vs.append(torch.where(hit, v.gather(1, k[:, None])[:, 0], 0.0))
    return torch.cat(ts), torch.cat(us), torch.cat(vs)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("render", "batch") or case.get("any"):
        return None
    count = case["width"] * case["height"] if kind == "probe" else case.get("rays", QUERY_RAYS)
    if float(count) * case["triangles"] > EXACT_TESTS:
        return None
    if kind == "probe":
        v, w, h = _view(case, seed), case["width"], case["height"]
        ahead = v["forward"] / np.linalg.norm(v["forward"])
        right = np.cross(ahead, (0.0, 1.0, 0.0))
        right /= np.linalg.norm(right)
        above = np.cross(right, ahead)
        half_h, half_w = v["tan"], v["tan"] * w / h
        y, x = np.mgrid[0:h, 0:w]
        fx, fy = (x.reshape(-1, 1) + 0.5) / w * 2.0 - 1.0, 1.0 - (y.reshape(-1, 1) + 0.5) / h * 2.0
        film = torch.from_numpy(ahead + fx * half_w * right + fy * half_h * above).cuda()
        o = torch.from_numpy(v["position"]).cuda().expand(count, 3).contiguous()
        limit = torch.full((count,), float(np.float32(3.0e38)), dtype=torch.float64, device="cuda")
        return {"faces": None, "distances": _closest(o, film, limit, _triangles(case, seed))[0]}
    rays = _rays(case, seed, count, "cuda").double()
    t, u, v = _closest(rays[:, 0:3].contiguous(), rays[:, 4:7].contiguous(), rays[:, 7].contiguous(), _triangles(case, seed))
    return {"t": t, "id": None, "uv": torch.stack([u, v], 1)}
