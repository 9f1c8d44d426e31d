"""The work that a user of ntrace has it do, as measurable cases.

Each case is a call that a program makes through the public Python API (math_b200.ntrace, which mirrors
the C ABI call for call, and math_b200.denoise): frames and pixel lists rendered, ray sets traced,
scenes built, batches of scenes, and the denoiser's inputs, inference and training.  Sizes are those of
scenes.config, bench.py, math_b200.batched and math_b200.train_denoiser, or generic ones between them.

`listed` names the cases, `draw` gives more of the same ranges, `prepare` makes what a program has in
hand before the call, `run` is the call, `work` its unavoidable bytes and operations, `tolerance` how
far another correct implementation may be off, and `exact` the same outputs in 64-bit torch where they
have such a value.

Meshes are closed or open surfaces around the origin, turned by a rotation of the seed; the light, the
albedos and the view come from the seed too, as in the denoiser's scene variations.
"""

from __future__ import annotations

import itertools
import math
import os
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

os.environ.setdefault("NTRACE_NO_BUILD", "1")  # the library as built, never rebuilt by an import

from math_b200 import denoise, ntrace, scenes  # noqa: E402

WEIGHTS = Path(denoise.__file__).resolve().parent / "weights"
MAX_DEPTH = 5


def listed() -> list[dict]:
    return [
        # the smallest whole render: a preview of a coarse mesh; latency and launches
        dict(name="frame_n3_small", kind="frame", n=3, mesh="ico", size=2, screen="48x48", spp=16, pool=0),
        # the n = 3 configuration: a 20,480-triangle sphere, 400 x 400 pixels
        dict(name="frame_n3", kind="frame", n=3, mesh="ico", size=5, screen="400x400", spp=16, pool=0),
        # the headline workload: 675,461 tetrahedra, 128^3 pixels at 27 samples, the pool a frame loop tunes to
        dict(name="frame_n4", kind="frame", n=4, mesh="hull", size=100_000, screen="128x128x128", spp=16, pool=1 << 25),
        # an open n = 5 mesh under ragged axes near the configuration's screen, the default pool
        dict(name="frame_n5", kind="frame", n=5, mesh="open", size=3, screen="48x33x29x41", spp=4, pool=0),
        # a pixel list of an n = 6 scene (a region looked at closely; convergence checks)
        dict(name="pixels_n6", kind="pixels", n=6, mesh="cube", size=1, screen="12x11x12x9x13", spp=200, count=3001),
        # two meshes, vertex normals, perspective: the scene types outside the one-mesh path
        dict(name="smooth_n3", kind="smooth", n=3, size=4, screen="320x241", spp=9),
        # closest hits of a given ray set, device arrays
        dict(name="rays_n4", kind="rays", n=4, mesh="hull", size=10_000, count=300_007),
        # scenes of several dimensions side by side in one graph
        dict(name="batch_mixed", kind="batch", plan=11, scenes=7, scale=1.0),
        # a mesh made renderable: facet setup and the tree, built on the GPU
        dict(name="build_n4", kind="build", n=4, mesh="hull", size=8_000),
        # the denoiser's inputs: per-pixel moments, first-hit normal and depth
        dict(name="inputs_n3", kind="inputs", n=3, mesh="ico", size=5, screen="400x400", spp=4),
        # inference on a whole n = 4 frame (the committed weights)
        dict(name="denoise_n4", kind="denoise", n=4, screen="128x128x128", spp=8),
        # a training step on one n = 4 crop
        dict(name="train_n4", kind="train", n=4, screen="24x24x24", spp=8),
    ]


# facets per hull point, measured on the configuration meshes, and the screens, meshes and samples of
# the drawn cases per dimension: (pixels per axis, mesh sizes of kind "cube", samples)
HULL_FACETS = {3: 2.0, 4: 6.75, 5: 31.0, 6: 110.0}
DRAW_SCREEN = {3: (40, 480), 4: (12, 100), 5: (7, 36), 6: (5, 13)}
DRAW_CUBE = {3: (6, 60), 4: (3, 12), 5: (2, 3), 6: (1, 1)}


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame", "frame", "frame", "pixels", "smooth", "rays", "batch", "build", "inputs", "denoise",
                       "train"])
    n = rng.choice([3, 3, 3, 4, 4, 4, 5, 5, 6])  # a tree at n = 6 takes seconds to build
    if kind == "smooth":
        return dict(kind=kind, n=3, size=rng.choice([2, 3, 4]), spp=rng.choice([1, 4, 9, 16]),
                    screen="%dx%d" % (_log(rng, 40, 400), _log(rng, 40, 400)))
    if kind == "batch":
        return dict(kind=kind, plan=rng.randrange(1 << 20), scenes=rng.randint(2, 8), scale=rng.uniform(0.2, 1.0))
    axes = [_log(rng, *DRAW_SCREEN[n]) for _ in range(n - 1)]
    screen = "x".join(map(str, axes))
    if kind == "denoise":
        return dict(kind=kind, n=n, screen=screen, spp=rng.choice([1, 2, 3]) ** (n - 1))
    if kind == "train":
        axes = [max(6, a // 2) for a in axes]
        return dict(kind=kind, n=n, screen="x".join(map(str, axes)), spp=rng.choice([1, 2, 3]) ** (n - 1))
    mesh = rng.choice(["cube", "open", "hull"] if n <= 4 else ["cube", "open"])
    size = _log(rng, 500, 10_000) if mesh == "hull" else _log(rng, *DRAW_CUBE[n])
    if kind == "rays":
        return dict(kind=kind, n=n, mesh=mesh, size=size, count=_log(rng, 2_000, 2_000_000))
    if kind == "build":
        return dict(kind=kind, n=n, mesh=mesh, size=size)
    if kind == "pixels":
        return dict(kind=kind, n=n, mesh=mesh, size=size, screen=screen, spp=_log(rng, 16, 1000),
                    count=_log(rng, 100, 4000))
    case = dict(kind=kind, n=n, mesh=mesh, size=size, screen=screen, spp=_log(rng, 1, 27))
    if kind == "frame":
        case["pool"] = rng.choice([0, 0, 1 << 20, 1 << 24])
    # no more paths than the headline frame has
    while math.prod(axes) * _spp(n, case["spp"]) > 50_000_000 and case["spp"] > 1:
        case["spp"] = max(1, case["spp"] // 2)
    return case


# ------------------------------------------------------------------------------------------------
# meshes


def _cube_sphere(n: int, k: int) -> tuple[np.ndarray, np.ndarray]:
    """The boundary of the n-cube, each face cut into k^(n-1) cells and each cell into (n-1)! simplices
    (one per order of its axes), projected to the unit sphere: 2 n k^(n-1) (n-1)! facets."""
    m = n - 1
    cells = np.stack(np.meshgrid(*[np.arange(k)] * m, indexing="ij"), -1).reshape(-1, m)
    corners = []
    for order in itertools.permutations(range(m)):
        steps = np.zeros((m + 1, m), np.int64)
        for i, axis in enumerate(order):
            steps[i + 1] = steps[i]
            steps[i + 1, axis] += 1
        corners.append(cells[:, None, :] + steps[None])
    grid = np.concatenate(corners)  # simplices x n vertices x m grid coordinates
    faces = []
    for axis in range(n):
        for side in (0, k):
            faces.append(np.insert(grid, axis, side, axis=2))
    points = np.concatenate(faces).reshape(-1, n)
    key = (points * (k + 1) ** np.arange(n)).sum(1)
    uniq, first, inverse = np.unique(key, return_index=True, return_inverse=True)
    v = np.tan((points[first] * (2.0 / k) - 1.0) * (math.pi / 4))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return v, inverse.reshape(-1, n).astype(np.int32)


@lru_cache(maxsize=None)
def _mesh(mesh: str, n: int, size: int) -> tuple[np.ndarray, np.ndarray]:
    if mesh == "ico":
        v, f = scenes.icosphere(size)
    elif mesh == "hull":
        v, f = scenes.sphere_hull(n, size, seed=0)
    else:
        v, f = _cube_sphere(n, size)
    return np.asarray(v, np.float64), f


def _facet_count(case: dict) -> int:
    n, size = case["n"], case["size"]
    if case.get("mesh", "ico") == "ico":
        return 20 * 4 ** size
    return int(HULL_FACETS[n] * size) if case["mesh"] == "hull" else 2 * n * size ** (n - 1) * math.factorial(n - 1)


def _turned(mesh: str, n: int, size: int, rng: np.random.Generator) -> tuple[np.ndarray, np.ndarray]:
    """The mesh under a rotation of the seed; "open": without the facets around +x_(n-1)."""
    v, f = _mesh(mesh, n, size)
    q, r = np.linalg.qr(rng.standard_normal((n, n)))
    v = v @ (q * np.sign(np.diag(r)))
    if mesh == "open":
        c = v[f].mean(1)
        f = f[c[:, n - 1] < 0.88 * np.linalg.norm(c, axis=1)]
        used, f = np.unique(f, return_inverse=True)
        v, f = v[used], f.reshape(-1, n).astype(np.int32)
    return np.ascontiguousarray(v, np.float32), np.ascontiguousarray(f)


# ------------------------------------------------------------------------------------------------
# scenes


def _screen(case: dict) -> tuple[int, ...]:
    return tuple(int(x) for x in case["screen"].split("x"))


def _spp(n: int, spp: int) -> int:
    return scenes.effective_spp(n, spp)


def _spec(case: dict, seed: int) -> dict:
    """The scene as plain arrays: mesh, floor slab, point light, view, albedos."""
    n = case["n"]
    rng = np.random.default_rng([seed, 17])
    if case.get("kind") == "build":
        # one shape, its facets in the seed's order: trees of the same size, their lists different
        verts, facets = _turned(case["mesh"], n, case["size"], np.random.default_rng(3))
        facets = rng.permutation(facets)
    else:
        verts, facets = _turned(case.get("mesh", "ico"), n, case["size"], rng)
    view = denoise.random_variant(n, rng, 2)
    screen = _screen(case) if "screen" in case else (16,) * (n - 1)
    org, edges = scenes.floor_slab(n)
    return dict(n=n, verts=verts, facets=facets, light=view["light"], mesh_albedo=view["mesh_albedo"],
                floor_albedo=view["floor_albedo"], dir=view["dir"], org=view["org"],
                axes=denoise.screen_axes(view["dir"]), param=8.0 / max(screen), screen=screen, floor=(org, edges))


def _scene(spec: dict, *, smooth: dict | None = None) -> ntrace.Scene:
    n = spec["n"]
    s = ntrace.Scene(n)
    a, b = spec["mesh_albedo"], spec["floor_albedo"]
    s.add_mesh(spec["verts"], spec["facets"], color=(a, a, a))
    if smooth:
        s.set_mesh_normals(0, smooth["normals"])
        s.add_mesh(smooth["verts2"], smooth["facets2"], color=(b, a, a))
    s.add_parallelotope(*spec["floor"], color=(b, b, b))
    s.add_point_light(spec["light"], (1.0, 1.0, 1.0), float(np.linalg.norm(spec["light"].astype(np.float64))))
    if smooth:
        s.set_projector(ntrace.PERSPECTIVE, spec["org"] * 0.5, spec["dir"], spec["axes"], 55.0, spec["screen"])
    else:
        s.set_projector(ntrace.PARALLEL, spec["org"], spec["dir"], spec["axes"], spec["param"], spec["screen"])
    s.set_background(scenes.BACKGROUND, True, scenes.BACKGROUND_LIGHT)
    s.build(tree_on_gpu=True)
    return s


def _batch_plan(case: dict) -> list[dict]:
    """The scenes of a batch: n = 3, 4, 5 in turn, sizes from the case's plan number."""
    rng = np.random.default_rng(case["plan"])
    plan = []
    for i in range(case["scenes"]):
        n = 3 + i % 3
        lo, hi = DRAW_SCREEN[n]
        hi = max(lo + 1, int(hi * case["scale"]))
        axes = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(n - 1)]
        lo, hi = DRAW_CUBE[n] if n < 5 else (2, 2)
        plan.append(dict(n=n, mesh="cube", size=int(rng.integers(lo, hi + 1)), screen="x".join(map(str, axes)),
                         spp=int(rng.integers(1, 9))))
    return plan


def _pinned(rows: int) -> np.ndarray:
    return torch.empty((rows, 3), dtype=torch.float32, pin_memory=True).numpy()


def _rays(case: dict, spec: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """A camera's parallel rays, rays from around the mesh, and rays leaving points near its surface."""
    n, count = case["n"], case["count"]
    g = torch.Generator("cuda").manual_seed(seed)
    unit = lambda m: torch.nn.functional.normalize(torch.randn((m, n), generator=g, device="cuda"), dim=1)  # noqa: E731
    a, b = count // 4, count // 2
    c = count - a - b
    d = torch.from_numpy(spec["dir"]).cuda()
    lateral = (torch.rand((a, n - 1), generator=g, device="cuda") * 2.4 - 1.2) @ torch.from_numpy(spec["axes"]).cuda()
    org = [lateral - 10.0 * d, unit(b) * (1.5 + 2 * torch.rand((b, 1), generator=g, device="cuda")), unit(c) * 1.001]
    aim = unit(b) * 1.05 * torch.rand((b, 1), generator=g, device="cuda") ** (1.0 / n)
    out = unit(c)
    out = torch.where((out * org[2]).sum(1, keepdim=True) < 0, -out, out) - 0.3 * org[2]
    return torch.cat(org).contiguous(), torch.cat([d.expand(a, n), aim - org[1], out]).contiguous()


def _noisy_image(case: dict, seed: int) -> dict:
    """A noisy render's stand-in: smooth shading with an object's silhouette, Monte Carlo noise of the
    sample count, normals and depth of the silhouette."""
    n, screen, spp = case["n"], _screen(case), case["spp"]
    g = torch.Generator("cuda").manual_seed(seed)
    rand = lambda *s: torch.rand(s, generator=g, device="cuda")  # noqa: E731
    pix = torch.arange(math.prod(screen), device="cuda")
    x = []
    for size in screen:
        x.append((pix % size).float() / size * 2 - 1)
        pix = pix // size
    x = torch.stack(x, 1)
    radius = (x - 0.4 * (rand(n - 1) - 0.5)).norm(dim=1)
    inside = (radius < 0.6).float()[:, None]
    target = 0.35 + 0.15 * torch.sin(4 * x @ (rand(n - 1, 3) - 0.5) * 2 + 6 * rand(3)) + 0.25 * inside * (1 - radius[:, None])
    sigma = 0.3 / math.sqrt(spp) * (0.4 + rand(len(x), 3))
    noise = torch.randn((len(x), 3), generator=g, device="cuda")
    normal = torch.cat([x, (0.36 - radius * radius).clamp(min=0.0).sqrt()[:, None] + 0.01], 1) * inside
    normal[:, -1] += 1 - inside[:, 0]
    normal = torch.nn.functional.normalize(normal, dim=1)
    return dict(mean=(target + sigma * noise).clamp(min=0.0), var=(sigma * (0.7 + 0.6 * rand(len(x), 3))) ** 2,
                normal=normal.contiguous(), depth=(11.0 - 1.5 * inside[:, 0] * (1 - radius)).contiguous(),
                target=target.contiguous())


def _denoiser(case: dict, seed: int) -> denoise.Denoiser:
    """Inference takes the committed weights where there are some; training starts from new ones."""
    path = WEIGHTS / f"denoiser_n{case['n']}.npz"
    return denoise.Denoiser.load(path) if case["kind"] == "denoise" and path.exists() else denoise.Denoiser(case["n"], seed)


# ------------------------------------------------------------------------------------------------
# the calls


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    state = dict(case=case, kind=kind, seed=seed)
    if kind in ("frame", "inputs", "pixels"):
        spec = _spec(case, seed)
        scene = state["scene"] = _scene(spec)
        rows = scene.pixel_count
        if kind == "frame":
            state["out"] = _pinned(rows)
        elif kind == "pixels":
            rng = np.random.default_rng([seed, 5])
            state["pixels"] = np.sort(rng.choice(rows, min(rows, case["count"]), replace=False)).astype(np.int64)
        else:
            new = lambda *s: torch.empty(s, dtype=torch.float32, device="cuda")  # noqa: E731
            state.update(mean=new(rows, 3), var=new(rows, 3), normal=new(rows, case["n"]), depth=new(rows))
    elif kind == "smooth":
        spec = _spec(case, seed)
        ball, facets = _turned("ico", 3, 2, np.random.default_rng([seed, 3]))
        state["scene"] = _scene(spec, smooth=dict(normals=spec["verts"], facets2=facets,
                                                  verts2=ball * np.float32(0.5) + np.float32([1.4, 1.0, -0.4])))
        state["out"] = _pinned(state["scene"].pixel_count)
    elif kind == "rays":
        spec = _spec(case, seed)
        state["scene"] = _scene(spec)
        state["org"], state["dir"] = _rays(case, spec, seed)
        state["facet"] = torch.empty(case["count"], dtype=torch.int32, device="cuda")
        state["t"] = torch.empty(case["count"], dtype=torch.float32, device="cuda")
    elif kind == "batch":
        plan = _batch_plan(case)
        state["scenes"] = [_scene(_spec(p, seed + 101 * i)) for i, p in enumerate(plan)]
        state["opts"] = [dict(samples_per_pixel=p["spp"], max_depth=MAX_DEPTH, seed=seed + i) for i, p in enumerate(plan)]
        state["out"] = [_pinned(s.pixel_count) for s in state["scenes"]]
    elif kind == "build":
        state["spec"] = _spec(case, seed)
    else:
        state["image"] = _noisy_image(case, seed)
        state["den"] = _denoiser(case, seed)
        state["out"] = torch.empty_like(state["image"]["mean"])
    return state


def run(state: dict):
    kind, case, seed = state["kind"], state["case"], state["seed"]
    if kind in ("frame", "smooth"):
        scene = state["scene"]
        scene.clear()
        scene.render(case["spp"], max_depth=MAX_DEPTH, seed=seed, pool_paths=case.get("pool", 0),
                     smooth_normal=kind == "smooth")
        return scene.image(state["out"])[0]
    if kind == "pixels":
        return state["scene"].render_pixels(state["pixels"], case["spp"], max_depth=MAX_DEPTH, seed=seed)[0]
    if kind == "inputs":
        scene = state["scene"]
        out = [state[k] for k in ("mean", "var", "normal", "depth")]
        scene.render_moments(case["spp"], out[0].data_ptr(), out[1].data_ptr(), max_depth=MAX_DEPTH, seed=seed)
        scene.render_aux(out[2].data_ptr(), out[3].data_ptr())
        return out
    if kind == "rays":
        state["scene"].trace_closest_device(state["org"].data_ptr(), state["dir"].data_ptr(), len(state["t"]),
                                            state["facet"].data_ptr(), state["t"].data_ptr())
        return [state["t"], state["facet"]]
    if kind == "batch":
        for s in state["scenes"]:
            s.clear()
        ntrace.render_batch(state["scenes"], state["opts"])
        return [s.image(o)[0] for s, o in zip(state["scenes"], state["out"])]
    if kind == "build":
        scene = _scene(state["spec"])
        tree = scene.tree_export()
        scene.close()
        return [tree["nodes"], tree["indices"]]
    den, image = state["den"], state["image"]
    den.set_input(_screen(case), image["mean"], image["var"], image["normal"], image["depth"], case["spp"])
    if kind == "denoise":
        return den.apply(state["out"])
    loss = den.train_step(image["target"], 1e-3)
    return [loss, den.get_params()]


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without


def _trace_work(case: dict, paths: int, outputs: int) -> tuple[float, float]:
    """The mesh read once (indices and vertices), `outputs` values written; per path about four rays
    (extension and shadow, as counted on the configuration scenes), each with two box tests and one
    facet test."""
    n = case["n"]
    f = _facet_count(case)
    return f * n * 4 * 1.25 + outputs * 4, paths * 4.0 * (2 * 8 * n + 2 * n * n + 4 * n)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(p, kind="frame")) for p in _batch_plan(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["n"]
    if kind == "build":
        # facets and vertices in; per facet its FP64 record and the nodes and list entries it makes out
        f = _facet_count(case)
        return dict(bytes=f * (n * 4 * 1.25 + (n * n + 2 * n) * 12.0), flops=f * 40.0 * n ** 3)
    if kind == "rays":
        b, fl = _trace_work(case, case["count"] / 4, 0)
        return dict(bytes=b + case["count"] * (8 * n + 8), flops=fl)
    pixels = math.prod(_screen(case))
    if kind in ("denoise", "train"):
        feats, outs = (n + 10) * (2 * n - 1) + 1, 12 * (n - 1)
        params = 64 * (feats + 64 + outs)
        flops = pixels * (2.0 * params + (n - 1) * 9 * 60)
        values = 3 + 3 + n + 1 + 3
        return dict(bytes=4.0 * (pixels * values + (3 if kind == "train" else 1) * params),
                    flops=flops * (3 if kind == "train" else 1))
    rows = min(pixels, case["count"]) if kind == "pixels" else pixels
    b, fl = _trace_work(case, rows * _spp(n, case["spp"]), rows * (7 + n if kind == "inputs" else 3))
    return dict(bytes=b, flops=fl)


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "build":
        return "exact"
    if kind in ("denoise", "train"):
        # bf16 operands: measured 3e-4 to 1.2e-3 from exact(), over the dimensions and sample counts
        return {"rel": 4e-3}
    if kind == "rays":
        # t agrees to FP32 rounding; one ray in 10^5 meets a facet's edge, where hit and miss are both
        # within rounding: measured 2e-3 to 3e-3 from exact()
        return {"rel": 1e-2, "max": 0.99, "differ": 5e-5}
    # a path agrees with its 64-bit value to 1e-7 (measured) unless a rounding puts one of its rays on the
    # other side of an edge, about one ray in 10^6; such a path changes its pixel by 1 / spp of its value
    # (3e-4 of a small image, 2e-4 of the configurations')
    return {"rel": 1e-3, "max": 0.99}


# ------------------------------------------------------------------------------------------------
# the outputs in 64 bits


def exact(case: dict, seed: int):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "frame" and case["n"] == 3:
            spec = _spec(case, seed)
            paths = math.prod(spec["screen"]) * _spp(3, case["spp"])
            return _exact_frame(case, spec, seed) if paths * len(spec["facets"]) < 2e8 else None
        if kind == "rays":
            spec = _spec(case, seed)
            if case["count"] * len(spec["facets"]) < 6e10:
                mesh = _ExactMesh(spec["verts"], spec["facets"])
                org, d = _rays(case, spec, seed)
                d = torch.nn.functional.normalize(d.double(), dim=1)
                t, facet = mesh.closest(org.double(), d)
                return [torch.where(facet >= 0, t, torch.zeros_like(t)), facet.int()]
            return None
        if kind == "denoise":
            return _exact_denoise(case, _noisy_image(case, seed), _flat(case, seed))
    if kind == "train":
        return _exact_train(case, _noisy_image(case, seed), _flat(case, seed))
    # the other renders are Monte Carlo sums of millions of paths through large meshes, whose 64-bit
    # value takes minutes; a tree's whole numbers have no other value
    return None


class _ExactMesh:
    """Closest hits by testing every facet."""

    def __init__(self, verts: np.ndarray, facets: np.ndarray):
        v = torch.from_numpy(verts).cuda().double()[torch.from_numpy(facets).cuda().long()]
        n = v.shape[1]
        self.normal = torch.linalg.svd(v[:, 1:] - v[:, :1])[2][:, -1]
        self.d0 = (self.normal * v[:, 0]).sum(1)
        # barycentric coordinate i: plane[i] . p - offset[i]
        e = torch.cat([(v[:, :-1] - v[:, -1:]), self.normal[:, None]], 1)
        self.plane = torch.linalg.inv(e).transpose(1, 2)[:, : n - 1]
        self.offset = (self.plane * v[:, -1:]).sum(2)

    def closest(self, org: torch.Tensor, d: torch.Tensor, pairs: float = 1.5e8):
        step = max(1, int(pairs / len(self.d0)))
        parts = [self._closest(org[i:i + step], d[i:i + step]) for i in range(0, len(org), step)]
        return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])

    def _closest(self, org, d):
        t = (self.d0 - org @ self.normal.T) / (d @ self.normal.T)
        inside = t > 0
        last = torch.ones_like(t)
        for i in range(self.plane.shape[1]):
            b = org @ self.plane[:, i].T - self.offset[:, i] + t * (d @ self.plane[:, i].T)
            inside &= b > 0
            last -= b
        t = torch.where(inside & (last > 0), t, torch.full_like(t, torch.inf))
        best, facet = t.min(1)
        return best, torch.where(best < torch.inf, facet, torch.full_like(facet, -1))


def _philox(key: tuple[int, int], c: list[torch.Tensor]) -> list[torch.Tensor]:
    """Philox4x32-10 (Salmon, Moraes, Dror, Shaw 2011) on int64 tensors of 32-bit values."""
    low = 0xFFFFFFFF

    def mul(m: int, x: torch.Tensor):
        p0, p1 = x * (m & 0xFFFF), x * (m >> 16)
        s = p1 + (p0 >> 16)
        return s >> 16, ((s & 0xFFFF) << 16) | (p0 & 0xFFFF)

    k0, k1 = key
    for _ in range(10):
        hi0, lo0 = mul(0xD2511F53, c[0])
        hi1, lo1 = mul(0xCD9E8D57, c[2])
        c = [hi1 ^ c[1] ^ k0, lo1, hi0 ^ c[3] ^ k1, lo0]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    return c


def _uniform(seed: int, path: torch.Tensor, stream, draw: torch.Tensor) -> list[torch.Tensor]:
    zero = torch.zeros_like(path)
    words = _philox((seed & 0xFFFFFFFF, seed >> 32), [path & 0xFFFFFFFF, path >> 32, zero + stream, zero + draw])
    return [(w >> 8).double() / (1 << 24) for w in words]


def _exact_frame(case: dict, spec: dict, seed: int):
    """The same paths (same random numbers) in 64 bits, n = 3, facets tested one by one."""
    dev = "cuda"
    f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    mesh = _ExactMesh(spec["verts"], spec["facets"])
    screen, npix = spec["screen"], math.prod(spec["screen"])
    spp = _spp(3, case["spp"])
    k = round(spp ** 0.5)
    slab_lo = f64(spec["floor"][0])
    slab_hi = slab_lo + f64(np.diag(spec["floor"][1]))
    # the tracer starts secondary rays this far from the surface: 1000 FP32 epsilons of the largest coordinate
    offset = 4.0 * 1000 * 2.0 ** -23
    light, unit = f64(spec["light"]), float(np.linalg.norm(spec["light"].astype(np.float64)))
    bg, bg_light = f64(scenes.BACKGROUND), f64(scenes.BACKGROUND_LIGHT)
    norm = lambda a: a / a.norm(dim=1, keepdim=True)  # noqa: E731

    def floor_hit(o, d):
        a, b = (slab_lo - o) / d, (slab_hi - o) / d
        near, far = torch.minimum(a, b).amax(1), torch.maximum(a, b).amin(1)
        hit = (far > 0) & (near <= far)
        return torch.where(hit, torch.where(near > 0, near, far), torch.full_like(near, torch.inf))

    pixel = torch.arange(npix, device=dev).repeat_interleave(spp)
    sample = torch.arange(spp, device=dev).repeat(npix)
    path = sample * npix + pixel
    u = _uniform(seed, path, 0, torch.zeros_like(path))
    point = torch.stack([(pixel % screen[0]) + (sample % k + u[0]) / k, (pixel // screen[0]) + (sample // k + u[1]) / k], 1)
    d0 = norm(f64(spec["dir"])[None])
    axes = norm(f64(spec["axes"])) * float(np.float32(spec["param"]))
    org = f64(spec["org"]) + (point - f64(screen) / 2) @ axes
    d = d0.expand(len(path), 3).clone()
    beta = torch.ones((len(path), 3), dtype=torch.float64, device=dev)
    level_color = torch.ones(len(path), dtype=torch.float64, device=dev)
    out = torch.zeros((npix, 3), dtype=torch.float64, device=dev)
    for level in range(MAX_DEPTH + 1):
        tm, facet = mesh.closest(org, d)
        tf = floor_hit(org, d)
        miss = torch.isinf(torch.minimum(tm, tf))
        out.index_add_(0, pixel[miss], beta[miss] * (bg_light if level else bg))
        keep = ~miss
        org, d, beta, pixel, path, level_color, tm, tf, facet = (
            x[keep] for x in (org, d, beta, pixel, path, level_color, tm, tf, facet))
        on_mesh = tm < tf
        p = org + torch.minimum(tm, tf)[:, None] * d
        near = torch.stack([(p - slab_hi).abs(), (p - slab_lo).abs()], 2).reshape(len(p), -1).argmin(1)
        floor_normal = torch.nn.functional.one_hot(near // 2, 3).double() * torch.where(near % 2 == 0, 1.0, -1.0)[:, None]
        gn = torch.where(on_mesh[:, None], mesh.normal[facet.clamp(min=0)], floor_normal)
        gn = torch.where((d * gn).sum(1, keepdim=True) > 0, -gn, gn)
        albedo = torch.where(on_mesh, float(np.float32(spec["mesh_albedo"])), float(np.float32(spec["floor_albedo"])))
        level_color = level_color * albedo
        keep = level_color >= 1e-4
        beta = beta * albedo[:, None]
        to = light - p
        dist = to.norm(dim=1)
        ld = norm(to)
        power = unit ** 2 / dist ** 2
        dln = (ld * gn).sum(1)
        lit = keep & (power >= 1e-4) & (dln > 0)
        so = p + offset * ld
        blocked = torch.minimum(mesh.closest(so, ld)[0], floor_hit(so, ld)) < dist
        # the cosine-weighted lobe's constant at n = 3 is 2
        share = torch.where(lit & ~blocked, 2.0 * power * dln, torch.zeros_like(dln))
        out.index_add_(0, pixel, beta * share[:, None])
        if level == MAX_DEPTH:
            break
        v = torch.full((len(p), 2), 2.0, dtype=torch.float64, device=dev)
        for attempt in range(64):
            open_ = (v * v).sum(1) > 1
            if not open_.any():
                break
            w = _uniform(seed, path[open_], 1 + level, torch.full_like(path[open_], attempt))
            v[open_] = torch.stack([2 * w[0] - 1, 2 * w[1] - 1], 1)
        helper = torch.zeros_like(gn)
        first = gn[:, 0].abs() > 0.1
        helper[:, 1], helper[:, 0] = first.double(), (~first).double()
        b0 = norm(torch.cross(gn, helper, dim=1))
        b1 = torch.cross(gn, b0, dim=1)
        d = norm((1 - (v * v).sum(1)).clamp(min=0).sqrt()[:, None] * gn + v[:, :1] * b0 + v[:, 1:] * b1)
        keep &= ~(on_mesh & ((d * gn).sum(1) <= 0))
        org = p + offset * d
        org, d, beta, pixel, path, level_color = (x[keep] for x in (org, d, beta, pixel, path, level_color))
    return (out / spp).cpu().numpy()


def _flat(case: dict, seed: int) -> torch.Tensor:
    den = _denoiser(case, seed)
    p = torch.from_numpy(den.get_params()).double().cuda()
    den.close()
    return p


def _exact_denoise(case: dict, image: dict, flat: torch.Tensor) -> torch.Tensor:
    """The network of include/ntrace_denoise.h: features of the pixel and its axis neighbours, two hidden
    layers of 64, and per axis a 9-tap softmax filter whose logits carry the guide distances."""
    n, screen = case["n"], _screen(case)
    f = {k: v.double() for k, v in image.items()}
    pix = torch.arange(len(f["depth"]), device="cuda")

    def neighbour(axis: int, step: int) -> torch.Tensor:
        stride = math.prod(screen[:axis])
        x = pix // stride % screen[axis]
        return pix + ((x + step).clamp(0, screen[axis] - 1) - x) * stride

    sides = [(a, s) for a in range(n - 1) for s in (-1, 1)]
    spatial = (sum((f["mean"][neighbour(a, s)] - f["mean"]) ** 2 for a, s in sides) / (4 * (n - 1))).sqrt()
    std = f["var"].clamp(min=0).sqrt()
    base = torch.cat([f["mean"], std, f["normal"], f["depth"][:, None] * 0.1, spatial], 1)
    noise = torch.full((len(pix), 1), case["spp"] ** -0.5, dtype=torch.float64, device="cuda")
    x = torch.cat([base] + [base[neighbour(a, s)] for a, s in sides] + [noise], 1)
    at = 0
    for rows in (64, 64, 12 * (n - 1)):
        w = flat[at:at + rows * x.shape[1]].reshape(rows, -1)
        at += w.numel()
        x = x @ w.T + flat[at:at + rows]
        at += rows
        x = x.relu() if rows == 64 else x
    y = f["mean"]
    for a in range(n - 1):
        o = x[:, 9 * (n - 1) + 3 * a:9 * (n - 1) + 3 * a + 3].clamp(max=20.0).exp()
        taps, logits = [neighbour(a, j - 4) for j in range(9)], []
        for j, q in enumerate(taps):
            v = std ** 2 + std[q] ** 2
            mid = 0.5 * (f["mean"] + f["mean"][q])
            colour = ((((f["mean"] - f["mean"][q]) ** 2 - v).clamp(min=0)) / (1e-4 + 0.01 * mid ** 2 + v)).mean(1)
            logits.append(x[:, 9 * a + j] - 4.0 * o[:, 0] * ((f["normal"] - f["normal"][q]) ** 2).sum(1)
                          - o[:, 1] * (f["depth"] - f["depth"][q]) ** 2 - 0.05 * o[:, 2] * colour)
        weights = torch.stack(logits, 1).softmax(1)
        y = sum(weights[:, j:j + 1] * y[q] for j, q in enumerate(taps))
    return y


def _exact_train(case: dict, image: dict, flat: torch.Tensor):
    flat = flat.clone().requires_grad_()
    target = image["target"].double()
    loss = ((_exact_denoise(case, image, flat) - target) ** 2).sum() / ((image["mean"].double() - target) ** 2).sum()
    loss.backward()
    # the first Adam step: both moments are bias-corrected to the gradient and its square
    g = flat.grad
    return [float(loss), (flat - 1e-3 * g / (g.abs() + 1e-8)).detach()]
