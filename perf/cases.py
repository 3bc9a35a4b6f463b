"""Performance cases: the calls a program makes of this backend, over the range
of sizes it makes them at.

Four families, each through the package's public entry points:

* ``trace``  — DeviceAccelerator.intersect on device-resident rays (closest
  hit and any hit; camera, incoherent and shadow rays; flat and two-level
  scenes) and intersect_host on pinned host rays;
* ``build``  — build_bvh_device, the SAH hierarchy of a mesh scene;
* ``render`` — CudaBackend.render / render_many of whole images, from one
  preview sample to 64 samples per pixel;
* ``nrc``    — the radiance cache: inference and training steps.

A case is a dict of plain values; prepare() makes its inputs from a seed and
keeps what a program keeps between calls (the accelerator, the prepared
scene, the cache, a pinned film), run() is one call.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from yaoray_b200 import accel, batch, cornell, instanced, nrc, scenes
from yaoray_b200.render import CudaBackend, pinned_film

BOX = 100.0
T_MIN = scenes.RAY_T_MIN
SPHERE_TRIANGLES = 4096
FILM_FIELDS = ("sum", "samples", "luminance_mean", "luminance_m2", "albedo_sum", "normal_sum", "depth_sum",
               "aov_samples")


# --------------------------------------------------------------------- cases

def listed() -> list[dict]:
    return [
        # A picking or probing call of an interactive tool: a thousand rays
        # against a small mesh, where the launch path is the cost.
        dict(name="trace_small", family="trace", rays="incoherent", count=1000, spheres=3, any_hit=False,
             two_level=False, host=False, tuned=False),
        # The camera rays of one 1920 x 1080 frame of the 2M-triangle set.
        dict(name="trace_primary", family="trace", rays="coherent", width=1920, height=1080, spheres=512,
             any_hit=False, two_level=False, host=False, tuned=False),
        # The benchmark's traversal set: 2828^2 incoherent rays, 2M triangles,
        # the launch shape chosen by the accelerator's autotuner as there.
        dict(name="trace_incoherent", family="trace", rays="incoherent", count=2828 * 2828, spheres=512,
             any_hit=False, two_level=False, host=False, tuned=True),
        # Shadow rays of a renderer that shades elsewhere: any hit, a mid-size
        # scene and an odd ray count.
        dict(name="trace_shadow", family="trace", rays="shadow", count=1500001, spheres=100, any_hit=True,
             two_level=False, host=False, tuned=False),
        # The drop-in C path: rays and hits in (pinned) host memory.
        dict(name="trace_host", family="trace", rays="incoherent", count=2000000, spheres=512, any_hit=False,
             two_level=False, host=True, tuned=False),
        # Loading a scene: the SAH build of the 2M-triangle set.
        dict(name="build_flat", family="build", spheres=512, two_level=False),
        # One frame of an interactive preview: a view update and one sample
        # per pixel of a small image.
        dict(name="render_preview", family="render", scene="cornell", width=160, height=90, spp=1, max_depth=8,
             jobs=1, view=True, tuned=False),
        # The Cornell configuration: 256 x 256, 64 samples, depth 8, tuned as
        # the benchmark does.
        dict(name="render_cornell", family="render", scene="cornell", width=256, height=256, spp=64, max_depth=8,
             jobs=1, view=False, tuned=True),
        # The instanced configuration at its full image, depth and geometry,
        # one sample per pixel (31M instanced triangles, HDRI and emitters,
        # conductors, glass and coated surfaces).
        dict(name="render_instanced", family="render", scene="instanced", width=1920, height=1080, spp=1,
             max_depth=16, jobs=1, view=False, tuned=False),
        # Uneven batched jobs in shared launches: sphere scenes with the
        # instanced material mix plus subsurface, a small sky.
        dict(name="render_jobs", family="render", scene="jobs", width=128, height=128, spp=16, max_depth=8, jobs=4,
             view=False, tuned=False),
        # Cache queries of one 1920 x 1080 frame.
        dict(name="nrc_infer", family="nrc", train=False, count=1920 * 1080, steps=0),
        # Training: eight steps on a batch's 2^16 records, then the parameters
        # (a checkpoint) and a validation query.
        dict(name="nrc_train", family="nrc", train=True, count=65536, steps=8),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    family = rng.choice(("trace", "trace", "trace", "build", "render", "render", "render", "nrc", "nrc"))
    if family == "trace":
        rays = rng.choice(("coherent", "incoherent", "shadow"))
        c = dict(family=family, rays=rays, spheres=_log_int(rng, 1, 512), any_hit=rays == "shadow",
                 two_level=rng.random() < 0.3, host=rng.random() < 0.2, tuned=rng.random() < 0.3)
        if rays == "coherent":
            c["width"] = _log_int(rng, 40, 2800)
            c["height"] = max(1, int(c["width"] * rng.uniform(0.4, 1.0)))
        else:
            c["count"] = _log_int(rng, 1000, 2828 * 2828)
        return c
    if family == "build":
        return dict(family=family, spheres=_log_int(rng, 1, 512), two_level=rng.random() < 0.3)
    if family == "nrc":
        if rng.random() < 0.5:
            return dict(family=family, train=False, count=_log_int(rng, 1000, 1920 * 1080), steps=0)
        return dict(family=family, train=True, count=_log_int(rng, 1000, 65536), steps=rng.randint(1, 8))
    scene = rng.choice(("cornell", "textured", "cutout", "subsurface", "measured", "analytic", "instanced", "jobs",
                        "cached"))
    # Pixels x samples, capped so that a drawn render costs no more than the
    # listed ones of its kind.
    width = _log_int(rng, 64, 512 if scene in ("jobs", "cached") else 960)
    height = max(8, int(width * rng.uniform(0.5, 1.0)))
    limit = {"instanced": 1 << 20, "cached": 1 << 20, "jobs": 1 << 19}.get(scene, 1 << 21)
    spp = min(64, _log_int(rng, 1, max(2, limit // (width * height))))
    return dict(family=family, scene=scene, width=width, height=height, spp=spp,
                max_depth=16 if scene == "instanced" else rng.choice((5, 8)),
                jobs=rng.randint(2, 4) if scene == "jobs" else 1, view=scene == "cornell" and rng.random() < 0.5,
                tuned=scene != "jobs" and rng.random() < 0.3)


def _ray_count(case: dict) -> int:
    return case["width"] * case["height"] if case["rays"] == "coherent" else case["count"]


# ------------------------------------------------------------------- prepare

def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _directions(n: int, g: torch.Generator) -> torch.Tensor:
    """Unit vectors, uniform on the sphere."""
    z = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0
    phi = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2.0 * math.pi)
    s = (1.0 - z * z).clamp_min(0.0).sqrt()
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _rays(case: dict, seed: int) -> torch.Tensor:
    g = _generator(seed)
    n = _ray_count(case)
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 3] = T_MIN
    if case["rays"] == "coherent":
        # Pinhole camera outside the box, turned by the seed.
        w, h = case["width"], case["height"]
        a = torch.rand(2, generator=g, device="cuda").tolist()
        az, dist = 2.0 * math.pi * a[0], 140.0 + 20.0 * a[1]
        eye = np.array([BOX / 2 + dist * math.sin(az), 60.0, BOX / 2 + dist * math.cos(az)])
        o, f, r, u = scenes.camera_basis(eye, (BOX / 2, BOX / 2, BOX / 2))
        f, r, u = (torch.tensor(v, device="cuda") for v in (f, r, u))
        half = math.tan(math.radians(40.0) / 2)
        sx = (2.0 * (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w - 1.0) * (w / h) * half
        sy = (1.0 - 2.0 * (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h) * half
        d = f + r * sx[None, :, None] + u * sy[:, None, None]
        d = (d / d.norm(dim=2, keepdim=True)).reshape(-1, 3)
        rays[:, 0:3] = torch.tensor(o, device="cuda")
        rays[:, 4:7] = d
        rays[:, 7] = math.inf
        return rays
    origin = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * BOX
    rays[:, 0:3] = origin
    if case["rays"] == "incoherent":
        rays[:, 4:7] = _directions(n, g)
        rays[:, 7] = math.inf
    else:
        d = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * BOX - origin
        dist = d.norm(dim=1).clamp_min(1e-6)
        rays[:, 4:7] = d / dist[:, None]
        rays[:, 7] = dist
    return rays


def _geometry(case: dict, seed: int) -> accel.SceneGeometry:
    """`spheres` noisy sphere meshes of 4096 triangles in the box; two-level:
    a quarter as many meshes, each instanced four times by affine maps."""
    if not case["two_level"]:
        return scenes.traversal_scene(seed=seed, spheres=case["spheres"])
    base = scenes.traversal_scene(seed=seed, spheres=max(1, case["spheres"] // 4))
    rng = np.random.default_rng(seed)
    instances = []
    for k in range(max(1, case["spheres"])):
        q = rng.normal(size=4)
        w, x, y, z = q / np.linalg.norm(q)
        rot = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                        [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                        [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
        m = np.eye(4)
        m[:3, :3] = rot @ np.diag(rng.uniform(0.6, 1.4, 3))
        # turned about the box's centre, then moved a little
        centre = np.full(3, BOX / 2)
        m[:3, 3] = centre - m[:3, :3] @ centre + rng.uniform(-10.0, 10.0, 3)
        instances.append((k % base.primitives.size, m.T.reshape(16)))
    prims = base.primitives
    inst = np.zeros(len(instances), dtype=accel._lib.INSTANCE_DTYPE)
    for k, (prim, m) in enumerate(instances):
        inst[k]["primitive"] = prim
        inst[k]["object_to_world"] = m
    return accel.SceneGeometry(base.positions, base.indices, prims, instances=inst)


def _build_geometry(case: dict, seed: int) -> accel.SceneGeometry:
    """The set's meshes in an order of the seed's and (flat) scaled by a
    power of two: other vertices, another order and another layout, with the same node
    count (the SAH's sets do not depend on the order)."""
    g = _geometry(case, 1)
    rng = np.random.default_rng(seed)
    order = rng.permutation(g.primitives.size)
    prims = g.primitives[order].copy()
    idx = np.concatenate([g.indices[p["first_index"]:p["first_index"] + p["index_count"]] for p in prims])
    prims["first_index"] = np.concatenate([[0], np.cumsum(prims["index_count"])[:-1]])
    scale = np.float32(1.0 if case["two_level"] else 2.0 ** int(rng.integers(-3, 4)))
    inst = g.instances.copy()
    if inst.size:
        inst["primitive"] = np.argsort(order)[inst["primitive"]]
    return accel.SceneGeometry(g.positions * scale, idx, prims, instances=inst)


def _prepare_trace(case: dict, seed: int) -> dict:
    geom = _geometry(case, seed)
    if case["two_level"]:
        dev = accel.DeviceAccelerator(geom, accel.build_two_level_bvh(geom, device=True))
    else:
        dev = accel.DeviceAccelerator(geom, accel.build_bvh_device(geom)[0])
    rays = _rays(case, seed + 1)
    n = rays.shape[0]
    s = dict(dev=dev, any_hit=case["any_hit"], host=case["host"])
    if case["host"]:
        host = torch.empty((n, 8), dtype=torch.float32).pin_memory()
        host.copy_(rays)
        out = torch.empty(n if case["any_hit"] else (n, 4), dtype=torch.uint8 if case["any_hit"] else torch.float32)
        s["pinned"] = (host, out.pin_memory())
        s["rays"], s["out"] = s["pinned"][0].numpy(), s["pinned"][1].numpy()
        if case["tuned"]:
            dev.autotune_host(s["rays"][: 1 << 21], any_hit=case["any_hit"])
    else:
        s["rays"] = rays
        if case["tuned"]:
            dev.autotune(rays[: 1 << 21], any_hit=case["any_hit"])
    return s


def _scene(case: dict, seed: int):
    w, h, spp, depth = case["width"], case["height"], case["spp"], case["max_depth"]
    kind = case["scene"]
    if kind == "instanced":
        s = instanced.scene(w, h, spp, depth, seed=seed)
        s.radiance_clamp = 20.0
    elif kind == "cached":
        s = instanced.scene(w, h, spp, depth, instances=64, mesh_scale=0.1, env_width=512, seed=seed)
        s.radiance_clamp = 20.0
    else:
        make = {"cornell": cornell.scene, "textured": cornell.textured_scene, "cutout": cornell.cutout_scene,
                "subsurface": cornell.subsurface_scene, "measured": cornell.measured_scene,
                "analytic": cornell.analytic_scene}[kind]
        s = make(w, h, spp, depth)
    s.seed = int(seed)
    return s


def _job_scenes(case: dict, seed: int) -> list:
    """Uneven jobs: images of one, two and four times the case's width, scenes
    of a few to a few hundred spheres."""
    rng = np.random.default_rng(seed)
    out = []
    for j in range(case["jobs"]):
        scale = (1, 4, 2, 1)[j % 4]
        spheres = int(round(math.exp(rng.uniform(math.log(3), math.log(256)))))
        spp = max(1, case["spp"] * (4, 1, 1, 2)[j % 4])
        out.append(batch.job_scene(case["width"] * scale, spp, spheres, seed * 1000 + j, case["max_depth"]))
    return out


def _prepare_render(case: dict, seed: int) -> dict:
    backend = CudaBackend()
    if case["scene"] == "jobs":
        return dict(backend=backend, many=[backend.prepare(s) for s in _job_scenes(case, seed)])
    scene = _scene(case, seed)
    prepared = backend.prepare(scene)
    if case["tuned"]:
        prepared.autotune()
    s = dict(backend=backend, prepared=prepared, film=pinned_film(scene.width, scene.height), many=None,
             view=(scene.camera, scene.seed) if case["view"] else None)
    if case["scene"] == "cached":
        p = scene.geometry.positions
        cache = nrc.RadianceCache(p.min(0) - 100.0, float((p.max(0) - p.min(0)).max()) + 200.0, seed=1)
        prepared.set_radiance_cache(cache, spread_threshold=1e-3, train_steps=2, averaged=True)
        s["cache"] = cache
    return s


def _queries(n: int, g: torch.Generator) -> torch.Tensor:
    """Cache queries (position, roughness, direction, normal, albedos) on the
    surfaces of a scene: points of 64 spheres in the box."""
    q = torch.rand((n, 16), generator=g, device="cuda")
    centre = torch.rand((64, 3), generator=g, device="cuda") * 80.0 + 10.0
    radius = torch.rand(64, generator=g, device="cuda") * 8.0 + 1.0
    k = torch.randint(64, (n,), generator=g, device="cuda")
    normal = _directions(n, g).float()
    q[:, 0:3] = centre[k] + normal * radius[k][:, None]
    q[:, 4:7] = _directions(n, g).float()
    q[:, 7:10] = normal
    return q


def _targets(q: torch.Tensor) -> torch.Tensor:
    """A smooth radiance over position, direction and albedo."""
    t = torch.zeros((q.shape[0], 4), device="cuda")
    t[:, 0:3] = (0.3 + torch.sin(q[:, 0:3] * 0.15).abs() + 0.3 * (1.0 + (q[:, 4:7] * q[:, 7:10]).sum(1, keepdim=True)))
    t[:, 0:3] *= 0.2 + q[:, 10:13]
    return t


def _cache_params(seed: int) -> tuple[np.ndarray, np.ndarray]:
    """Network weights (Xavier-uniform) and grid features of the spread that a
    trained cache has, on the values the device stores: bf16 and fp16."""
    g = torch.Generator().manual_seed(seed)
    w = torch.zeros((6, 64, 64))
    for layer in range(6):
        rows = 64 if layer < 5 else 3
        a = math.sqrt(6.0 / (64 + rows))
        w[layer, :rows] = (torch.rand((rows, 64), generator=g) * 2 - 1) * a
    grid = (torch.rand((16, 1 << 19, 2), generator=g) * 2 - 1) * 0.5
    return w.bfloat16().float().numpy(), grid.half().float().numpy()


def _prepare_nrc(case: dict, seed: int) -> dict:
    cache = nrc.RadianceCache((0.0, 0.0, 0.0), BOX, seed=seed)
    g = _generator(seed)
    if not case["train"]:
        cache.set_params(*_cache_params(seed))
        return dict(cache=cache, queries=_queries(case["count"], g), steps=None)
    both = _queries(case["count"] * (case["steps"] + 1), g).reshape(case["steps"] + 1, case["count"], 16)
    steps = [(q.contiguous(), _targets(q)) for q in both[:-1]]
    return dict(cache=cache, queries=both[-1].contiguous(), steps=steps, loss=torch.zeros(1, device="cuda"))


def prepare(case: dict, seed: int) -> dict:
    family = case["family"]
    if family == "trace":
        return _prepare_trace(case, seed)
    if family == "build":
        return dict(geometry=_build_geometry(case, seed), two_level=case["two_level"])
    if family == "render":
        return _prepare_render(case, seed)
    return _prepare_nrc(case, seed)


# ----------------------------------------------------------------------- run

def _hits(h) -> dict:
    ids = h[:, 1].view(np.int32) if isinstance(h, np.ndarray) else h[:, 1].view(torch.int32)
    return dict(t=h[:, 0], id=ids, uv=h[:, 2:4])


def _bvh(b: accel.RenderBvh) -> dict:
    out = {f: b.nodes[f] for f in b.nodes.dtype.names}
    out.update({f: b.primitives[f] for f in b.primitives.dtype.names})
    return dict(out, order=b.primitive_indices, depth=b.max_depth)


def _film(result) -> dict:
    if not result.ok:
        raise RuntimeError(result.error)
    return dict({f: result.film[f] for f in FILM_FIELDS}, bad=result.bad_samples)


def run(s: dict):
    if "dev" in s:
        if s["host"]:
            out = s["dev"].intersect_host(s["rays"], any_hit=s["any_hit"], out=s["out"])
        else:
            out = s["dev"].intersect(s["rays"], any_hit=s["any_hit"])
        return out if s["any_hit"] else _hits(out)
    if "geometry" in s:
        if s["two_level"]:
            t = accel.build_two_level_bvh(s["geometry"], device=True)
            # One array of each kind over all BLASes (their node counts differ).
            return dict(tlas=_bvh(t.tlas), nodes=np.concatenate([b.nodes for _, _, b in t.blases]).view(np.int32),
                        order=np.concatenate([b.primitive_indices for _, _, b in t.blases]))
        return _bvh(accel.build_bvh_device(s["geometry"])[0])
    if "backend" in s:
        if s["many"] is not None:
            return [_film(r) for r in s["backend"].render_many(s["many"])]
        if s["view"] is not None:
            s["prepared"].set_view(*s["view"])
        return _film(s["backend"].render(s["prepared"], film_out=s["film"]))
    if s["steps"] is None:
        return s["cache"].infer(s["queries"])
    for q, t in s["steps"]:
        s["cache"].train_step(q, t, loss_out=s["loss"])
    # The network's weights; the grid shows in the validation query (its
    # rarely visited entries take steps of Adam's full size whatever the
    # gradient, whose last bits depend on the order of the sums).
    return dict(weights=s["cache"].get_params()[0], radiance=s["cache"].infer(s["queries"]), loss=s["loss"])


# ---------------------------------------------------------------------- work

def work(case: dict) -> dict:
    family = case["family"]
    if family == "trace":
        n = _ray_count(case)
        triangles = case["spheres"] * SPHERE_TRIANGLES / (4 if case["two_level"] else 1)
        # Rays in, hits out, the part of the tree (32-byte nodes, 36-byte
        # triangles) that so many rays can touch; 44 box and 2 triangle tests
        # of about 20 operations a ray.
        tree = min(triangles * (36 + 0.65 * 32), n * (44 * 32 + 2 * 36))
        return dict(bytes=n * (32 + (1 if case["any_hit"] else 16)) + tree, flops=n * 46 * 20.0)
    if family == "build":
        t = case["spheres"] * SPHERE_TRIANGLES / (4 if case["two_level"] else 1)
        # Vertices and indices in; nodes, order and primitives out; per
        # triangle and level two box unions and a bucket.
        return dict(bytes=t * (6 + 12 + 0.65 * 32 + 24), flops=t * max(1.0, math.log2(t / 3)) * 15.0)
    if family == "render":
        if case["scene"] == "jobs":
            pixels = sum((case["width"] * (1, 4, 2, 1)[j % 4]) ** 2 for j in range(case["jobs"]))
            samples = sum((case["width"] * (1, 4, 2, 1)[j % 4]) ** 2 * max(1, case["spp"] * (4, 1, 1, 2)[j % 4])
                          for j in range(case["jobs"]))
        else:
            pixels = case["width"] * case["height"]
            samples = pixels * case["spp"]
        # The film; per sample about four path vertices, each with a
        # closest-hit and a shadow ray (about 900 operations) and its shading.
        return dict(bytes=pixels * 56.0, flops=samples * 4 * (2 * 900 + 600.0))
    n, layers = case["count"], 5 * 2 * 64 * 64 + 2 * 64 * 3
    encode = 16 * 8 * 12.0
    table = 16 * (1 << 19) * 4
    if not case["train"]:
        return dict(bytes=n * (64 + 16) + min(table, n * 16 * 8 * 4) + 6 * 8192, flops=n * (layers + encode))
    touched = min(16 * (1 << 19), n * 16 * 8)
    # Forward and twice backward per step; of each touched entry its
    # features, moments and average in and out; the validation query and the
    # parameters read once.
    step = dict(bytes=n * (64 + 16) + touched * 2 * (4 + 4 * 8), flops=n * (3 * layers + 3 * encode))
    return dict(bytes=case["steps"] * step["bytes"] + table * 2 + n * 80,
                flops=case["steps"] * step["flops"] + n * (layers + encode))


# ----------------------------------------------------------------- tolerance

def tolerance(case: dict):
    family = case["family"]
    if family == "trace":
        # Bit-identical hits are this backend's contract; t, u and v of
        # another correct float32 intersection differ in the last bits.
        return "exact" if case["any_hit"] else dict(rel=1e-6, max=1e-5, differ=0.0)
    if family == "build":
        return "exact"
    if family == "render":
        # Seen when the shading kernels alone are compiled with fused
        # multiply-adds: 1e-4 (largest 0.04) on the Cornell boxes, 4e-3 (1.2)
        # on the job scenes, 0.06 (19) on one-sample instanced images, where a
        # last bit turns a path to another of the bright lights.
        if case["scene"] in ("instanced", "cached"):
            return dict(rel=0.03, max=0.99, differ=1e-4)
        if case["scene"] == "jobs":
            return dict(rel=0.015, max=0.99, differ=1e-4)
        return dict(rel=5e-4, max=0.15, differ=1e-4)
    if not case["train"]:
        # bf16 activations: 3.5e-4 off float64.
        return dict(rel=2e-3, max=0.05)
    # Two runs of the same steps differ by 1.2e-3 (largest 0.015): the order
    # of the gradients' sums through Adam.
    return dict(rel=1e-2, max=0.2)


# --------------------------------------------------------------------- exact

def _exact_closest(case: dict, seed: int):
    """Closest hits by testing every ray with every triangle in float64."""
    geom = _geometry(case, seed)
    rays = _rays(case, seed + 1).double()
    tri = torch.from_numpy(geom.positions[geom.indices.astype(np.int64)].reshape(-1, 3, 3)).cuda().double()
    p, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = rays.shape[0]
    out_t = torch.empty(n, dtype=torch.float64, device="cuda")
    out_uv = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    out_id = torch.empty(n, dtype=torch.int32, device="cuda")
    chunk = max(1, (1 << 25) // tri.shape[0])
    for a in range(0, n, chunk):
        o, d, far = rays[a:a + chunk, None, 0:3], rays[a:a + chunk, None, 4:7], rays[a:a + chunk, 7:8]
        h = torch.linalg.cross(d, e2[None])
        det = (e1 * h).sum(-1)
        inv = 1.0 / det
        s = o - p
        u = (s * h).sum(-1) * inv
        qv = torch.linalg.cross(s, e1[None].expand_as(s))
        v = (d * qv).sum(-1) * inv
        t = (e2 * qv).sum(-1) * inv
        miss = ~((u >= 0) & (v >= 0) & (u + v <= 1) & (t > T_MIN) & (t <= far) & (det != 0))
        t = torch.where(miss, math.inf, t)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        rows = torch.arange(best.shape[0], device="cuda")
        out_t[a:a + chunk] = torch.where(hit, best, far[:, 0])
        out_uv[a:a + chunk, 0] = torch.where(hit, u[rows, k], 0.0)
        out_uv[a:a + chunk, 1] = torch.where(hit, v[rows, k], 0.0)
        out_id[a:a + chunk] = torch.where(hit, k, -1).int()
    return dict(t=out_t, id=out_id, uv=out_uv)


def _exact_infer(case: dict, seed: int):
    """The cache's forward pass in float64: hash grid, spherical harmonics and
    surface attributes into the network."""
    weights, grid = (torch.from_numpy(v).cuda().double() for v in _cache_params(seed))
    queries = _queries(case["count"], _generator(seed)).double()
    growth = math.exp(math.log(2048.0 / 16.0) / 15)
    mask, chunk = (1 << 19) - 1, 1 << 17
    out = torch.zeros((queries.shape[0], 4), dtype=torch.float64, device="cuda")
    for a in range(0, queries.shape[0], chunk):
        q = queries[a:a + chunk]
        x = torch.zeros((q.shape[0], 64), dtype=torch.float64, device="cuda")
        pos = (q[:, 0:3] / BOX).clamp(0.0, 1.0)
        for level in range(16):
            scale = float(np.float32(16.0 * growth ** level))
            side = math.ceil(scale) + 2
            g = pos * scale
            cell = g.floor().long()
            f = g - cell
            for c in range(8):
                bit = torch.tensor([c & 1, (c >> 1) & 1, (c >> 2) & 1], device="cuda")
                at = cell + bit
                if side ** 3 <= 1 << 19:
                    idx = at[:, 0] + at[:, 1] * side + at[:, 2] * side * side
                else:
                    idx = (at[:, 0] ^ ((at[:, 1] * 2654435761) & 0xFFFFFFFF) ^ ((at[:, 2] * 805459861) & 0xFFFFFFFF)) & mask
                wgt = torch.where(bit == 1, f, 1.0 - f).prod(1)
                x[:, 2 * level:2 * level + 2] += grid[level][idx] * wgt[:, None]
        dx, dy, dz = q[:, 4], q[:, 5], q[:, 6]
        xx, yy, zz = dx * dx, dy * dy, dz * dz
        pi = math.pi
        k1, k2 = math.sqrt(3 / (4 * pi)), math.sqrt(15 / (4 * pi))
        k3, k4, k5 = math.sqrt(35 / (32 * pi)), math.sqrt(105 / (4 * pi)), math.sqrt(21 / (32 * pi))
        x[:, 32] = math.sqrt(1 / (4 * pi))
        x[:, 33], x[:, 34], x[:, 35] = -k1 * dy, k1 * dz, -k1 * dx
        x[:, 36], x[:, 37], x[:, 39], x[:, 40] = k2 * dx * dy, -k2 * dy * dz, -k2 * dx * dz, k2 / 2 * (xx - yy)
        x[:, 38] = math.sqrt(5 / (16 * pi)) * (3 * zz - 1)
        x[:, 41], x[:, 47] = k3 * dy * (-3 * xx + yy), k3 * dx * (-xx + 3 * yy)
        x[:, 42], x[:, 46] = k4 * dx * dy * dz, k4 / 2 * dz * (xx - yy)
        x[:, 43], x[:, 45] = k5 * dy * (1 - 5 * zz), k5 * dx * (1 - 5 * zz)
        x[:, 44] = math.sqrt(7 / (16 * pi)) * dz * (5 * zz - 3)
        x[:, 48:51] = q[:, 7:10] * 0.5 + 0.5
        x[:, 51] = q[:, 3]
        x[:, 52:58] = q[:, 10:16]
        x[:, 58] = 1.0
        for layer in range(5):
            x = (x @ weights[layer].T).clamp_min(0.0)
        out[a:a + chunk, 0:3] = (x @ weights[5].T)[:, 0:3].clamp_max(15.0).exp()
    return out


def exact(case: dict, seed: int):
    if case["family"] == "trace" and not (case["any_hit"] or case["two_level"]):
        if _ray_count(case) * case["spheres"] * SPHERE_TRIANGLES <= 1 << 30:
            return _exact_closest(case, seed)
    if case["family"] == "nrc" and not case["train"]:
        return _exact_infer(case, seed)
    return None
