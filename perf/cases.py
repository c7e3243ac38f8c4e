"""Performance cases: the work a host application has this library do.

Every case runs through the Python mirror of the C ABI (`PathTracer`, the
differentiable `Renderer` / `render`), as an application's frame loop, a
headless render, an inverse-rendering loop or a picking query does.

Kinds of a case (`kind`):
  frame    one `encode`: `spp` more samples of every pixel, folded into the
           running mean. The output is the accumulation where it lives, on the
           device. With `show`, the frame is also metered (automatic exposure)
           and resolved to 8-bit sRGB in host memory, as a viewer does.
  grad     one optimisation step's render and gradient: `render` of `spp`
           fresh samples, mean squared difference from a target image, and the
           gradients of the scene's material parameters.
  hits     closest hits of `rays` rays held by the host.
  shadows  star visibility of `rays` rays held by the host.

Scenes (`scene`), seeded:
  spheres  a star, a planet under the observer and a moon
  rings    a ringed giant with a tabulated optical-depth profile, a binary
           star, a moon under the observer
  system   the rings scene dressed as the application shows it: a banded gas
           giant, a cratered moon, the star catalogue and the Milky Way
  terrain  a heightfield of `cells` cells a side with rocks, boxes and bushes
  air      the terrain scene under an earthlike atmosphere

Sizes follow the repository's workloads (256 x 256, 512 x 512, 640 x 360,
1920 x 1080; 64 samples per dispatch; 2048 cells is the reference's largest
grid, 512 its default) and its tests' odd and small images.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from stargaze_b200 import PathTracer, abi, sky
from stargaze_b200 import workloads as W
from stargaze_b200.autograd import Renderer, render
from stargaze_b200.pathtracer import rays_array

# Operations per sample that the algorithm needs (every add, multiply,
# divide, square root and comparison one operation): the events the
# library's counting kernel reports for these scenes at six bounces, priced
# from the shader's source as bench.py prices them. A gradient replays each
# sample once more and differentiates what it meets.
OPS_PER_SAMPLE = {"spheres": 390.0, "rings": 715.0, "system": 1100.0, "terrain": 4700.0, "air": 8800.0}

# Rough nanoseconds per sample on one B200: keeps a drawn case no dearer than
# the largest listed one. Not used for anything else.
COST_NS = {"spheres": 0.09, "rings": 0.11, "system": 0.8, "terrain": 1.5, "air": 5.0}
MOST_NS = 1.2e8


def listed() -> list[dict]:
    return [
        # The application's view while it is being moved: one sample per frame
        # of a small window; launches and host work are all that is felt.
        dict(name="frame_spheres_256", kind="frame", scene="spheres", width=256, height=256, spp=1, bounces=6),
        # A viewer's frame with everything it shows: one sample, metering,
        # the resolve to sRGB and its read-back.
        dict(name="viewer_system_720p", kind="frame", scene="system", width=1280, height=720, spp=1, bounces=6,
             show=True),
        # One sample per frame over the default terrain grid, odd-sized window.
        dict(name="frame_terrain_odd", kind="frame", scene="terrain", width=959, height=541, spp=1, bounces=8,
             cells=512, props=250),
        # A thumbnail rendered headless in one dispatch.
        dict(name="still_spheres_256", kind="frame", scene="spheres", width=256, height=256, spp=64, bounces=6),
        # A mid-sized progressive render, odd sizes, a few samples per frame.
        dict(name="still_rings_odd", kind="frame", scene="rings", width=1001, height=563, spp=7, bounces=8),
        # The headline workload's dispatch: 1080p, 64 samples.
        dict(name="still_rings_1080p", kind="frame", scene="rings", width=1920, height=1080, spp=64, bounces=6),
        # The largest landscape render: 1080p over the reference's largest grid.
        dict(name="still_terrain_1080p", kind="frame", scene="terrain", width=1920, height=1080, spp=32, bounces=6,
             cells=2048, props=700),
        # A landscape under air: the camera march dominates.
        dict(name="still_air_360p", kind="frame", scene="air", width=640, height=360, spp=16, bounces=6, cells=1024,
             props=250),
        # One step of the ring inverse problem at its stated size.
        dict(name="grad_rings_512", kind="grad", scene="rings", width=512, height=512, spp=64, bounces=6),
        # One step of an albedo-map fit.
        dict(name="grad_terrain_540p", kind="grad", scene="terrain", width=960, height=540, spp=16, bounces=6,
             cells=1024, props=250, texels=1024),
        # Offline queries against the celestial scene.
        dict(name="hits_rings_million", kind="hits", scene="rings", rays=1_000_003),
        # A light curve's worth of eclipse and ring-transmission queries.
        dict(name="shadows_rings_64k", kind="shadows", scene="rings", rays=65_521),
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choices(["frame", "grad", "hits", "shadows"], [7, 2, 1, 1])[0]
    if kind in ("hits", "shadows"):
        return dict(kind=kind, scene=rng.choice(["spheres", "rings"]), rays=round(_log_uniform(rng, 256, 1_000_000)))
    scene = rng.choice(["rings", "terrain"] if kind == "grad" else ["spheres", "rings", "system", "terrain", "air"])
    width = round(_log_uniform(rng, 64, 1920))
    height = max(36, min(1080, round(width / rng.choice([16 / 9, 4 / 3, 1.0, 2.35]))))
    spp = round(_log_uniform(rng, 1, 64))
    per_sample = COST_NS[scene] * (6.0 if kind == "grad" else 1.0)
    spp = max(1, min(spp, int(MOST_NS / (width * height * per_sample))))
    case = dict(kind=kind, scene=scene, width=width, height=height, spp=spp, bounces=rng.randint(2, 8))
    if scene in ("terrain", "air"):
        case |= dict(cells=rng.choice([256, 512, 1024, 2048]), props=rng.randint(60, 700))
        if kind == "grad":
            case |= dict(texels=rng.choice([256, 512, 1024]))
    if kind == "frame" and rng.random() < 0.3:
        case |= dict(show=True)
    return case


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _sky_tables():
    """The application's own sky: the same catalogue and panorama in every run."""
    stars, cells = sky.ray_catalogue(sky.generate(3500, 2500, 0x5EED1234))
    return stars, cells, sky.panorama()


def _style(body, code: float, secondary, detail: float, params) -> None:
    """A procedural surface (build_frame's packing of a configured body)."""
    body.axis_x[3] = code
    body.axis_y[3] = 17.0
    body.surface_color[:] = [*secondary, detail]
    body.surface_params[:] = [float(p) for p in params]


def _workload(case: dict, seed: int):
    """The case's packed scene; the seed sets its materials, its ring profile,
    its ground and its objects."""
    rng = np.random.default_rng(seed)
    scene, width, height = case["scene"], case.get("width", 1920), case.get("height", 1080)
    if scene == "spheres":
        wl = W.spheres_256(width, height)
    elif scene in ("rings", "system"):
        wl = W.rings_1080p(width, height)
        wl.ring_tables = {0: W.ring_tau_profile(512, seed=seed)}
    else:
        rocks = case["props"] * 2 // 7
        wl, _ = W.terrain_1080p(width, height, cells=case["cells"], rocks=rocks, foliage=case["props"] - rocks,
                                seed=seed % 65536)
    for b in wl.frame.bodies:
        if b.emissive < 0.5:
            b.color[:] = [float(c) * rng.uniform(0.8, 1.2) for c in b.color]
    if scene == "system":
        W.with_mottle(wl.frame)
        planet, moon = wl.frame.bodies[2], wl.frame.bodies[3]
        _style(planet, 1.0, [0.3, 0.27, 0.22], 0.5, [7.0, 1.0, 0.0, 0.0])
        _style(moon, 2.0, [0.06, 0.06, 0.06], 0.8, [0.0, 0.65, 0.4, 0.0])
    if scene == "air":
        W.with_air(wl.frame, 1)
    wl.max_bounces = case.get("bounces", 6)
    return wl


class _Accumulation:
    """The library's accumulation, as a tensor sees it (not copied). The tensor
    holds this object, and with it the tracer that owns the memory."""

    def __init__(self, tracer: PathTracer):
        self.tracer = tracer
        width, height = tracer.size()
        self.__cuda_array_interface__ = dict(shape=(height, width, 4), typestr="<f4", version=3,
                                             data=(tracer.accumulation_device_ptr(), False))


def _frame_state(case: dict, seed: int) -> dict:
    wl = _workload(case, seed)
    options = W.render_options(wl, case["spp"], noise_seed=seed * 2654435761)
    if case.get("show"):
        options.auto_exposure = 1
    if case["scene"] == "system":
        options.milky_way = 4.0e-4
    tracer = PathTracer((wl.width, wl.height), options)
    W.upload_workload(tracer, wl)
    if case["scene"] == "system":
        stars, cells, panorama = _sky_tables()
        tracer.upload_catalogue(stars, cells)
        tracer.upload_milky_way(panorama)
    return dict(tracer=tracer, frame=wl.frame, image=torch.as_tensor(_Accumulation(tracer), device="cuda"))


def _grad_state(case: dict, seed: int) -> dict:
    wl = _workload(case, seed)
    width, height = case["width"], case["height"]
    generator = torch.Generator(device="cuda").manual_seed(seed)
    land = wl.landscape
    if case["scene"] == "terrain":
        start = 0.05 + 0.55 * torch.rand((case["texels"], case["texels"]), generator=generator, device="cuda")
        renderer = Renderer(wl.frame, width, height, case["spp"], wl.max_bounces, terrain=(land.terrain, land.cells),
                            albedo_map=start.cpu().numpy(), map_extent_m=2000.0, noise_seed=seed)
        params = dict(albedo_map=start)
    else:
        renderer = Renderer(wl.frame, width, height, case["spp"], wl.max_bounces, ring_tables=wl.ring_tables,
                            noise_seed=seed)
        params = dict(ring_tau=torch.as_tensor(wl.ring_tables[0], device="cuda"),
                      ring_albedo=torch.tensor([list(b.ring_color[:3]) for b in wl.frame.bodies], device="cuda"),
                      body_color=torch.tensor([list(b.color[:3]) for b in wl.frame.bodies], device="cuda"))
    # A target a little off the start's image: the residual's sign and size
    # vary over the image as they do while fitting.
    with torch.no_grad():
        target = render(renderer, **params) * (0.8 + 0.4 * torch.rand((height, width, 1), generator=generator,
                                                                       device="cuda"))
    return dict(renderer=renderer, target=target, params={k: v.requires_grad_() for k, v in params.items()})


def _bodies64(frame):
    """Centres (64-bit sums of the packed high and low parts) and radii."""
    centre = np.array([[float(b.center[k]) + float(b.center_low[k]) for k in range(3)] for b in frame.bodies])
    return centre, np.array([float(b.radius) for b in frame.bodies])


def _rays(wl, n: int, seed: int, at_stars: bool):
    """Rays as queries make them: half through the view, half from points on
    the bodies; all of them toward points of a star's disc and just beyond it
    when `at_stars` (returned with their lights)."""
    rng = np.random.default_rng(seed + 1)
    frame = wl.frame
    centre, radius = _bodies64(frame)
    tangent, aspect = frame.globals.cam_forward[3], frame.globals.viewport[0] / frame.globals.viewport[1]
    unit = lambda v: v / np.linalg.norm(v, axis=1, keepdims=True)  # noqa: E731
    m = n // 2
    xy = rng.uniform(-1.0, 1.0, (m, 2))
    camera = unit(np.stack([xy[:, 0] * tangent * aspect, xy[:, 1] * tangent, -np.ones(m)], axis=1))
    solid = np.array([i for i, b in enumerate(frame.bodies) if b.emissive < 0.5])
    lit = np.array([i for i, b in enumerate(frame.bodies) if b.emissive >= 0.5])
    on = solid[rng.integers(0, len(solid), n - m)]
    normal = unit(rng.normal(size=(n - m, 3)))
    leaving = unit(normal + 0.95 * unit(rng.normal(size=(n - m, 3))))
    anchor = np.concatenate([np.full(m, abi.MISS, np.uint32), on.astype(np.uint32)])
    offset = np.concatenate([np.zeros((m, 3)), normal * (radius[on] * (1.0 + 2.0e-6))[:, None]]).astype(np.float32)
    direction = np.concatenate([camera, leaving])
    lights = lit[rng.integers(0, len(lit), n)].astype(np.uint32)
    if at_stars:
        base = np.where((anchor == abi.MISS)[:, None], 0.0, centre[np.minimum(anchor, len(centre) - 1)])
        jitter = unit(rng.normal(size=(n, 3))) * (radius[lights] * rng.uniform(0.0, 1.2, n))[:, None]
        direction = unit(centre[lights] + jitter - base - offset)
    return rays_array(offset, direction.astype(np.float32), anchor), lights


def _query_state(case: dict, seed: int) -> dict:
    wl = _workload(case, seed)
    tracer = PathTracer((64, 64), W.render_options(wl))
    W.upload_workload(tracer, wl)
    rays, lights = _rays(wl, case["rays"], seed, case["kind"] == "shadows")
    return dict(tracer=tracer, frame=wl.frame, rays=rays, lights=lights)


def prepare(case: dict, seed: int) -> dict:
    make = dict(frame=_frame_state, grad=_grad_state, hits=_query_state, shadows=_query_state)[case["kind"]]
    return dict(kind=case["kind"], show=case.get("show", False), **make(case, seed))


def run(state: dict):
    if state["kind"] == "frame":
        tracer = state["tracer"]
        tracer.encode(state["frame"], torch.cuda.current_stream())
        out = dict(image=state["image"])
        if state["show"]:
            out["shown"] = tracer.display(stream=torch.cuda.current_stream())
        return out
    if state["kind"] == "grad":
        params = state["params"]
        image = render(state["renderer"], **params)
        loss = ((image - state["target"]) ** 2).mean()
        grads = torch.autograd.grad(loss, list(params.values()))
        return dict(image=image.detach(), loss=loss.detach(), grads=dict(zip(params, grads)))
    if state["kind"] == "hits":
        hits = state["tracer"].closest_hit(state["frame"], state["rays"])
        return dict(index=hits["index"], distance=hits["distance"], normal=hits["normal"])
    return dict(visibility=state["tracer"].light_visibility(state["frame"], state["rays"], state["lights"]))


def work(case: dict) -> dict:
    if case["kind"] in ("hits", "shadows"):
        bodies = 3 if case["scene"] == "spheres" else 4
        # A ray in (28 B) and a hit out (20 B), or a light index in and a
        # transmission out (4 B each); 40 operations per sphere, 70 per ring.
        return dict(bytes=case["rays"] * (48 if case["kind"] == "hits" else 36),
                    flops=case["rays"] * (40.0 * bodies + 70.0 * (case["scene"] == "rings")))
    pixels = case["width"] * case["height"]
    samples = pixels * case["spp"]
    # The running sum, its compensation and the mean: 16 B each, the first two
    # also read.
    n_bytes = pixels * 80.0
    ops = OPS_PER_SAMPLE[case["scene"]]
    if case.get("show"):
        n_bytes += pixels * 36.0  # accumulation and backdrop read, sRGB written
    if case["kind"] == "grad":
        n_bytes += pixels * 48.0 + 8.0 * case.get("texels", 23) ** 2  # image, target, d loss; parameters and gradients
        ops *= 2.0
    return dict(bytes=n_bytes, flops=samples * ops)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def exact(case: dict, seed: int):
    """The queries in 64 bits: sphere distances and normals, eclipses and ring
    transmissions of the packed scene. A rendered image is a Monte-Carlo
    estimate whose random decisions are defined in 32 bits: the same walk in 64
    bits takes another turn wherever a decision lies within rounding of its
    threshold, so images and their gradients have no such value."""
    if case["kind"] not in ("hits", "shadows"):
        return None
    wl = _workload(case, seed)
    rays, lights = _rays(wl, case["rays"], seed, case["kind"] == "shadows")
    centre, radius = _bodies64(wl.frame)
    n = len(rays)
    offset, d = rays["offset"].astype(np.float64), rays["direction"].astype(np.float64)
    away = rays["anchor"] != abi.MISS
    base = np.where(away[:, None], centre[np.minimum(rays["anchor"], len(centre) - 1)], 0.0)
    a = np.einsum("ij,ij->i", d, d)

    def sphere(i):
        """Distance of the nearest root ahead and the point there, relative to the centre."""
        oc = (centre[i] - base) - offset
        b = np.einsum("ij,ij->i", oc, d)
        cross = np.cross(oc, d)
        h = a * radius[i] ** 2 - np.einsum("ij,ij->i", cross, cross)
        root = np.sqrt(np.maximum(h, 0.0))
        q = b + np.where(b >= 0.0, root, -root)
        gap = np.linalg.norm(oc, axis=1)
        c = (gap - radius[i]) * (gap + radius[i])
        with np.errstate(divide="ignore", invalid="ignore"):
            t0, t1 = np.where(b < 0.0, q / a, c / q), np.where(b < 0.0, c / q, q / a)
        far = ~(t0 > 0.0)
        t = np.where(far, t1, t0)
        hit = (h >= 0.0) & (q != 0.0) & (t > 0.0)
        perpendicular = np.cross(d, cross) / a[:, None]
        return np.where(hit, t, 1.0e30), -perpendicular + d * (np.where(far, root, -root) / a)[:, None], oc

    if case["kind"] == "hits":
        best, normal = np.full(n, 1.0e30), np.zeros((n, 3))
        for i in range(len(radius)):
            t, point, _ = sphere(i)
            nearer = t < best
            best = np.where(nearer, t, best)
            unit = point / np.maximum(np.linalg.norm(point, axis=1, keepdims=True), 1e-300)
            normal = np.where(nearer[:, None], unit, normal)
        return dict(index=None, distance=best, normal=normal)

    to_light, seen = np.full(n, 1.0e30), np.ones(n)
    distance = [sphere(i) for i in range(len(radius))]
    for i in range(len(radius)):
        to_light = np.where(lights == i, distance[i][0], to_light)
    seen[to_light >= 1.0e30] = 0.0
    for i in range(len(radius)):
        t = distance[i][0]
        seen[(lights != i) & (t < 1.0e30) & ((t < to_light) | ((t == to_light) & (i < lights)))] = 0.0
    for i, body in enumerate(wl.frame.bodies):
        inner, outer, depth = float(body.ring_plane[3]), float(body.ring_params[0]), float(body.ring_params[1])
        if outer <= inner or depth <= 0.0:
            continue
        pole, oc = np.array([float(v) for v in body.ring_plane[:3]]), distance[i][2]
        slope = d @ pole
        with np.errstate(divide="ignore", invalid="ignore"):
            t = (oc @ pole) / slope
            point = d * t[:, None] - oc
        r = np.linalg.norm(point, axis=1) / radius[i]
        through = (np.abs(slope) >= 1.0e-7) & (t > 0.0) & (r >= inner) & (r <= outer) & (t < to_light)
        table = wl.ring_tables[int(body.ring_params[3]) - 1].astype(np.float64)
        x = np.where(through, (r - inner) / (outer - inner), 0.0)
        tau = depth * table[np.clip((x * len(table)).astype(np.int64), 0, len(table) - 1)]
        seen = np.where(through, seen * np.exp(-tau / np.maximum(np.abs(slope), 1.0e-7)), seen)
    return dict(visibility=seen)
