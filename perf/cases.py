"""The work a user of syfrack_gb300 has it do, as cases that can be timed and compared.

Each kind of case goes through one public entry point, on host buffers as that entry
point takes them:

probe     Renderer.compile(graph).probe(points): batched distances, traps, iterations
primary   Renderer.primary: primary rays, hit distance, steps and normals
render    Renderer.render: a path-traced frame, both integrators
batch     Batch.run, sync and every job's film: many uneven jobs in one wavefront
serve     Server: a burst of previews, escape-time tiles and refinements
tile      escape2d: a 2D escape-time tile with every trap
deepzoom  deep_zoom: a perturbation frame with its reference orbit

Sizes are those of the repository's workloads, tests and benchmark, or lie between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from syfrack_gb300 import (AreaLight, Batch, Camera, Canvas, Finish, GpuContext, Material, PlanarFractal, RenderConfig,
                           Renderer, Scene, Server, deep_zoom, escape2d, workloads)
from syfrack_gb300.graph import Graph, Kind, Link, Node
from syfrack_gb300.scene import EnvironmentLight, SunLight

# a point of the Mandelbrot set's boundary: workloads.deep_zoom_center(2026, 50000)
ZOOM_CENTER = (0.27868532354762443, 0.5820921261345181)

FORMS = ("bulb", "box", "menger", "world")
FAMILIES = ("Julia", "Mandelbrot", "BurningShip", "Newton", "Nova", "Phoenix")


def listed():
    return [
        # the reference's audit of one graph: 100,000 points of the Mandelbox
        {"name": "probe_box_100k", "kind": "probe", "form": "box", "n": 100_000},
        # a small interactive frame: 256x256 primary rays of the Mandelbulb, 256 steps
        {"name": "primary_bulb_256", "kind": "primary", "form": "bulb", "w": 256, "h": 256, "rule": "absolute",
         "normal": "central"},
        # a full-screen primary frame of an odd size, the reference's own hit rule
        {"name": "primary_menger_1919x1079", "kind": "primary", "form": "menger", "w": 1919, "h": 1079,
         "rule": "cone", "normal": "tetrahedral"},
        # one view of an orbiting client: 480x270, 1 sample, 1 bounce
        {"name": "render_bulb_480x270", "kind": "render", "form": "bulb", "w": 480, "h": 270, "spp": 1, "bounces": 1,
         "integrator": "wavefront", "rule": "cone"},
        # a composed world (copies, bounded forms, finishes, sky) with RenderConfig's
        # defaults: the per-pixel integrator, 256-pixel tiles
        {"name": "render_world_640x360", "kind": "render", "form": "world", "w": 640, "h": 360, "spp": 4,
         "bounces": 2, "integrator": "megakernel", "rule": "cone"},
        # the benchmark's frame: Mandelbox, 1280x720, 64 samples, 4 bounces, epsilon 1e-4
        {"name": "render_box_1280x720x64", "kind": "render", "form": "box", "w": 1280, "h": 720, "spp": 64,
         "bounces": 4, "integrator": "wavefront", "rule": "epsilon"},
        # uneven jobs of three forms, 64 to 512 pixels a side, 1 to 16 samples
        {"name": "batch_mixed_16", "kind": "batch", "jobs": 16, "mix": 7},
        # a burst of clients: previews, tiles and refinements queued at once
        {"name": "serve_burst_20", "kind": "serve", "previews": 8, "tiles": 8, "refines": 4, "mix": 5, "side": 640,
         "iters": 4000},
        # a small tile of the root-finding families
        {"name": "tile_newton_513x385", "kind": "tile", "family": "Newton", "w": 513, "h": 385, "iters": 256,
         "power": 3, "zoom": 2.0, "stripes": 12.0, "twist": 0.0},
        # the serving mix's largest tile: Burning Ship, 20,000 iterations
        {"name": "tile_ship_2048", "kind": "tile", "family": "BurningShip", "w": 2048, "h": 2048, "iters": 20000,
         "power": 2, "zoom": 2.0, "stripes": 12.0, "twist": 0.0},
        # a preview frame of a deep view
        {"name": "deepzoom_480x270", "kind": "deepzoom", "w": 480, "h": 270, "iters": 20000, "width": 1e-12},
        # the deep-zoom frame of the benchmark
        {"name": "deepzoom_3840x2160", "kind": "deepzoom", "w": 3840, "h": 2160, "iters": 50000, "width": 1e-12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("probe", "primary", "render", "batch", "serve", "tile", "deepzoom"))
    if kind == "probe":
        return {"kind": kind, "form": rng.choice(FORMS), "n": _log(rng, 1000, 150_000)}
    if kind == "primary":
        return {"kind": kind, "form": rng.choice(FORMS), "w": _log(rng, 96, 2048), "h": _log(rng, 96, 2048),
                "rule": rng.choice(("absolute", "cone")), "normal": rng.choice(("central", "tetrahedral"))}
    if kind == "render":
        form = rng.choice(FORMS)
        w = _log(rng, 96, 1280)
        h = max(54, int(w * rng.uniform(0.5, 0.8)))
        # generic graphs and the per-pixel integrator cost more a sample
        most = 400_000 if form == "world" else 16_000_000
        spp = max(1, min(_log(rng, 1, 32), most // (w * h)))
        return {"kind": kind, "form": form, "w": w, "h": h, "spp": spp, "bounces": rng.randint(1, 4),
                "integrator": "megakernel" if w * h * spp < 2_000_000 and rng.random() < 0.4 else "wavefront",
                "rule": rng.choice(("cone", "epsilon"))}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 16), "mix": rng.randint(1, 1000)}
    if kind == "serve":
        previews = rng.randint(1, 10)
        return {"kind": kind, "previews": previews, "tiles": rng.randint(0, 10), "refines": rng.randint(0, 6),
                "mix": rng.randint(1, 1000), "side": _log(rng, 256, 1024), "iters": _log(rng, 1000, 8000)}
    if kind == "tile":
        family = rng.choice(FAMILIES)
        root = family in ("Newton", "Nova")
        plain = rng.random() < 0.5
        return {"kind": kind, "family": family, "w": _log(rng, 64, 2048), "h": _log(rng, 64, 2048),
                "iters": _log(rng, 64, 512 if root else 20000) if plain else _log(rng, 64, 512),
                "power": rng.randint(3, 5) if root else 2 if plain else rng.randint(2, 5),
                "zoom": round(rng.uniform(1.0, 4.0), 3), "stripes": 12.0 if plain else rng.choice((0.0, 5.0, 7.5, 12.0)),
                "twist": 0.0 if plain else rng.choice((0.0, 10.0))}
    w = _log(rng, 160, 2560)
    return {"kind": kind, "w": w, "h": max(90, w * 9 // 16 + rng.randint(0, 5)), "iters": _log(rng, 2000, 50000),
            "width": 10.0 ** rng.uniform(-12.5, -3.0)}


# ------------------------------------------------------------------ what a program keeps
_kept = {}


def _renderer() -> Renderer:
    if "renderer" not in _kept:
        _kept["renderer"] = Renderer(GpuContext(0))
    return _kept["renderer"]


def _server() -> Server:
    if "server" not in _kept:
        _kept["server"] = Server(_renderer(), hbm_budget=16 << 30)
    return _kept["server"]


# ------------------------------------------------------------------ scenes
def _world() -> Graph:
    """A ground plane, a bounded Mandelbulb, copies of a torus and a rounded box melted
    into a sphere, each with its finish."""
    nodes, links = [Node(0, Kind("Input"))], []

    def add(kind, *inputs):
        nodes.append(Node(len(nodes), kind))
        links.extend(Link((src, 0), (len(nodes) - 1, port)) for port, src in enumerate(inputs))
        return len(nodes) - 1

    ground = add(Kind("Plane", normal=[0.0, 1.0, 0.0], offset=-1.2), 0)
    at = add(Kind("Translate", offset=[-1.3, 0.0, 0.0]), 0)
    body = [add(Kind("Trap", slot=0, measure="Norm", scale=4.0)), add(Kind("Power", power=8.0)),
            add(Kind("AddSeed", multiplier=[1.0, 1.0, 1.0]))]
    bulb = add(Kind("BulbFence"), add(Kind("Iterate", iterations=8, bailout=2.0, body=body), at))
    bulb = add(Kind("MaterialTag", index=1),
               add(Kind("Bounded", half=[1.25, 1.25, 1.25], margin=0.05), at, bulb))
    torus = add(Kind("MaterialTag", index=2), add(Kind("Torus", radius=0.35, tube=0.1), 0))
    copies = add(Kind("Instances", placements=[
        ((1.6 * math.cos(a) + 0.2, -0.9, 1.6 * math.sin(a)), (15.0 * k - 90.0, 30.0 * k - 180.0, 0.0), (1.0, 1.0, 1.0))
        for k, a in enumerate(2 * math.pi * i / 12 for i in range(12))], half=[0.5, 0.5, 0.5], margin=0.05), torus)
    turned = add(Kind("Rotate", angles=[15.0, 40.0, 0.0]), add(Kind("Translate", offset=[1.5, 0.1, 0.0]), 0))
    box = add(Kind("RoundBox", half=[0.6, 0.6, 0.6], radius=0.1), turned)
    ball = add(Kind("Sphere", radius=0.5), add(Kind("Translate", offset=[1.5, 0.9, 0.0]), 0))
    melt = add(Kind("SmoothUnion", k=0.25), box, ball)
    root = add(Kind("Union"), add(Kind("Union"), ground, bulb), add(Kind("Union"), copies, melt))
    add(Kind("Output"), root)
    return Graph(nodes, links, safety=0.8, bounding_radius_hint=6.0)


def _graph(form) -> Graph:
    if form == "bulb":
        return workloads.mandelbulb_primary_graph()
    if form == "box":
        return workloads.mandelbox_graph()
    if form == "menger":
        return Graph.bundled("menger")
    return _world()


def _camera(form, rng) -> Camera:
    """The form's view, turned by up to half a degree."""
    pos, fov = {"bulb": ((0.0, 0.0, -3.0), 60.0), "box": ((3.2, 2.6, -5.5), 45.0), "menger": ((2.2, 1.6, -2.8), 50.0),
                "world": ((0.6, 1.4, -5.0), 50.0)}[form]
    a = math.radians(rng.uniform(-0.5, 0.5))
    x, y, z = pos
    return Camera.look_at((x * math.cos(a) - z * math.sin(a), y, x * math.sin(a) + z * math.cos(a)), (0.0, 0.0, 0.0), fov)


def _scene(form, seed, rng) -> Scene:
    if form == "box":
        s = workloads.mandelbox_scene(seed=seed)
        s.camera = _camera(form, rng)
        return s
    lights = [AreaLight(position=(1.0, 3.5, -3.5), normal=(-1.0, -3.5, 3.5), size=(1.0, 1.0), intensity=10.0)]
    material = Material(albedo=(0.7, 0.7, 0.7), roughness=0.4)
    if form == "world":
        lights += [SunLight(), EnvironmentLight()]
        material.finishes = [Finish(albedo=(0.8, 0.5, 0.3), roughness=0.3),
                             Finish(albedo=(0.9, 0.8, 0.5), roughness=0.2, metallic=1.0)]
    return Scene(graph=_graph(form), camera=_camera(form, rng), material=material, lights=lights, seed=seed)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    r = _renderer()
    state = {"case": case, "renderer": r}
    if kind == "probe":
        extent = {"bulb": 1.4, "box": 2.4, "menger": 1.4, "world": 2.5}[case["form"]]
        state["graph"] = r.compile(_graph(case["form"]))
        state["points"] = rng.uniform(-extent, extent, (case["n"], 3)).astype(np.float32)
    elif kind == "primary":
        state["graph"] = _graph(case["form"])
        state["camera"] = _camera(case["form"], rng)
        r.compile(state["graph"])
    elif kind == "render":
        state["scene"] = _scene(case["form"], int(rng.integers(0, 2**31)), rng)
        r.compile(state["scene"].graph)
        state["cfg"] = RenderConfig(width=case["w"], height=case["h"], samples_per_pixel=case["spp"],
                                    max_bounces=case["bounces"], max_steps=512,
                                    hit_epsilon=workloads.PATHTRACE_EPSILON if case["rule"] == "epsilon" else 0.0)
        if case["integrator"] == "wavefront":  # the whole frame in one dispatch
            state["cfg"].integrator = "wavefront"
            state["cfg"].tile_size = max(case["w"], case["h"])
            state["cfg"].samples_per_dispatch = case["spp"]
    elif kind == "batch":
        jobs = workloads.mixed_batch(seed=case["mix"], jobs=case["jobs"])
        for scene, _ in jobs:
            scene.seed = int(rng.integers(0, 2**31))
        state["batch"] = Batch(r, jobs)
    elif kind == "serve":
        state["server"] = _server()
        fixed = np.random.default_rng(case["mix"])
        graphs = workloads.serving_graphs()
        state["previews"] = []
        for _ in range(case["previews"]):
            scene, cfg = workloads._preview_scene(fixed, graphs)
            scene.seed = int(rng.integers(0, 2**31))
            r.compile(scene.graph)
            state["previews"].append((scene, cfg))
        state["refines"] = [int(fixed.integers(0, case["previews"])) for _ in range(case["refines"])]
        state["tiles"] = []
        for _ in range(case["tiles"]):
            side = (max(64, case["side"] // 2), case["side"])
            fractal, canvas = workloads._tile(fixed, side, (max(64, case["iters"] // 4), case["iters"]))
            canvas.center = _nudged(canvas, rng)
            state["tiles"].append((fractal, canvas))
    elif kind == "tile":
        state["fractal"], canvas = _tile(case)
        canvas.center = _nudged(canvas, rng)
        state["canvas"] = canvas
    elif kind == "deepzoom":
        # the same view, moved by a fraction of itself below the centre's last bit
        state["lo"] = tuple((rng.uniform(-0.01, 0.01, 2) * case["width"]).tolist())
    return state


def _tile(case):
    f = PlanarFractal(family=case["family"], power=case["power"], iterations=case["iters"], stripes=case["stripes"],
                      twist=case["twist"])
    center = {"BurningShip": (-0.45, -0.5), "Mandelbrot": (-0.6, 0.0)}.get(case["family"], (0.0, 0.0))
    return f, Canvas(width=case["w"], height=case["h"], center=center, zoom=case["zoom"])


def _nudged(canvas, rng):
    """The canvas's centre moved by less than a pixel."""
    pitch = 6.0 / canvas.zoom / canvas.width
    return tuple(float(c + rng.uniform(-0.5, 0.5) * pitch) for c in canvas.center)


def run(state):
    case = state["case"]
    kind = case["kind"]
    r = state["renderer"]
    if kind == "probe":
        return state["graph"].probe(state["points"])
    if kind == "primary":
        return r.primary(state["graph"], state["camera"], case["w"], case["h"], rule=case["rule"],
                         normal=case["normal"])
    if kind == "render":
        out = r.render(state["scene"], state["cfg"])
        return {"color": out.color, "accum": out.accum, "depth": out.depth, "normals": out.normals}
    if kind == "batch":
        b = state["batch"]
        b.run(1)
        b.sync()
        films = [b.readback(j) for j in range(case["jobs"])]
        return {"accum": [f.accum for f in films], "depth": [f.depth for f in films],
                "normals": [f.normals for f in films]}
    if kind == "serve":
        s = state["server"]
        views = [s.preview(scene, cfg) for scene, cfg in state["previews"]]
        tiles = [s.tile(fractal, canvas) for fractal, canvas in state["tiles"]]
        refines = [s.refine(views[k], workloads.SERVE_REFINE_SPP) for k in state["refines"]]
        out = {"films": [s.wait(t).accum for t in views + refines], "iterations": [], "smooth": [], "traps": []}
        for t in tiles:
            res = s.wait(t)
            out["iterations"].append(res.iterations)
            out["smooth"].append(res.smooth)
            out["traps"].append(res.traps)
        for t in views + tiles + refines:
            s.release(t)
        return out
    if kind == "tile":
        out = escape2d(r.ctx, state["fractal"], state["canvas"])
    else:
        out = deep_zoom(r.ctx, ZOOM_CENTER, state["lo"], case["width"], case["w"], case["h"], case["iters"])
    # the counts as int32, a view of the same bytes: torch has few operations on uint32
    out["iterations"] = out["iterations"].view(np.int32)
    return out


# ------------------------------------------------------------------ work
# (evaluations a ray or segment, iterations an evaluation, flops an iteration, flops an
# evaluation besides) of each form: the algorithm's counts, FMA = 2
_DE = {"bulb": (25, 5, 75, 60), "box": (31, 14, 31, 29), "menger": (18, 5, 30, 40), "world": (30, 6, 60, 150)}


def _de_flops(form):
    _, its, per_it, per_eval = _DE[form]
    return its * per_it + per_eval


def _tile_flops(family, n, iters, power):
    root = family in ("Newton", "Nova")
    mean = min(iters, 16) if root else 0.15 * iters + 20
    return n * mean * (6 * (power - 1) + (30 if root else 5) + 20)


def work(case):
    kind = case["kind"]
    if kind == "probe":
        return {"bytes": case["n"] * (12 + 28), "flops": case["n"] * _de_flops(case["form"])}
    if kind == "primary":
        n = case["w"] * case["h"]
        return {"bytes": n * 20, "flops": n * (_DE[case["form"]][0] + 6) * _de_flops(case["form"])}
    if kind == "render":
        n = case["w"] * case["h"]
        segments = n * case["spp"] * (1 + 0.5 * case["bounces"])
        return {"bytes": n * 52, "flops": segments * _DE[case["form"]][0] * _de_flops(case["form"])}
    if kind == "batch":
        jobs = workloads.mixed_batch(seed=case["mix"], jobs=case["jobs"])
        pixels = sum(c.width * c.height for _, c in jobs)
        paths = sum(c.width * c.height * c.samples_per_pixel for _, c in jobs)
        return {"bytes": pixels * 52, "flops": 2 * paths * 25 * 400}
    if kind == "serve":
        p = workloads.SERVE_PREVIEW
        n = p["width"] * p["height"]
        paths = n * (case["previews"] + workloads.SERVE_REFINE_SPP * case["refines"])
        pixels = case["tiles"] * (0.75 * case["side"]) ** 2
        return {"bytes": 16 * n * (case["previews"] + case["refines"]) + 24 * pixels,
                "flops": 1.5 * paths * 25 * 400 + _tile_flops("Julia", pixels, 0.6 * case["iters"], 2)}
    n = case["w"] * case["h"]
    if kind == "tile":
        return {"bytes": 24 * n, "flops": _tile_flops(case["family"], n, case["iters"], case["power"])}
    return {"bytes": 8 * n, "flops": n * 0.4 * case["iters"] * 20}


# ------------------------------------------------------------------ exact: 64 bits
def _f64(x, dev):
    return torch.as_tensor(np.asarray(x, np.float64), device=dev)


def _de64(form, p):
    """(distance, trap 0) of a bundled form at points p (n, 3), in binary64."""
    inf = torch.full_like(p[:, 0], math.inf)
    c, z, dr, trap, live = p, p, torch.ones_like(inf), inf.clone(), torch.ones_like(inf, dtype=torch.bool)
    bail, its, scale = {"bulb": (2.0, 12, 4.0), "box": (1000.0, 15, 2.0), "menger": (1.0e6, 5, 4.0)}[form]
    for _ in range(its):
        r = z.norm(dim=1)
        live = live & (r <= bail)
        if form == "bulb":
            seen = r
            theta, phi = 8.0 * torch.atan2(torch.hypot(z[:, 0], z[:, 1]), z[:, 2]), 8.0 * torch.atan2(z[:, 1], z[:, 0])
            st = theta.sin()
            n = torch.stack([st * phi.cos(), st * phi.sin(), theta.cos()], 1) * (r**8)[:, None] + c
            d = 8.0 * r**7 * dr + 1.0
        elif form == "box":
            q = z.clamp(-1.0, 1.0) * 2.0 - z
            r2 = (q * q).sum(1)
            seen = r2.sqrt()
            k = torch.where(r2 < 0.25, torch.full_like(r2, 4.0), torch.where(r2 < 1.0, 1.0 / r2, torch.ones_like(r2)))
            n = q * (k * -1.5)[:, None] + c
            d = dr * (k * 1.5) + 1.0
        else:
            q = z.abs().sort(dim=1, descending=True).values * 3.0 - 2.0
            n = torch.stack([q[:, 0], q[:, 1], torch.where(q[:, 2] < -1.0, q[:, 2] + 2.0, q[:, 2])], 1)
            seen = n.norm(dim=1)
            d = dr * 3.0
        z = torch.where(live[:, None], n, z)
        dr = torch.where(live, d, dr)
        trap = torch.where(live, torch.minimum(trap, seen), trap)
    if form == "bulb":
        r = z.norm(dim=1).clamp_min(1e-12)
        dist = 0.5 * r.log() * r / dr
    elif form == "box":
        dist = z.norm(dim=1) / dr.abs()
    else:
        q = z.abs() - 1.0
        dist = (q.clamp_min(0.0).norm(dim=1) + q.max(dim=1).values.clamp_max(0.0)) / dr
    return dist, (trap / scale).clamp_max(1.0)


def _primary64(case, camera, dev):
    """Hit distance of each primary ray (-1 on a miss), in binary64."""
    w, h, form = case["w"], case["h"], case["form"]
    b = camera.basis()
    fw, rt, up, org = (_f64(v, dev) for v in (b.forward, b.right, b.up, b.origin))
    aspect = float(np.float32(w) / np.float32(h))
    y, x = torch.meshgrid(_f64(np.arange(h), dev), _f64(np.arange(w), dev), indexing="ij")
    nx, ny = ((x + 0.5) / w * 2 - 1).reshape(-1, 1), ((y + 0.5) / h * 2 - 1).reshape(-1, 1)
    rd = fw + rt * (nx * b.tan_half_fov) - up * (ny * b.tan_half_fov / aspect)
    rd = rd / rd.norm(dim=1, keepdim=True)
    absolute = case["rule"] == "absolute"
    accept = 1e-4 if absolute else b.tan_half_fov * 2.0 / w
    safety = {"bulb": 0.7, "box": 0.6, "menger": 0.9}[form]
    far, steps = 10.0, 256
    out = torch.full((w * h,), -1.0, dtype=torch.float64, device=dev)
    at = torch.arange(w * h, device=dev)
    t = torch.zeros(w * h, dtype=torch.float64, device=dev)
    om, pr, sl, ct = t + 1.2, t.clone(), t.clone(), t.clone()
    ce = t + 1e30
    for _ in range(steps):
        radius = _de64(form, org + rd[at] * t[:, None])[0].abs() * safety
        failed = (om > 1.0) & (radius + pr < sl * 1.0001)
        sl = torch.where(failed, sl - om * sl, radius * om)
        om = torch.where(failed, torch.ones_like(om), om)
        pr = radius
        err = radius if absolute else radius / t.clamp_min(1e-6)
        better = ~failed & (err < ce)
        ct, ce = torch.where(better, t, ct), torch.where(better, err, ce)
        hit = ~failed & ((err <= accept) if absolute else (err < accept))
        out[at[hit]] = t[hit]
        last = ~failed & (t + sl >= far)
        gone = last & (radius >= far - t)
        om = torch.where(last, torch.ones_like(om), om)
        sl = torch.where(last, radius, sl)
        t = t + sl
        live = ~hit & ~gone & (t < far)
        at, t, om, pr, sl, ct, ce = (v[live] for v in (at, t, om, pr, sl, ct, ce))
        if not len(at):
            return out
    taken = ce < accept * 4.0
    out[at[taken]] = ct[taken]
    return out


def _cpow(x, y, n):
    a, b = x, y
    for _ in range(n - 1):
        a, b = a * x - b * y, a * y + b * x
    return a, b


def _root64(case, f, canvas, dev):
    """distance and traps of a Newton tile in binary64."""
    w, h, n = case["w"], case["h"], case["power"]
    y, x = torch.meshgrid(_f64(np.arange(h), dev), _f64(np.arange(w), dev), indexing="ij")
    scale = 6.0 / canvas.zoom
    zx = ((x + 0.5) / w - 0.5).reshape(-1) * scale + canvas.center[0]
    zy = (0.5 - (y + 0.5) / h).reshape(-1) / (w / h) * scale + canvas.center[1]
    one = torch.ones_like(zx)
    ring, stripe, count, measured, last = one * 1e20, one * 0, one * 0, one * 0, one.clone()
    smooth, live = one * f.iterations, torch.ones_like(zx, dtype=torch.bool)
    for _ in range(f.iterations):
        r = torch.hypot(zx, zy)
        live = live & (r <= f.bailout)
        ring = torch.where(live, torch.minimum(ring, (r - f.trap_radius).abs()), ring)
        stripe = torch.where(live, stripe + 0.5 + 0.5 * torch.sin(f.stripes * torch.atan2(zy, zx)), stripe)
        measured = torch.where(live, measured + 1, measured)
        ax, ay = _cpow(zx, zy, n)
        ax = ax - 1.0
        size = torch.hypot(ax, ay)
        done = live & (size < 1e-6)
        size = size.clamp_min(1e-20)
        part = (torch.log(1e-6 / last) / torch.log(size / last)).clamp(0.0, 1.0)
        smooth = torch.where(done, torch.where(count == 0, one * 0, count - 1 + part), smooth)
        live = live & ~done
        if not bool(live.any()):
            break
        last = torch.where(live, size, last)
        dx, dy = _cpow(zx, zy, n - 1)
        dx, dy = dx * n, dy * n
        den = (dx * dx + dy * dy).clamp_min(1e-24)
        sx, sy = (ax * dx + ay * dy) / den, (ay * dx - ax * dy) / den
        zx, zy = torch.where(live, zx - sx, zx), torch.where(live, zy - sy, zy)
        count = torch.where(live, count + 1, count)
    r = torch.hypot(zx, zy).clamp_max(1e20)
    smooth = torch.where(r > f.bailout, count, smooth)
    angle = torch.where(r == 0, one * 0.5, torch.atan2(zy, zx) / (2 * math.pi) + 0.5)
    traps = torch.stack([(smooth / f.iterations).clamp(0, 1), ring / (1 + ring), stripe / measured.clamp_min(1), angle])
    return (r / (1 + r)).reshape(h, w), traps.reshape(4, h, w)


def exact(case, seed):
    """None for path-traced films, whose samples branch on every rounding, and for the
    chaotic orbits of escape time and deep zoom."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    rng = np.random.default_rng([seed, 77])
    if kind == "probe" and case["form"] != "world":
        extent = {"bulb": 1.4, "box": 2.4, "menger": 1.4}[case["form"]]
        p = _f64(rng.uniform(-extent, extent, (case["n"], 3)).astype(np.float32), dev)
        d, t0 = _de64(case["form"], p)
        one = torch.ones_like(t0)
        return {"distance": d, "iterations": None, "material": None, "traps": torch.stack([t0, one, one, one], 1)}
    if kind == "primary" and case["form"] != "world":
        return {"normal": None, "steps": None, "t": _primary64(case, _camera(case["form"], rng), dev)}
    if kind == "tile" and case["family"] == "Newton" and case["twist"] == 0.0:
        f, canvas = _tile(case)
        canvas.center = _nudged(canvas, rng)
        d, traps = _root64(case, f, canvas, dev)
        return {"distance": d, "iterations": None, "traps": traps}
    return None
