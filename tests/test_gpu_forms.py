"""Kernels compiled per form: primary rays of every form at odd sizes against the f32
oracle, with the normals as planes and as rows; batches whose jobs are traced group by
group (forms and their variants, and more of those than groups) against each job alone."""
import ctypes as C

import numpy as np
import pytest

from helpers import bounded_bulb, golden_scene
from syfrack_gb300 import Batch, RenderSession
from syfrack_gb300.graph import Graph
from syfrack_gb300.scene import AreaLight, Camera, Material, RenderConfig, Scene

pytestmark = pytest.mark.gpu


def graph_of(form, trap="Minimum", **params):
    g = bounded_bulb() if form == "any" else Graph.bundled(form, **params)
    if form != "any":
        for n in g.nodes:
            if n.kind.name == "Trap":
                n.kind.fields["mode"] = trap
    return g


def camera_of(form):
    return Camera.look_at({"mandelbox": (3.2, 2.6, -5.5), "menger": (1.6, 1.3, -2.6)}.get(form, (1.0, 0.8, -3.0)),
                          (0.0, 0.0, 0.0), 45.0)


@pytest.mark.parametrize("trap", ["Minimum", "Maximum"])
@pytest.mark.parametrize("form", ["mandelbulb", "mandelbox", "menger", "any"])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 3), (61, 37)])
def test_primary_forms(renderer, oracle_mod, form, trap, w, h):
    g, cam = graph_of(form, trap, **({"scale": -1.5} if form == "mandelbox" else {})), camera_of(form)
    gpu = renderer.primary(g, cam, w, h, max_steps=256, rule="cone", eps=1e-4, t_far=20.0, normal="central")
    desc = Scene(graph=None, camera=cam).desc(w, h).camera
    ref = oracle_mod.OracleGraph(g).primary(desc, w, h, 256, 0, 1e-4, 20.0, 1.0, 0, precision=32)
    hit, rhit = gpu["t"] >= 0, ref["t"] >= 0
    assert (hit != rhit).sum() <= 0.01 * w * h
    both = hit & rhit
    if both.any():
        near = np.abs(gpu["t"][both] - ref["t"][both]) <= 1e-3 * ref["t"][both]
        assert near.mean() >= 0.98
    assert (np.abs(gpu["steps"].astype(np.int64) - ref["steps"].astype(np.int64)) <= 2).mean() >= 0.98
    np.testing.assert_allclose(np.linalg.norm(gpu["normal"][hit], axis=1), 1.0, atol=1e-5)
    assert np.all(gpu["normal"][~hit] == 0)


def test_normals_as_planes_and_as_rows(renderer):
    """sf_primary_trace's (3, pixels) planes hold what sf_primary_trace_rows' rows do."""
    from syfrack_gb300 import _lib as abi
    from syfrack_gb300._lib import check

    w, h = 61, 37
    g, cam = graph_of("menger"), camera_of("menger")
    rows = renderer.primary(g, cam, w, h, max_steps=256, rule="cone", eps=1e-4, t_far=20.0)
    d = abi.sf_primary_desc()
    d.camera = Scene(graph=None, camera=cam).desc(w, h).camera
    d.width, d.height, d.max_steps, d.rule, d.normal_mode = w, h, 256, 0, 0
    d.eps, d.t_far, d.pixel_tolerance = 1e-4, 20.0, 1.0
    t, steps, planes = np.empty(w * h, np.float32), np.empty(w * h, np.uint32), np.empty((3, w * h), np.float32)
    fp = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))
    check(renderer.ctx.lib.sf_primary_trace(renderer.compile(g).h, C.byref(d), fp(t),
                                            steps.ctypes.data_as(C.POINTER(C.c_uint32)), fp(planes)))
    np.testing.assert_array_equal(t, rows["t"])
    np.testing.assert_array_equal(steps, rows["steps"])
    np.testing.assert_array_equal(planes.T, rows["normal"])


VARIANTS = [("mandelbulb", "Minimum", {}), ("mandelbox", "Minimum", {"scale": -1.5}), ("any", "", {}),
            ("menger", "Minimum", {"iterations": 4}), ("mandelbox", "Maximum", {"scale": 2.0}),
            ("mandelbulb", "Maximum", {"power": 5.0}), ("mandelbox", "Minimum", {"scale": 2.0}),
            ("menger", "Maximum", {"iterations": 3}),
            ("mandelbox", "Minimum", {"min_radius": 1.2, "fixed_radius": 1.0}),
            ("mandelbox", "Maximum", {"min_radius": 1.2, "fixed_radius": 1.0})]


@pytest.mark.parametrize("picks", [[0], [2, 2], [1, 6], [0, 1, 2, 3, 4], list(range(10)), [9, 2, 0, 5, 3, 0, 8]])
def test_batch_groups(renderer, picks):
    """One form, the generic one alone, both signs of the Mandelbox scale, a mixture, ten
    jobs of nine variants (more than there are groups) and an unsorted order."""
    light = AreaLight(position=(1.0, 3.5, -3.5), normal=(-1.0, -3.5, 3.5), size=(1.0, 1.0), intensity=10.0)
    jobs = []
    for i, k in enumerate(picks):
        form, trap, params = VARIANTS[k]
        sc = Scene(graph=graph_of(form, trap, **params), camera=camera_of(form),
                   material=Material(albedo=(0.7, 0.7, 0.7), roughness=0.2, metallic=0.0, specular=0.04),
                   lights=[light], seed=5 + i)
        jobs.append((sc, RenderConfig(21 + 7 * i, 17 + i, 2, max_bounces=3, max_steps=256, pixel_tolerance=1.0,
                                      tile_size=128, samples_per_dispatch=2, integrator="wavefront")))
    b = Batch(renderer, jobs)
    b.run(1, use_graph=False)
    assert b.sync() == 0
    for i, (sc, cfg) in enumerate(jobs):
        got = b.readback(i)
        s = RenderSession(renderer, sc, cfg)
        while not s.step(0):
            pass
        ref = s.readback()
        s.close()
        np.testing.assert_array_equal(got.depth, ref.depth, err_msg=str(VARIANTS[picks[i]]))
        np.testing.assert_array_equal(got.accum, ref.accum, err_msg=str(VARIANTS[picks[i]]))
    b.close()


# Batches of several groups: more variants than groups; scenes with one and with three
# shadow slots (area lights, then a sun and a sky) over four forms.
def launch_shape_jobs(kind):
    light = AreaLight(position=(1.0, 3.5, -3.5), normal=(-1.0, -3.5, 3.5), size=(1.0, 1.0), intensity=10.0)
    scenes = []
    for i, k in enumerate(range(10) if kind == "variants" else (1, 2, 7)):
        form, trap, params = VARIANTS[k]
        scenes.append(Scene(graph=graph_of(form, trap, **params), camera=camera_of(form),
                            material=Material(albedo=(0.7, 0.7, 0.7), roughness=0.2, metallic=0.0, specular=0.04),
                            lights=[light], seed=5 + i))
    if kind == "slots":
        scenes += [golden_scene("menger"), golden_scene("mandelbulb")]
    return [(sc, RenderConfig(21 + 7 * i, 17 + i, 2, max_bounces=3, max_steps=256, pixel_tolerance=1.0, tile_size=128,
                              samples_per_dispatch=2, integrator="wavefront")) for i, sc in enumerate(scenes)]


@pytest.fixture(scope="module", params=["variants", "slots"])
def jobs_alone(renderer, request):
    jobs, films = launch_shape_jobs(request.param), []
    for sc, cfg in jobs:
        s = RenderSession(renderer, sc, cfg)
        while not s.step(0):
            pass
        films.append(s.readback())
        s.close()
    return jobs, films


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("shape", [(3, 16, 4), (2, 8, 1), (4, 128, 32), (4, 0, 8)])
def test_batch_launch_shapes(renderer, jobs_alone, shape, use_graph):
    """Segments cut at a step quantum and resumed, group by group, launched one by one and
    replayed as a graph: every film is the job's alone, bit for bit."""
    jobs, films = jobs_alone
    b = Batch(renderer, jobs)
    b.set_launch(*shape)
    b.run(1, use_graph=use_graph)
    assert b.sync() == 0
    for i, ref in enumerate(films):
        got = b.readback(i)
        np.testing.assert_array_equal(got.depth, ref.depth, err_msg=str(i))
        np.testing.assert_array_equal(got.accum, ref.accum, err_msg=str(i))
    b.close()
