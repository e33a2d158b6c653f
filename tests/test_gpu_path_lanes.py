"""The per-pixel integrator's persistent path lanes against the wavefront, which runs the
same bounce body, march and order of sums: films are equal bit for bit at every tile shape
(fewer rows than a band, ragged bands, one pixel), sample count, form, step budget and
number of shadow segments a bounce (up to the eight a lane holds)."""
import numpy as np
import pytest

from syfrack_gb300 import RenderSession, workloads
from syfrack_gb300.graph import Graph
from syfrack_gb300.scene import AreaLight, Camera, EnvironmentLight, Material, RenderConfig, Scene, SunLight

pytestmark = pytest.mark.gpu
W, H = 70, 45
SHAPES = [(0, 0, 1, 1, 9), (3, 1, 1, 11, 3), (5, 20, 37, 3, 2), (40, 13, 13, 9, 5), (0, 12, 33, 8, 32), (0, 0, W, H, 3)]


def graph_of(form):
    if form == "any":
        from helpers import bounded_bulb

        return bounded_bulb()
    if form == "menger":
        return Graph.bundled("menger", iterations=4)
    return workloads.mandelbox_graph() if form == "box" else workloads.mandelbulb_primary_graph()


def films(renderer, scene, shapes, **cfg):
    out = []
    for integrator in ("wavefront", "megakernel"):
        c = RenderConfig(width=W, height=H, samples_per_pixel=64, tile_size=128, samples_per_dispatch=32,
                         integrator=integrator, **cfg)
        s = RenderSession(renderer, scene, c)
        for x, y, w, h, n in shapes:
            s.dispatch((x, y, w, h, 0), n)
        assert s.sync() == 0
        out.append(s.readback())
        s.close()
    a, b = out
    np.testing.assert_array_equal(a.accum, b.accum)
    np.testing.assert_array_equal(a.depth, b.depth)
    np.testing.assert_array_equal(a.normals, b.normals)
    return a


def scene_of(form, suns=0):
    far = {"box": (3.2, 2.6, -5.5), "menger": (1.6, 1.3, -2.6)}.get(form, (1.0, 0.8, -3.0))
    lights = [AreaLight(position=(1.0, 3.5, -3.5), normal=(-1.0, -3.5, 3.5), size=(1.0, 1.0), intensity=10.0)]
    lights += [SunLight(direction=(0.3 * k - 1.0, 0.8, -0.5), intensity=1.0 + k) for k in range(suns)]
    if suns:
        lights.append(EnvironmentLight())
    return Scene(graph=graph_of(form), camera=Camera.look_at(far, (0.0, 0.0, 0.0), 45.0),
                 material=Material(albedo=(0.7, 0.7, 0.7), roughness=0.2, metallic=0.0, specular=0.04),
                 lights=lights, seed=11)


@pytest.mark.parametrize("form", ["bulb", "box", "menger", "any"])
def test_tile_shapes(renderer, form):
    a = films(renderer, scene_of(form), SHAPES, max_bounces=3, max_steps=512, pixel_tolerance=1.0)
    assert (a.depth[:, :] >= 0).any() and a.accum[..., :3].mean() > 1e-3


@pytest.mark.parametrize("suns", [1, 6])  # 3 shadow segments a bounce; 8, the most a lane holds
@pytest.mark.parametrize("steps", [1, 24, 512])  # budgets that end on candidates, and exhausted paths
def test_shadow_segments_and_step_budgets(renderer, suns, steps):
    films(renderer, scene_of("bulb", suns), SHAPES[3:], max_bounces=4, max_steps=steps, pixel_tolerance=1.0)
    films(renderer, scene_of("any", suns), SHAPES[3:5], max_bounces=1, max_steps=steps, pixel_tolerance=1.0)
