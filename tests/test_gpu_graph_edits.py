"""Value edits of a graph (sf_graph_update) while another thread renders with it: a frame
shows the values of before or of after an edit, nothing in between."""
import contextlib
import ctypes as C
import threading

import numpy as np
import pytest

from syfrack_gb300 import Camera, RenderSession, Server, workloads
from syfrack_gb300.graph import Kind
from syfrack_gb300.scene import AreaLight, Material, RenderConfig, Scene
from test_union_bound import _Builder

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def edited(cg, graphs):
    """Edits the compiled graph to each of `graphs` in turn, over and over, in a thread."""
    stop, bad = threading.Event(), []
    descs = [g.to_desc() for g in graphs]

    def loop():
        while not stop.is_set():
            for desc, _keep in descs:
                st = cg.ctx.lib.sf_graph_update(cg.h, C.byref(desc))
                if st:
                    bad.append(st)

    t = threading.Thread(target=loop)
    t.start()
    try:
        yield
    finally:
        stop.set()
        t.join()
    assert not bad


def prepared_scene():
    """A scene whose program holds each op with constants prepared on the device."""
    b = _Builder()
    turned = b.add(Kind("Rotate", angles=[20.0, 35.0, 50.0]), [0])
    halves = b.add(Kind("Mirror", normal=[0.3, 1.0, 0.2], offset=0.1), [turned])
    fan = b.add(Kind("Kaleido", planes=5, phase=10.0), [halves])
    fold = b.add(Kind("SphereFold", min_radius=0.4, fixed_radius=0.9), [fan])
    box = b.add(Kind("RoundBox", half=[0.7, 0.3, 0.4], radius=0.1), [fold])
    ground = b.add(Kind("Plane", normal=[0.1, 1.0, 0.0], offset=-1.0), [0])
    g = b.graph(b.add(Kind("Union"), [ground, box]))
    light = AreaLight(position=(1.0, 3.5, -3.5), normal=(-1.0, -3.5, 3.5), size=(1.0, 1.0), intensity=10.0)
    return Scene(graph=g, camera=Camera.look_at((1.0, 1.2, -3.5), (0.0, 0.0, 0.0), 45.0),
                 material=Material(albedo=(0.7, 0.7, 0.7), roughness=0.4), lights=[light], seed=3)


def test_served_frames_during_edits_to_the_same_values(renderer):
    scene = prepared_scene()
    cg = renderer.compile(scene.graph)
    assert cg.info()["form"] == "generic"
    cfg = RenderConfig(width=120, height=80, samples_per_pixel=1, max_bounces=2, max_steps=128, tile_size=120,
                       samples_per_dispatch=1, integrator="wavefront")
    srv = Server(renderer, hbm_budget=1 << 30, slots=2)

    def frame():
        t = srv.preview(scene, cfg)
        out = srv.wait(t).accum
        srv.release(t)
        return out

    want = frame()
    assert want[..., :3].mean() > 1e-3
    with edited(cg, [scene.graph]):
        for _ in range(150):
            np.testing.assert_array_equal(frame(), want)
    srv.close()


@pytest.mark.parametrize("integrator", ["wavefront", "megakernel"])
def test_dispatches_during_value_edits(renderer, integrator):
    """A session's frames while another thread switches its Mandelbox between two sets of
    values (fold limit, scale and trap scale): each is one set's frame, bit for bit."""
    scene = workloads.mandelbox_scene()
    scene.graph = workloads.mandelbox_graph(scale=-1.6)  # a handle of its own
    other = workloads.mandelbox_graph(scale=-2.0)
    for n in other.nodes:
        if n.kind.name == "BoxFold":
            n.kind.fields["limit"] = 0.8
        elif n.kind.name == "Trap":
            n.kind.fields["scale"] = 0.5
    cg = renderer.compile(scene.graph)
    cfg = RenderConfig(width=64, height=48, samples_per_pixel=1, max_bounces=3, max_steps=128, tile_size=64,
                       samples_per_dispatch=1, integrator=integrator)
    s = RenderSession(renderer, scene, cfg)
    kept = {}

    def frame():
        s.dispatch((0, 0, 64, 48, 0), 1)
        assert s.sync() == 0
        return s.readback().accum

    # one sample more is added to the film by every dispatch of sample 0: differences are frames
    def edit(g):
        desc, kept[0] = g.to_desc()
        assert cg.ctx.lib.sf_graph_update(cg.h, C.byref(desc)) == 0

    last = np.zeros((48, 64, 4), np.float32)
    want = []
    for g in (scene.graph, other):
        edit(scene.graph)  # every session takes the march's constants from the first set
        fresh = RenderSession(renderer, scene, cfg)
        edit(g)
        fresh.dispatch((0, 0, 64, 48, 0), 1)
        assert fresh.sync() == 0
        want.append(fresh.readback().accum)
        fresh.close()
    assert not np.array_equal(want[0], want[1])
    seen = set()
    with edited(cg, [scene.graph, other]):
        for _ in range(200):
            now = frame()
            match = [k for k in (0, 1) if np.array_equal(now, last + want[k])]
            assert match
            seen.add(match[0])
            last = now
    edit(scene.graph)
    s.close()
    assert seen == {0, 1}
