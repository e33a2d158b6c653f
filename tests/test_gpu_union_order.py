"""Unions leave out a second operand whose lower bound their first operand already
beats: a Union is symmetric but for ties, so every order of its leaves (each with
other branches left out) must give the same sample bit for bit."""
import numpy as np
import pytest

from helpers import bounded_bulb, lcg_points
from syfrack_gb300 import Camera
from syfrack_gb300.graph import Graph, Kind
from test_gpu_de import kitchen_sink
from test_union_bound import _Builder, _bulb, _shape, union_world

pytestmark = pytest.mark.gpu

COPIES = [((0.0, -1.9, 0.3), (20.0, 0.0, 10.0), (1.0, 1.0, 1.0)), ((1.2, -1.8, 0.6), (-30.0, 45.0, 0.0), (0.7, 0.8, 0.9)),
          ((-1.1, -1.7, -0.4), (0.0, 90.0, 0.0), (1.0, 0.5, 1.0))]


def world(order, nested):
    b = _Builder()

    def leaf(k):
        if k == 0:
            return b.add(Kind("MaterialTag", index=4), [b.add(Kind("Plane", normal=[0.0, 1.0, 0.0], offset=-2.2), [0])])
        if k == 1:
            return _bulb(b, (0.8, -0.9, 0.0), 1)
        if k == 2:
            t = b.add(Kind("MaterialTag", index=2), [b.add(Kind("Torus", radius=0.5, tube=0.15), [0])])
            return b.add(Kind("Instances", placements=COPIES, half=[0.7, 0.7, 0.7], margin=0.05), [t])
        return _shape(b, Kind("RoundBox", half=[0.4, 0.3, 0.5], radius=0.1), (-1.6, -1.0, 0.2), tag=3, bounded=0.55)

    x, y, z, w = (leaf(k) for k in order)
    u = lambda p, q: b.add(Kind("Union"), [p, q])
    root = u(u(x, y), u(z, w)) if nested else u(u(u(x, y), z), w)
    return b.graph(root)


@pytest.mark.parametrize("nested", [False, True])
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 2, 1, 0), (2, 0, 3, 1)])
def test_every_order_gives_the_same_sample(renderer, order, nested):
    pts = np.concatenate([lcg_points(4096, 2.5, 7), lcg_points(4096, 0.9, 8) + np.array([0.2, -1.8, 0.1], np.float32)])
    base, other = world((1, 3, 0, 2), False), world(order, nested)
    a, c = renderer.compile(base).probe(pts), renderer.compile(other).probe(pts)
    for k in ("distance", "material", "iterations", "traps"):
        np.testing.assert_array_equal(a[k], c[k], err_msg=k)
    # the march's fast samples, flags and exact re-evaluations
    cam = Camera.look_at((0.5, -0.6, -4.5), (0.0, -1.4, 0.0), 50.0)
    p, q = (renderer.primary(g, cam, 120, 90, rule="cone") for g in (base, other))
    for k in ("t", "steps", "normal"):
        np.testing.assert_array_equal(p[k], q[k], err_msg=k)


def copies_of_a_bulb(depth):
    """Copies of a bounded loop, `depth` Instances deep, beside a loop of no iterations."""
    b = _Builder()
    d = _bulb(b, (0.0, 0.0, 0.0), 1)
    for _ in range(depth):
        d = b.add(Kind("Instances", placements=COPIES, half=[2.5, 2.5, 2.5], margin=0.05), [d])
    still = b.add(Kind("Iterate", iterations=1, bailout=0.01, body=[b.add(Kind("Abs", x=True, y=True, z=True))]), [0])
    return b.graph(b.add(Kind("Union"), [d, b.add(Kind("Torus", radius=1.5, tube=0.1), [still])]))


GRAPHS = {"one op": lambda: Graph.bundled("sphere"), "kitchen sink": kitchen_sink, "bounded": bounded_bulb,
          "union": lambda: world((3, 1, 2, 0), True), "nine leaves": union_world, "copies": lambda: copies_of_a_bulb(1),
          "nested copies": lambda: copies_of_a_bulb(2)}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_lanes_together_and_apart(renderer, name):
    """Runs of ops between the places where a warp's lanes part and join: the same points
    beside others of every distance, and with a warp to each, sample for sample."""
    g = renderer.compile(GRAPHS[name]())
    pts = np.concatenate([lcg_points(500, 2.5, 17), lcg_points(499, 30.0, 18)])
    mixed, alone = g.probe(pts[np.random.default_rng(4).permutation(len(pts))]), g.probe(np.repeat(pts, 32, axis=0))
    order = np.random.default_rng(4).permutation(len(pts))
    for k in ("distance", "material", "iterations", "traps"):
        np.testing.assert_array_equal(mixed[k], alone[k][::32][order], err_msg=k)
        np.testing.assert_array_equal(alone[k][::32], alone[k][31::32], err_msg=k)
