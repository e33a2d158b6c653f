"""The Mandelbox form's two-instruction fold and its loop of iteration pairs: limits of
zero, inside and past the points, and the largest it takes, with odd and even iteration
counts; a limit past 1e38 takes the plain loop. All follow the f32 oracle (the rule and the
few-ulp quantile of the form tests). A negative limit, where clamp(-x, -l, l) is l, folds x
to -2 l - x on this form; a value edit between the two kinds reaches a batch that exists."""
import numpy as np
import pytest

from helpers import lcg_points
from syfrack_gb300.graph import Graph
from test_gpu_de import gpu_de_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0.0, 0.35, 1.0, 2.5, 1e38, 2e38])
@pytest.mark.parametrize("iterations", [1, 2, 3, 4])
def test_limits_and_iteration_pairs(renderer, oracle_mod, limit, iterations):
    g = Graph.bundled("mandelbox", limit=limit, iterations=iterations, scale=-1.5, bailout=1000.0)
    cg = renderer.compile(g)
    assert cg.info()["form"] == "box"
    pts = lcg_points(4096, 4.0, 21 + iterations)
    pts[:8] = [(x, y, z) for x in (0.35, -0.7) for y in (1.0, -2.0) for z in (2.5, 0.0)]  # at l and 2 l
    gpu = cg.probe(pts)
    ref = oracle_mod.OracleGraph(g).de(pts, precision=32)
    assert gpu_de_rule(gpu, ref) <= 0.005
    rel = np.abs(gpu["distance"] - ref["distance"]) / np.maximum(np.abs(ref["distance"]), 1.0)
    assert np.quantile(rel, 0.99) < 1e-5
    assert (gpu["iterations"] == ref["iterations"]).mean() >= 0.995


@pytest.mark.parametrize("iterations", [1, 2, 3])
def test_negative_limit(renderer, iterations):
    limit, scale = -0.5, -1.5
    g = Graph.bundled("mandelbox", limit=limit, iterations=iterations, scale=scale, bailout=1000.0)
    pts = lcg_points(4096, 2.0, 33)
    gpu = renderer.compile(g).probe(pts)
    p = c = pts.astype(np.float64)
    dr = np.ones(len(pts))
    for _ in range(iterations):
        q = -2.0 * limit - p
        k = np.minimum(4.0, np.maximum(1.0 / (q * q).sum(1), 1.0))  # radii 0.5 and 1
        p, dr = q * (k * scale)[:, None] + c, dr * k * abs(scale) + 1.0
    fence = [n for n in g.nodes if n.kind.name == "NormFence"][0].kind.fields["inset"]
    ref = (np.linalg.norm(p, axis=1) - fence) / dr
    rel = np.abs(gpu["distance"] - ref) / np.maximum(np.abs(ref), 1.0)
    assert np.quantile(rel, 0.99) < 1e-5
    assert np.all(gpu["iterations"] == iterations)


def test_value_edit_across_the_limits(renderer):
    """sf_graph_update from a limit of 1 to -0.5 and back: the batch made before renders as
    one made after."""
    from syfrack_gb300 import Batch, workloads
    from syfrack_gb300.scene import RenderConfig

    cfg = RenderConfig(48, 32, 2, max_bounces=2, max_steps=128, pixel_tolerance=1.0, tile_size=48,
                       samples_per_dispatch=2, integrator="wavefront")

    def film(scene, edit=None):
        b = Batch(renderer, [(scene, cfg)])
        if edit is not None:
            edit(b)
        b.run(1, use_graph=False)
        assert b.sync() == 0
        out = b.readback(0)
        b.close()
        return out

    scene = workloads.mandelbox_scene()
    other = workloads.mandelbox_scene()
    for n in other.graph.nodes:
        if n.kind.name == "BoxFold":
            n.kind.fields["limit"] = -0.5
    want = film(other)
    cg = renderer.compile(scene.graph)
    got = film(scene, lambda b: cg.update(other.graph))
    cg.update(scene.graph)
    np.testing.assert_array_equal(got.accum, want.accum)
    np.testing.assert_array_equal(got.depth, want.depth)


@pytest.mark.parametrize("measure", ["AngleXY", "AngleXZ", "AngleYZ"])
@pytest.mark.parametrize("limit", [0.5, 1.0])
def test_angles_of_folded_lattice_points(renderer, oracle_mod, measure, limit):
    """Components that fold to zero (0, -0 and both ends 2 l, -2 l) fold to +0: an angle on
    the negative axis is pi, not -pi. One iteration, so the folds are exact and the angle
    is within 3 ulp of pi (7e-7) over 2 pi, plus the rounding of the sum with a half."""
    g = Graph.bundled("mandelbox", limit=limit, iterations=1, scale=-1.5, bailout=1000.0, trap_scale=1.0)
    for n in g.nodes:
        if n.kind.name == "Trap":
            n.kind.fields["measure"] = measure
    axis = np.array([-4.0, -2.0, -1.4, -1.0, -0.6, -0.0, 0.0, 0.6, 1.0, 1.4, 2.0, 4.0], np.float32) * np.float32(limit)
    pts = np.stack(np.meshgrid(axis, axis, axis, indexing="ij"), -1).reshape(-1, 3)
    gpu = renderer.compile(g).probe(pts)
    ref = oracle_mod.OracleGraph(g).de(pts, precision=32)
    np.testing.assert_allclose(gpu["traps"][:, 0], ref["traps"][:, 0], rtol=0, atol=1e-6)
