"""The Mandelbox form's two-instruction fold and its loop of iteration pairs: limits of
zero, inside and past the points, and the largest it takes, with odd and even iteration
counts; limits outside 0..1e38 run on the generic interpreter. All follow the f32 oracle
(the rule and the few-ulp quantile of the form tests)."""
import numpy as np
import pytest

from helpers import lcg_points
from syfrack_gb300.graph import Graph
from test_gpu_de import gpu_de_rule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit,form", [(0.0, "box"), (0.35, "box"), (1.0, "box"), (2.5, "box"), (1e38, "box"),
                                        (-0.5, "generic"), (2e38, "generic")])
@pytest.mark.parametrize("iterations", [1, 2, 3, 4])
def test_limits_and_iteration_pairs(renderer, oracle_mod, limit, form, iterations):
    g = Graph.bundled("mandelbox", limit=limit, iterations=iterations, scale=-1.5, bailout=1000.0)
    cg = renderer.compile(g)
    assert cg.info()["form"] == form
    pts = lcg_points(4096, 4.0, 21 + iterations)
    pts[:8] = [(x, y, z) for x in (0.35, -0.7) for y in (1.0, -2.0) for z in (2.5, 0.0)]  # at l and 2 l
    gpu = cg.probe(pts)
    ref = oracle_mod.OracleGraph(g).de(pts, precision=32)
    assert gpu_de_rule(gpu, ref) <= 0.005
    rel = np.abs(gpu["distance"] - ref["distance"]) / np.maximum(np.abs(ref["distance"]), 1.0)
    assert np.quantile(rel, 0.99) < 1e-5
    assert (gpu["iterations"] == ref["iterations"]).mean() >= 0.995
