"""Escape-time sampling on the GPU against the oracle (GPU).

Iteration counts are bit-exact against the reference's binary32 arithmetic
(the f32 oracle): the device evaluates the orbit with unfused, explicitly
rounded operations. Traps follow gpu_planar.rs:101-130 (within 0.006; Newton
and Nova smooth time within 0.09)."""
import numpy as np
import pytest

from syfrack_gb300 import Canvas, PlanarFractal, escape2d
from syfrack_gb300.render import FAMILIES

pytestmark = pytest.mark.gpu


def oracle_params(oracle_mod, f: PlanarFractal):
    p = oracle_mod.PlanarParams()
    p.family = FAMILIES.index(f.family)
    p.power, p.iterations = f.power, f.iterations
    p.julia[:] = [float(np.float32(x)) for x in f.julia]
    p.center[:] = [float(np.float32(x)) for x in f.center]
    for k in ("zoom", "angle", "inversion", "twist", "relaxation", "memory", "bailout", "trap_radius", "stripes"):
        setattr(p, k, float(np.float32(getattr(f, k))))
    return p


def grid289():
    xs = np.linspace(-1.6, 1.6, 17, dtype=np.float32)
    return np.array([[x, y] for y in xs for x in xs], np.float32)


@pytest.mark.parametrize("family", FAMILIES)
def test_planar_iterations_bit_exact(gpu_ctx, oracle_mod, family):
    rng = np.random.default_rng(5)
    pts = np.concatenate([grid289(), rng.uniform(-2, 2, (4000, 2)).astype(np.float32)])
    for power in (2, 3):
        f = PlanarFractal(family=family, power=power, iterations=256)
        gpu = f.sample(gpu_ctx, pts)
        ref = oracle_mod.planar(oracle_params(oracle_mod, f), pts, precision=32)
        np.testing.assert_array_equal(gpu["iterations"], ref["iterations"])
        d = np.abs(gpu["traps"] - ref["traps"])
        assert np.quantile(d[:, 1:], 0.999) <= 0.006
        tol = 0.09 if family in ("Newton", "Nova") else 0.006
        assert np.quantile(d[:, 0], 0.999) <= tol
        np.testing.assert_allclose(gpu["distance"], ref["distance"], atol=1e-5)


def test_planar_mapping_bit_exact(gpu_ctx, oracle_mod):
    f = PlanarFractal(family="Julia", iterations=300, zoom=1.7, angle=30.0, inversion=0.8, twist=12.0,
                      center=(0.1, -0.2))
    pts = np.random.default_rng(2).uniform(-1.5, 1.5, (8192, 2)).astype(np.float32)
    np.testing.assert_array_equal(f.sample(gpu_ctx, pts)["iterations"],
                                  oracle_mod.planar(oracle_params(oracle_mod, f), pts, precision=32)["iterations"])


def canvas_points(c: Canvas, sample=None):
    """The flat-canvas map (pathtrace.wgsl:1226-1239) in unfused binary32."""
    f = np.float32
    ys, xs = np.mgrid[0:c.height, 0:c.width]
    jx = np.full(xs.shape, f(0.5), np.float32)
    jy = jx.copy()
    u = (xs.astype(np.float32) + jx) / f(c.width)
    v = (ys.astype(np.float32) + jy) / f(c.height)
    scale = f(6.0) / f(c.zoom)
    aspect = f(c.width) / f(c.height)
    ax = (u - f(0.5)) * scale
    ay = ((f(0.5) - v) / aspect) * scale
    r = f(c.rotation) * f(np.pi / 180.0)
    cs, sn = f(np.cos(r)), f(np.sin(r))
    qx = f(c.center[0]) + (cs * ax - sn * ay)
    qy = f(c.center[1]) + (sn * ax + cs * ay)
    return np.stack([qx.ravel(), qy.ravel()], 1).astype(np.float32)


def test_escape2d_canvas_against_oracle(gpu_ctx, oracle_mod):
    c = Canvas(width=160, height=90, center=(-0.5, 0.0), zoom=2.0)
    f = PlanarFractal(family="Mandelbrot", iterations=2000)
    out = escape2d(gpu_ctx, f, c)
    ref = oracle_mod.planar(oracle_params(oracle_mod, f), canvas_points(c), precision=32)
    np.testing.assert_array_equal(out["iterations"].ravel(), ref["iterations"])


def test_beyond_reference_caps(gpu_ctx, oracle_mod):
    # 20,000 iterations and zoom 1e5 (the reference caps 512 and 1e4), seahorse valley
    f = PlanarFractal(family="Mandelbrot", iterations=20000, zoom=1e5, center=(-0.7436, 0.1318))
    pts = np.random.default_rng(8).uniform(-1, 1, (2048, 2)).astype(np.float32)
    gpu = f.sample(gpu_ctx, pts)
    ref = oracle_mod.planar(oracle_params(oracle_mod, f), pts, precision=32)
    np.testing.assert_array_equal(gpu["iterations"], ref["iterations"])
    assert gpu["iterations"].max() > 512


def test_tiles_and_jitter(gpu_ctx):
    c = Canvas(width=64, height=48, seed=3)
    f = PlanarFractal(family="Julia", iterations=200)
    full = escape2d(gpu_ctx, f, c, sample=5)
    part = escape2d(gpu_ctx, f, c, tile=(16, 8, 32, 20), sample=5)
    np.testing.assert_array_equal(part["iterations"], full["iterations"][8:28, 16:48])
    other = escape2d(gpu_ctx, f, c, sample=6)
    assert (other["iterations"] != full["iterations"]).any()


@pytest.mark.parametrize("stripes", [12.0, -5.0, 7.5, 0.0])
def test_stripe_bands_integer_and_general(gpu_ctx, oracle_mod, stripes):
    # integer stripe counts use sin(k theta) = Im(u^k); others use sin(k * atan2)
    f = PlanarFractal(family="Mandelbrot", iterations=400, stripes=stripes)
    pts = np.random.default_rng(12).uniform(-2.0, 1.0, (6000, 2)).astype(np.float32)
    gpu = f.sample(gpu_ctx, pts)
    ref = oracle_mod.planar(oracle_params(oracle_mod, f), pts, precision=32)
    np.testing.assert_array_equal(gpu["iterations"], ref["iterations"])
    d = np.abs(gpu["traps"] - ref["traps"])
    assert np.quantile(d, 0.999) <= 0.006


def test_escape2d_without_traps_keeps_counts(gpu_ctx):
    from syfrack_gb300 import Renderer, Server

    c = Canvas(width=200, height=120, center=(-0.45, -0.5), zoom=2.0)
    f = PlanarFractal(family="BurningShip", iterations=3000)
    full = escape2d(gpu_ctx, f, c)
    srv = Server(Renderer(gpu_ctx), hbm_budget=1 << 28)
    lean = srv.wait(srv.tile(f, c, traps=False))
    srv.close()
    assert lean.traps is None and lean.distance is None
    np.testing.assert_array_equal(lean.iterations, full["iterations"])
    np.testing.assert_array_equal(lean.smooth, full["traps"][0])


@pytest.mark.parametrize("iterations", [1, 15, 16, 17, 32, 49])
@pytest.mark.parametrize("family", ["Julia", "Mandelbrot", "BurningShip", "Phoenix"])
def test_escape2d_around_the_chunk(gpu_ctx, oracle_mod, family, iterations):
    """Budgets around the 16 iterations an orbit runs without a branch: counts bit for
    bit, traps within the 0.006 of the reference's own parity test on all but one pixel
    in a thousand (a ring or band next to a discontinuity)."""
    c = Canvas(width=97, height=61, center=(-0.4, -0.1), zoom=1.7)
    f = PlanarFractal(family=family, iterations=iterations)
    out = escape2d(gpu_ctx, f, c)
    ref = oracle_mod.planar(oracle_params(oracle_mod, f), canvas_points(c), precision=32)
    np.testing.assert_array_equal(out["iterations"].ravel(), ref["iterations"])
    d = np.abs(out["traps"].reshape(4, -1).T - ref["traps"])
    assert np.quantile(d, 0.999) <= 0.006
    # the general loop (five stripes) runs the same orbit
    g = escape2d(gpu_ctx, PlanarFractal(family=family, iterations=iterations, stripes=5.0), c)
    np.testing.assert_array_equal(g["iterations"], out["iterations"])
    np.testing.assert_array_equal(g["distance"], out["distance"])
    np.testing.assert_array_equal(g["traps"][0], out["traps"][0])


@pytest.mark.parametrize("family,twist,bailout", [("Julia", 10.0, 1000.0), ("Mandelbrot", -25.0, 50.0),
                                                  ("BurningShip", 10.0, 1000.0), ("Phoenix", 10.0, 1000.0),
                                                  ("Mandelbrot", 0.0, 1.2e19), ("BurningShip", 0.0, 1.5e19),
                                                  ("Phoenix", 0.0, 1.2e19), ("Julia", 0.0, 1e30)])
def test_escape2d_twelve_stripes_off_the_common_loop(gpu_ctx, oracle_mod, family, twist, bailout):
    """The default 12 stripes with a twist (their own loop) and with bailouts on either side
    of the largest that the z^2 loop takes: counts bit for bit, traps within the 0.006 of the
    reference's own parity test on all but one pixel in a thousand."""
    c = Canvas(width=97, height=61, center=(-0.4, -0.1), zoom=1.7)
    f = PlanarFractal(family=family, iterations=85, twist=twist, bailout=bailout)
    out = escape2d(gpu_ctx, f, c)
    ref = oracle_mod.planar(oracle_params(oracle_mod, f), canvas_points(c), precision=32)
    np.testing.assert_array_equal(out["iterations"].ravel(), ref["iterations"])
    d = np.abs(out["traps"].reshape(4, -1).T - ref["traps"])
    assert np.quantile(d, 0.999) <= 0.006
    np.testing.assert_allclose(out["distance"].ravel(), ref["distance"], atol=1e-5)


@pytest.mark.parametrize("bailout,term", [(16.0, 7.4e-6), (1e30, 1.4e-5)])
def test_long_stripe_sums_against_64_bits(gpu_ctx, bailout, term):
    """The stripe band of interior pixels after 20,000 iterations, in the z^2 loop (double
    angle) and the unrolled recurrence (a bailout past that loop), against the sum in 64
    bits over the same binary32 orbit. A term is off by at most `term`, and each addition to
    a sum of at most n by half of an ulp of n; the band is half of the mean."""
    n = 20000
    c = Canvas(width=33, height=17, center=(-0.1, 0.1), zoom=20.0)
    out = escape2d(gpu_ctx, PlanarFractal(family="Mandelbrot", iterations=n, bailout=bailout), c)
    assert np.all(out["iterations"] == n)
    cx, cy = np.ascontiguousarray(canvas_points(c).astype(np.float32).T)
    x, y, total = np.zeros_like(cx), np.zeros_like(cx), np.zeros(len(cx))
    for _ in range(n):
        total += np.sin(12.0 * np.arctan2(y.astype(np.float64), x.astype(np.float64)))
        m = x * y
        x, y = (x * x - y * y) + cx, (m + m) + cy
    assert x.dtype == np.float32
    err = np.abs(out["traps"][2].ravel() - (0.5 + 0.5 * total / n))
    print(f"bailout {bailout:g}: stripe band error max {err.max():.3e}, rms {np.sqrt(np.mean(err ** 2)):.3e}")
    assert err.max() <= 0.5 * term + 0.25 * float(np.spacing(np.float32(n))) + 1e-6


def test_tiles_around_the_staged_size(gpu_ctx):
    """Three planes, 24 bytes a pixel: 16,384 go through the pinned staging (3 x 128 KB), 16,385
    straight to the caller."""
    f, c = PlanarFractal(family="Julia", iterations=60), Canvas(width=16385, height=1, center=(-0.1, 0.05), zoom=1.5)
    a, b = escape2d(gpu_ctx, f, c), escape2d(gpu_ctx, f, c, tile=(0, 0, 16384, 1))
    assert len(np.unique(a["iterations"])) > 10
    for k in ("iterations", "distance", "traps"):
        np.testing.assert_array_equal(a[k][..., :16384], b[k], err_msg=k)
