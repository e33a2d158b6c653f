"""Deep zoom: FP64 reference orbit + FP32 perturbation with rebasing (GPU),
checked against IEEE binary128 direct iteration on a seeded pixel subsample
(the truth) and against full-FP64 direct iteration on every pixel."""
import numpy as np
import pytest

from syfrack_gb300 import deep_zoom, workloads

pytestmark = pytest.mark.gpu


def offsets(w, h, pitch, idx):
    f = np.float32
    px, py = idx % w, idx // w
    dx = (px.astype(np.float32) - f(w) * f(0.5) + f(0.5)) * f(pitch)
    dy = (f(h) * f(0.5) - py.astype(np.float32) - f(0.5)) * f(pitch)
    return np.stack([dx, dy], 1).astype(np.float64)


def test_deep_zoom_against_binary128(gpu_ctx, oracle_mod):
    max_iter = 20000
    c = workloads.deep_zoom_center(seed=2026, max_iter=max_iter)
    w, h, width = 192, 108, 1e-12
    out = deep_zoom(gpu_ctx, c, (0.0, 0.0), width, w, h, max_iter, bailout=16.0, reference_f64=True)
    it = out["iterations"].ravel()
    assert it.min() < max_iter and it.max() > 100  # the view straddles the boundary
    idx = np.random.default_rng(0).choice(w * h, 96, replace=False)
    pitch = np.float32(width / w)
    truth, _ = oracle_mod.mandel_escape(np.array(c), np.zeros(2), offsets(w, h, pitch, idx), max_iter, 16.0,
                                        precision=128)
    match = (it[idx] == truth).mean()
    near = (np.abs(it[idx].astype(np.int64) - truth.astype(np.int64)) <= 1).mean()
    agree64 = (out["iterations_f64"].ravel() == it).mean()
    match64 = (out["iterations_f64"].ravel()[idx] == truth).mean()
    print(f"deep zoom: match vs binary128 {match:.3f} (+-1: {near:.3f}), FP64 direct vs binary128 {match64:.3f}, "
          f"perturbation vs FP64 {agree64:.3f}, rebases {out['rebases']}")
    # FP32 deltas resolve most pixels; near the set's boundary the remaining orbit is
    # too sensitive for binary32 once it leaves the reference. Regression floor, and
    # no worse than full-FP64 direct iteration (whose pixel pitch is ~1 ulp of c).
    assert match >= 0.65 and near >= 0.70, (match, near)
    assert match >= match64 - 0.05, (match, match64)
    assert agree64 >= 0.3
    s = out["smooth"].ravel()[idx]
    esc = truth < max_iter
    # n + 1 - log2(ln|z_n|) with bailout < |z_n| <= bailout^2 lies in (n - 1.46, n - 0.47) for bailout 16
    assert np.all(np.isfinite(s)) and np.all(s[esc] >= it[idx][esc] - 1.5) and np.all(s[esc] <= it[idx][esc])


def test_shallow_zoom_matches_fp64_everywhere(gpu_ctx):
    # at width 1e-3 FP64 direct iteration is trustworthy: counts agree on almost every pixel
    out = deep_zoom(gpu_ctx, (-0.743, 0.131), (0.0, 0.0), 1e-3, 160, 90, 4000, bailout=16.0, reference_f64=True)
    agree = (out["iterations"] == out["iterations_f64"]).mean()
    near = (np.abs(out["iterations"].astype(np.int64) - out["iterations_f64"].astype(np.int64)) <= 1).mean()
    print(f"shallow zoom: perturbation vs FP64 {agree:.4f} (+-1: {near:.4f})")
    assert agree >= 0.93 and near >= 0.95, (agree, near)


def test_full_frame_against_binary128_with_orbit_decomposition(gpu_ctx, oracle_mod):
    """The deep-zoom configuration as stated (3840x2160, 50,000 iterations, width
    1e-12 around the seeded boundary point, FP64 reference orbit on the GPU, FP32
    deltas with rebasing) on 4096 seeded pixels against binary128 direct iteration.
    The same frame with the oracle's binary128 reference orbit (stored as the same
    hi/lo float pairs) separates the FP64 orbit's error from the FP32 deltas'; the
    host's FP64 orbit gives the device's bit for bit."""
    MI, W, H, width = 50000, 3840, 2160, 1e-12
    c = workloads.deep_zoom_center(seed=2026, max_iter=MI)
    dev = deep_zoom(gpu_ctx, c, (0.0, 0.0), width, W, H, MI, bailout=16.0, reference_f64=True)
    host = deep_zoom(gpu_ctx, c, (0.0, 0.0), width, W, H, MI, bailout=16.0, orbit="host")
    np.testing.assert_array_equal(dev["iterations"], host["iterations"])
    np.testing.assert_array_equal(dev["smooth"], host["smooth"])
    q = deep_zoom(gpu_ctx, c, (0.0, 0.0), width, W, H, MI, bailout=16.0, orbit="given",
                  given_orbit=oracle_mod.mandel_orbit(c, MI, 16.0, precision=128))
    idx = np.random.default_rng(11).choice(W * H, 4096, replace=False)
    truth, _ = oracle_mod.mandel_escape(np.array(c), np.zeros(2), offsets(W, H, np.float32(width / W), idx), MI, 16.0,
                                        precision=128)
    it, it64, itq = (x.ravel()[idx] for x in (dev["iterations"], dev["iterations_f64"], q["iterations"]))
    m = lambda a: float((a == truth).mean())
    near = float((np.abs(it.astype(np.int64) - truth.astype(np.int64)) <= 1).mean())
    agree64 = float((dev["iterations"] == dev["iterations_f64"]).mean())
    print(f"deep zoom 3840x2160 50k vs binary128 on 4096 px: perturbation (FP64 orbit) {m(it):.3f} (+-1 {near:.3f}), "
          f"perturbation (binary128 orbit) {m(itq):.3f}, FP64 direct {m(it64):.3f}; "
          f"perturbation vs FP64 direct on all pixels {agree64:.3f}; interior {(truth == MI).mean():.3f}")
    assert it.min() < MI and (truth == MI).mean() < 0.9  # the view straddles the boundary
    # floors of this chaotic view (pixel pitch ~1 FP64 ulp of c): no worse than full-FP64 iteration
    assert m(it) >= 0.25 and near >= 0.30, (m(it), near)
    assert m(it) >= m(it64) - 0.05, (m(it), m(it64))
    # a more accurate orbit does not make the perturbation worse
    assert m(itq) >= m(it) - 0.05, (m(itq), m(it))


def test_centre_lo_moves_the_view_below_an_fp64_ulp(gpu_ctx, oracle_mod):
    """The centre's lo part (a fraction of a pixel here, below an FP64 ulp of hi) joins
    every pixel's offset: the counts change, and they follow binary128 iteration at
    hi + lo as well as the lo = 0 view follows its own."""
    max_iter, w, h, width = 20000, 192, 108, 1e-12
    c = workloads.deep_zoom_center(seed=2026, max_iter=max_iter)
    pitch = np.float32(width / w)
    lo = (0.37 * float(pitch), -0.21 * float(pitch))
    a = deep_zoom(gpu_ctx, c, (0.0, 0.0), width, w, h, max_iter, bailout=16.0)["iterations"].ravel()
    b = deep_zoom(gpu_ctx, c, lo, width, w, h, max_iter, bailout=16.0)["iterations"].ravel()
    assert (a != b).mean() > 0.05
    idx = np.random.default_rng(5).choice(w * h, 96, replace=False)
    off = offsets(w, h, pitch, idx)
    ta, _ = oracle_mod.mandel_escape(np.array(c), np.zeros(2), off, max_iter, 16.0, precision=128)
    tb, _ = oracle_mod.mandel_escape(np.array(c), np.array(lo), off, max_iter, 16.0, precision=128)
    print(f"centre lo: view changed on {(a != b).mean():.3f} of pixels; match vs binary128 lo=0 "
          f"{(a[idx] == ta).mean():.3f}, with lo {(b[idx] == tb).mean():.3f}")
    assert (b[idx] == tb).mean() >= 0.6


@pytest.mark.parametrize("max_iter", [1, 2, 7, 8, 9, 12, 16, 17, 40])
def test_budgets_around_the_chunk(gpu_ctx, max_iter):
    """Budgets around the 8 iterations a pixel runs without a branch and the 4 orbit
    entries of a load. At this width a count differs from FP64 direct iteration only
    where binary32's rounding, grown by the orbit, decides the last step: under a
    hundredth of the pixels. The host's orbit gives the device's frame bit for bit."""
    args = dict(center_hi=(-0.75, 0.1), center_lo=(0.0, 0.0), width_units=2.5, width=101, height=67,
                max_iter=max_iter)
    a = deep_zoom(gpu_ctx, **args, reference_f64=True)
    b = deep_zoom(gpu_ctx, **args, orbit="host")
    assert (a["iterations"] == a["iterations_f64"]).mean() >= 0.99
    for k in ("iterations", "smooth", "rebases"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("max_iter", [59, 60, 61, 700])
@pytest.mark.parametrize("centre,width", [((0.5, 0.6), 3.0), ((-0.75, 0.1), 0.3), ((-0.75, 0.1), 0.01),
                                          ((0.27868532354762443, 0.5820921261345181), 0.01)])
def test_dense_rebases(gpu_ctx, centre, width, max_iter):
    """Views whose pixels rebase every few iterations (a reference that escapes after 5 or
    33 iterations, offsets of the orbit's own size), where warps leave the chunks for runs
    of 60 checked iterations and come back. Counts differ from FP64 direct iteration only
    where binary32's rounding, grown by the orbit, decides the last step."""
    args = dict(center_hi=centre, center_lo=(0.0, 0.0), width_units=width, width=131, height=93, max_iter=max_iter)
    a = deep_zoom(gpu_ctx, **args, reference_f64=True)
    b = deep_zoom(gpu_ctx, **args, orbit="host")
    inside = a["iterations_f64"] < max_iter
    # an offset grows by 2 |z| an iteration, so long orbits lose more of the 24 bits
    assert (a["iterations"] == a["iterations_f64"]).mean() >= (0.99 if max_iter <= 61 else 0.95)
    assert inside.any() and a["rebases"] >= 131 * 93 * (1 if width >= 0.3 else 0)
    for k in ("iterations", "smooth", "rebases"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
