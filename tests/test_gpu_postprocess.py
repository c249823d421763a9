"""What runs before and after the steps, at the sizes where its kernels change
shape: the rasteriser's identity shortcut against the CPU evaluation of the
same programs, spectra with one, a few and many monitors, phases of odd, even,
smallest and largest series."""
import numpy as np
import pytest

from oracle.oracle import rasterize as oracle_rasterize, rasterize_counts as oracle_counts
from sim_juncs_gb300 import _abi
from sim_juncs_gb300.configs import junction_instance
from sim_juncs_gb300.fields import Fields, rasterize, rasterize_counts
from sim_juncs_gb300.geometry import Box, Cylinder, Difference, Intersect, Plane, Sphere, Union, rotation
from sim_juncs_gb300.phases import extract_phases
from sim_juncs_gb300.spec import Grid, Probe, Region, Scene

pytestmark = pytest.mark.gpu

MINUS = (1.0, -0.0, 0.0, 0.0, 1.0, -0.0, -0.0, 0.0, 1.0)     # an identity with negative zeros
NEAR = (1.0, 1e-17, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0)       # not one
ROT = rotation(0.3, (1.0, 2.0, -0.5))


@pytest.mark.parametrize("trans", [None, MINUS, NEAR, ROT], ids=["identity", "minus", "near", "rotated"])
def test_rasteriser_matches_the_cpu_for_every_transform(lib, oracle_lib, trans):
    # faces through Yee points (0.125 spacing, origin at a negative corner, so that coordinates of 0 and -0 occur)
    kw = {} if trans is None else {"trans": trans}
    roots = [Union(Box((-0.5, -0.25, -0.125), (0.25, 0.5, 0.125), **kw), Sphere((0.0, 0.0, 0.0), 0.375, **kw)),
             Difference(Box((-1.0, -1.0, -1.0), (1.0, 1.0, 0.0), **kw), Cylinder((0.0, 0.0, -0.5), 0.5, 0.25, 0.375, **kw)),
             Intersect(Plane((1.0, 1.0, 0.0), 0.25), Box((-0.5, -0.5, -0.5), (0.5, 0.5, 0.0), invert=1, **kw))]
    scene = Scene([Region(r) for r in roots])
    g = Grid(17, 19, 15, 0.125, origin=(-1.0, -1.125, -0.9375))
    dev = rasterize(g, scene)
    np.testing.assert_array_equal(dev, oracle_rasterize(g, scene))
    assert all(0 < np.count_nonzero(dev & (1 << r)) < dev.size for r in range(3))


@pytest.mark.parametrize("origin", [(-1.0, -1.125, -0.9375), (1.2e308, 0.0, 0.0)], ids=["near", "overflow"])
def test_rasteriser_with_infinite_numbers(lib, oracle_lib, origin):
    """A centre that is not a number (a half-space given as a box) or so far that r - c overflows: then the product with
    an identity is not the point."""
    inf = float("inf")
    roots = [Box((-0.5, -0.5, -inf), (0.25, 0.5, 0.0)), Sphere((inf, 0.0, 0.0), 0.5), Cylinder((0.0, 0.0, -0.5), inf, 0.25, 0.375),
             Box((-0.5, -0.5, -0.5), (0.25, inf, 0.5)), Sphere((-1.5e308, 0.0, 0.0), inf)]
    scene = Scene([Region(r) for r in roots])
    g = Grid(17, 19, 15, 0.125, origin=origin)
    np.testing.assert_array_equal(rasterize(g, scene), oracle_rasterize(g, scene))


@pytest.mark.parametrize("nx", [1, 15, 16, 17, 32, 75])
@pytest.mark.parametrize("x0", [-1.0, 1e101], ids=["near", "far"])
def test_rasteriser_rows_match_the_cpu(lib, oracle_lib, nx, x0):
    """Whole segments of a row decided at their ends: primitives smaller than a segment, tangent to rows, of zero,
    negative and infinite extent, around, left and right of each segment."""
    rng = np.random.default_rng(nx)
    inf = float("inf")

    def leaf():
        c = tuple(np.round(rng.uniform(-1, 1, 3) * [nx / 16 + 0.5, 1, 1], 2))
        s = [float(x) for x in np.round(rng.uniform(0.05, 0.8, 3), 2)]
        return [lambda: Box(tuple(np.subtract(c, s)), tuple(np.add(c, s)), invert=int(rng.integers(2))),
                lambda: Sphere(c, s[0], invert=int(rng.integers(2))),
                lambda: Cylinder(c, *s),
                lambda: Plane(tuple(rng.normal(size=3)), float(rng.uniform(-1, 1)))][rng.integers(4)]()

    roots = [Union(Intersect(leaf(), leaf()), Difference(leaf(), leaf())) for _ in range(3)]
    roots += [Union(Sphere((0.0625, 0.0, 0.0), 0.0), Sphere((0.5, 0.0, 0.0), 0.0625)),   # one point, two points of a row
              Intersect(Plane((1.0, 0.0, 0.0), 0.25), Plane((-1.0, 1.0, 0.0), -0.25)),
              Union(Box((0.25, -0.5, -0.5), (-0.25, 0.5, 0.5)), Sphere((0.0, 0.0, 0.0), -0.25))]
    endless = Union(Cylinder((0.0, 0.0, -0.5), inf, 0.25, 0.375), Box((-0.5, -0.5, -inf), (0.25, 0.5, 0.0)))
    n = int(np.sqrt(2 ** 19 / nx)) + 1   # enough points for the segments
    g = Grid(nx, n, n, 0.125, origin=(x0, -0.125 * (n // 2), -0.125 * (n // 3)))
    for rs in (roots, roots + [endless]):   # the second: every point evaluated
        scene = Scene([Region(r) for r in rs])
        np.testing.assert_array_equal(rasterize(g, scene), oracle_rasterize(g, scene))
        scene = Scene([Region(r) for r in rs], smooth_n=1, smooth_rad=0.1)
        counts = rasterize_counts(g, scene)
        np.testing.assert_array_equal(counts, oracle_counts(g, scene))
        assert x0 > 0 or np.count_nonzero((counts > 0) & (counts < 9))


@pytest.mark.parametrize("monitors", [1, 3, 8, 9, 700])
@pytest.mark.parametrize("samples", [1, 2, 3, 65, 300])
def test_spectrum_matches_the_direct_sum(lib, monitors, samples):
    inst = junction_instance(n=24, res=7.5, pml_um=0.4)
    inst.sources[0].start_time, inst.sources[0].end_time = -9.0, 11.0
    inst.probes = [Probe(_abi.EX, (1.6 + 0.0005 * q, 1.6, 0.7)) for q in range(monitors)]
    inst.freqs, inst.save_span = [], 1
    f = Fields(inst, "f64")
    f.step(samples)
    x, got = f.monitors(), f.monitor_spectrum()
    n2 = 1 << int(np.log(samples) / np.log(2.0))
    assert got.shape == (monitors, n2)
    if n2 == 1:
        assert not got.any()   # the reference's transform leaves a single sample at zero
        return
    k = np.where(np.arange(n2) < n2 // 2, np.arange(n2), np.arange(n2) - n2)
    ph = np.exp(-2j * np.pi * (np.outer(np.arange(n2), k) % samples) / samples)
    want = x[:, :n2] @ ph
    # n2 terms of relative rounding 2^-52 each
    assert np.max(np.abs(got - want)) <= 4 * n2 * 2.0 ** -52 * np.max(np.abs(x[:, :n2]).sum(1))
    assert samples < 65 or np.max(np.abs(want)) > 0


def reference_estimate(t, v):
    """f0, phi and t0_corr of one clean pulse: numpy's rfft of the series rolled by the |v|-weighted mean index of the
    peaks of v^2, the trapezoid-mean frequency below twice the largest bin, and the regression of the unwrapped
    phase over the bins above a tenth of |V(f0)|, recentred at most once."""
    n = len(v)
    x = v * v
    pk = np.array([i for i in range(1, n - 1) if x[i - 1] < x[i] > x[i + 1]])
    t0 = int((pk * np.abs(v[pk])).sum() / np.abs(v[pk]).sum())
    df = 1.0 / (n * (t[1] - t[0]))

    def regress(t0):
        V = 2 * np.fft.rfft(np.roll(v, -t0))
        mag = np.abs(V)
        top = min(2 * int(np.argmax(mag)), len(mag))
        fr = np.arange(len(mag)) * df
        trap = lambda y: ((y[1:] + y[:-1]) / 2).sum()  # noqa: E731
        f0 = trap((mag * fr)[:top]) / trap(mag[:top])
        fi = int(np.rint(f0 / df))
        jb = min(fi, len(mag) - fi - 1)
        lo = min(fi - j - 1 for j in range(jb) if mag[fi - j] > 0.1 * mag[fi])
        hi = max(fi + j + 1 for j in range(jb) if mag[fi + j] > 0.1 * mag[fi])
        ang = np.unwrap(np.angle(V[lo:hi]))
        slope, icpt = np.polyfit(fr[lo:hi], ang, 1)
        return f0, -slope / (2 * np.pi), icpt, lo, hi

    f0, tc, icpt, lo, hi = regress(t0)
    if abs(tc) > 2.0 / (hi - lo):
        _, tc, icpt, lo, hi = regress(t0 + int(tc / (t[1] - t[0])))
    return f0, tc, icpt, (lo, hi)


@pytest.mark.parametrize("n", [64, 65, 127, 128, 129, 257, 1000, 4095, 4096])
def test_phases_of_clean_pulses(lib, n):
    # a carrier at 0.3 of the sampling's Nyquist frequency under an envelope n / 12 samples wide
    rng = np.random.default_rng(n)
    t = np.arange(n) * 0.1
    v = np.array([a * np.exp(-0.5 * ((t - c * t[-1]) / (n / 120)) ** 2) * np.cos(2 * np.pi * 1.5 * (t - c * t[-1]) + p)
                  for a, c, p in zip(10 ** rng.uniform(-1, 1, 3), rng.uniform(0.48, 0.52, 3), rng.uniform(0, 6.28, 3))])
    for r, x in zip(extract_phases(t, v, 2.0), v):
        f0, tc, icpt, band = reference_estimate(t, x)
        assert r["lowpass_steps"] == 0
        assert (r["band_lo"], r["band_hi"]) == band
        assert r["f0"] == pytest.approx(f0, rel=1e-10)
        if r["status"] == _abi.PHASE_OK:
            # the phase at the band's edge carries |V| of a tenth of the peak: 1e-9 leaves 10^5 of 2^-52 for it
            assert abs((r["phi"] - icpt + np.pi) % (2 * np.pi) - np.pi) <= 1e-9 * max(1.0, abs(icpt))
            assert r["t0_corr"] == pytest.approx(tc, abs=1e-9 * n)
            assert r["t0"] == t[int(np.argmax(np.abs(x)))]
        else:
            assert r["status"] == _abi.PHASE_NARROW_BAND and band[1] - band[0] < 5
    alone = extract_phases(t, v[1:2], 2.0)
    assert alone[0] == extract_phases(t, v, 2.0)[1]


def test_shortest_series(lib):
    t = np.arange(8) * 0.1
    r = extract_phases(t, np.stack([np.sin(2 * np.pi * 2.0 * t), np.zeros(8)]), 1.0)
    assert r[0]["status"] != _abi.PHASE_BAD_F0 and r[1]["status"] == _abi.PHASE_BAD_F0
