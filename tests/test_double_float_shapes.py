"""Double-float far-field spectra on even axes (the sum over the steps by
transforms) at the sizes where those can go wrong.

Frequency counts around the bands and circles (16 is the least that is
transformed, 64 | 65 and 256 | 257 change the circle, above 512 there are
several bands, whose edges must not fall inside a lane's 8 frequencies),
direction counts that do not fill a warp, segments and tracks of any length,
steps cut by the |dphase| < pi rule (few, and so many that all is left to the
term-by-term kernel), axes that fall through zero or are not even, the comps,
shared memory asked for in changing amounts, and more tracks than are held at a
time.  The reference is the FP64 kernel.

Tolerance: the FP64 kernel rounds t - n.x, of some 20 units, to 2 ulp, times
omega of up to 2 pi 160 x 2.6 rad a unit: 20 x 2600 x 4.4e-16 = 2e-11 of phase,
4e-11 of the spectrum; this path rounds less.  1e-10, the bar of the golden
vectors, covers it.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import workloads as wl  # noqa: E402

TOL = 1e-10
N_OUT = {"total": 1, "cartesian": 3, "cartesian_complex": 6, "spheric_complex": 6}


def _tracks(periods, seed=5):
    rng = np.random.default_rng(seed)
    return [wl.undulator_track(g, 0.5, nper, 1 / 32, x0=rng.normal(0, 0.05),
                               y0=rng.normal(0, 0.05), xp=rng.normal(0, 0.01),
                               yp=rng.normal(0, 0.01), weight=float(rng.uniform(0.5, 2.0)))
            for g, nper in zip((10.0, 10.5, 9.5, 10.2), periods)]


def _run(tracks, n, lo, hi, prec, comp="total", even=True):
    from synchrad_gb300 import batch as bt
    om = np.linspace(lo, hi, n[0]) if even else np.geomspace(lo, hi, n[0])
    theta, phi = np.linspace(0.0, 0.12, n[1] + 1)[1:], 2 * np.pi * np.arange(n[2]) / n[2]
    f1 = 2 * 10.0 ** 2 / (1 + 0.5 ** 2 / 2)
    axes = [2 * np.pi * f1 * om, np.sin(theta), np.cos(theta), np.sin(phi), np.cos(phi)]
    grid = bt.make_grid("far", axes, n, torch.float64, "cuda", form_factor=np.ones(n[0]))
    out = [torch.zeros((1,) + n[::-1], dtype=torch.float64, device="cuda")
           for _ in range(N_OUT[comp])]
    bt.run_spectrum(bt.pack_tracks(tracks, np.float64, 1, 1 / 32, device="cuda"), grid, comp,
                    prec, out, check_status=True)
    return torch.stack(out).cpu().numpy()


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n,lo,hi,periods,comp,even", [
    ((16, 1, 1), 0.3, 2.6, (9,), "total", True),
    ((64, 5, 3), 0.3, 2.6, (9, 16, 12), "cartesian", True),
    ((65, 33, 1), 0.3, 2.6, (14, 8), "total", True),
    ((129, 6, 6), 2.6, -1.1, (9, 16, 12), "total", True),
    ((256, 3, 3), 0.3, 2.6, (30,), "cartesian_complex", True),
    ((257, 4, 1), 0.3, 2.6, (9, 16, 12), "spheric_complex", True),
    ((513, 3, 2), 0.3, 2.6, (9, 16), "total", True),
    ((1100, 2, 2), 0.3, 2.6, (9, 11), "total", True),
    ((90, 7, 4), 0.3, 12.0, (9, 16, 12), "total", True),
    ((90, 7, 4), 0.3, 40.0, (9, 16, 12), "total", True),
    ((90, 7, 4), 0.3, 2.6, (9, 16, 12), "total", False),
    ((64, 3, 2), 0.3, 2.6, (9, 16, 12), "total", True),
])
def test_double_float_sizes(n, lo, hi, periods, comp, even):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import _lib
    tracks = _tracks(periods)
    got = _run(tracks, n, lo, hi, _lib.SR_PREC_DF, comp, even)
    ref = _run(tracks, n, lo, hi, _lib.SR_PREC_DOUBLE, comp, even)
    print(n, comp, "%.1e" % _rel(got, ref))
    assert _rel(got, ref) <= TOL


def test_more_tracks_than_are_held():
    """4 GiB of circles are fewer than 300 of these tracks; three tracks over
    and over add up to a hundred times the three."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import _lib
    three, n = _tracks((9, 8, 10)), (300, 24, 24)
    few = _run(three, n, 0.3, 2.6, _lib.SR_PREC_DF)
    many = _run([three[i % 3] for i in range(300)], n, 0.3, 2.6, _lib.SR_PREC_DF)
    assert _rel(many, 100.0 * few) <= TOL
