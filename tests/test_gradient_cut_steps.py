"""Gradients of tracks most of whose steps the |dphase| < pi rule cuts.

Where many of a warp's 32 steps are cut, each lane walks its own included
frequencies in blocks of 32 and reseeds every 8; where few are, the warp's lanes
share one step's.  Sizes: fewer frequencies than a reseed's run, than a block, a
block and one, two bands; intervals that start inside the axis (one that crosses
zero), at its low or at its high end; a share of cut steps from a few to all.
The references are those of test_adjoint_shapes.py.

Tolerance: as there, 1e-6 of the sums by transforms and the chain rule; a walk
adds up to 7 chained rotations of 6e-8.  3e-6 is the bar of the adjoint's tests.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_adjoint_shapes import TOL, _axes, _gradients, _reference, _rel, _tracks  # noqa: E402


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n,lo,hi,periods,snaps", [
    ((8, 5, 3), 2.0, 60.0, (20, 9), 1),
    ((31, 4, 3), -40.0, 55.0, (20, 9), 1),
    ((33, 4, 3), 45.0, -30.0, (20, 9), 1),
    ((64, 9, 2), 8.0, 26.0, (20, 9, 11), 1),
    ((64, 5, 3), 2.0, 17.0, (20, 9), 3),
    ((257, 3, 2), 1.0, 80.0, (20,), 1),
    ((600, 3, 1), 12.0, 30.0, (20,), 1),
])
def test_cut_steps(mode, n, lo, hi, periods, snaps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    tracks, axes = _tracks(mode, periods), _axes(mode, n, lo, hi)
    g = np.random.default_rng(11).uniform(0.5, 1.5, size=(6, snaps, n[2], n[1], n[0]))
    got = _gradients(mode, tracks, axes, n, g, snaps, "cartesian_complex")
    ref = _reference(mode, tracks, axes, g, snaps)
    e = [_rel(got[:3], ref[:3]), _rel(got[3:6], ref[3:6])]
    print(mode, n, snaps, "positions %.1e momenta %.1e" % tuple(e))
    assert max(e) <= TOL
