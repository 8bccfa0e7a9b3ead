"""Spectra of tracks whose steps the |dphase| < pi rule cuts inside the axis, where
their direct sums are left to a kernel with a warp per direction and segment.

Sizes: lists of a few entries and of whole segments, directions that do not fill a
warp and more polar angles than lanes (the cut ones crowd in a few warps), one and
two passes over the frequencies, two bands, units between snapshots, complex comps,
the saved forward's amplitudes, and a track with many segments.

Tolerance: a listed term is a hardware sine and cosine (4e-7 rad) rotated up to
seven times (7 x 6e-8), independent from step to step; amplitudes of hundreds of
steps are good to 4e-7 of their norm and spectra to 8e-7, complex outputs to half
of that.  1.2e-6.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import workloads as wl  # noqa: E402

TOL = 1.2e-6


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n,n_tracks,steps,per,lo,comp,snaps", [
    ((40, 6, 5), 2, 900, 6, 0.0, "total", 1),
    ((256, 70, 2), 3, 600, 10, 0.5, "total", 1),
    ((300, 33, 3), 3, 700, 8, 0.5, "cartesian", 1),
    ((512, 5, 3), 2, 1100, 5, 0.2, "cartesian_complex", 1),
    ((700, 4, 3), 2, 1100, 6, 0.0, "total", 1),
    ((129, 9, 4), 3, 1500, 8, 0.3, "total", 3),
    ((64, 40, 2), 1, 6000, 7, 0.5, "total", 1),
])
def test_cut_steps(mode, n, n_tracks, steps, per, lo, comp, snaps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from test_transform_sum import _spectra
    from synchrad_gb300 import _lib
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=n_tracks, n_steps=steps, grid=n, n_periods=steps // per)
    g = list(w.args["grid"])
    g[0] = (lo / 0.5 * g[0][0], g[0][1])
    w.args["grid"] = g
    t, gr = _lib.SrTracks(), _lib.SrGrid()
    t.n_tracks, t.total_steps, t.n_snaps = n_tracks, n_tracks * steps, snaps
    gr.mode = _lib.SR_MODE_FAR if mode == "far" else _lib.SR_MODE_NEAR
    gr.n_omega, gr.n_theta, gr.n_phi = n
    args = (ctypes.byref(t), ctypes.byref(gr), _lib.COMP_IDS[comp], _lib.SR_PREC_MIXED)
    L = _lib.lib()
    L.sr_config_clear()
    if mode == "far" or (n[0] <= 256 or steps >= 800):
        assert L.sr_workspace_bytes(*args) > L.sr_workspace_bytes_min(*args)  # by transforms
    fast, _, ref = _spectra(w, comp, snaps)
    for i in range(snaps):
        err = np.linalg.norm(fast[:, i] - ref[:, i]) / np.linalg.norm(ref[:, i])
        print(mode, n, steps, comp, i, "%.1e" % err)
        assert err <= TOL
