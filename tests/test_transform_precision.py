"""Precision of sums by transforms on undulator tracks, against the FP64 kernel.

A norm over the whole output hides a wrong weak direction or band edge under the
strong ones, and a bar as wide as the term-by-term kernels' hides a loss of the
transforms' precision.  So the norm is held to what the transforms promise, every
point above a thousandth of the largest to a relative bound, and the scratch size
shows that the transforms were taken.

Tolerance: an FFT of M cells rounds its sums by 0.3 x 6e-8 x sqrt(log2 M) of their
norm, 6e-8 at M = 1024, the spreading kernel's aliasing is below 3e-8, the terms'
own rounding averages out over hundreds of steps: amplitudes good to 1.2e-7 of
their norm at most, spectra to 2.4e-7.  Tracks of the same parameters leave their
errors in phase at worst.  The norm of a direction's amplitudes is spread over its
frequencies, so that a point of 1e-3 of the largest spectrum, 3e-2 of its
amplitude, is off by up to 2 x 1.2e-7 / 3e-2 x 2 = 1.6e-5 of itself.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import _lib  # noqa: E402
from synchrad_gb300 import workloads as wl  # noqa: E402

TOL, TOL_POINT = 2.4e-7, 1.6e-5


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n,n_tracks,steps,periods,split", [
    ((64, 12, 3), 2, 2000, 20, True), ((129, 33, 2), 5, 1500, 15, True),
    ((512, 9, 4), 3, 2400, 24, True), ((700, 5, 5), 2, 2000, 20, True),
    ((64, 48, 40), 80, 700, 7, False), ((300, 40, 30), 60, 900, 9, False)])
def test_precision(mode, n, n_tracks, steps, periods, split):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import host as ohost
    from synchrad_gb300 import batch as bt
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=n_tracks, n_steps=steps, grid=n, n_periods=periods)
    a = ohost.init_args(dict(w.args, dtype="double"))
    grid = bt.make_grid(mode, ohost.device_axes(a), n, torch.float64, "cuda",
                        L_screen=w.L_screen or 0.0)
    batch = bt.pack_tracks(w.tracks, np.float64, 1, w.time_step, device="cuda")
    L = _lib.lib()
    L.sr_config_clear()
    ts, gs = batch.c_struct(), grid.c_struct()
    args = (ctypes.byref(ts), ctypes.byref(gs), 0, _lib.SR_PREC_MIXED)
    assert L.sr_workspace_bytes(*args) > L.sr_workspace_bytes_min(*args)
    # split in segments where there are few (track, 32 directions) units
    units = n_tracks * -(-n[1] * n[2] // 32) * -(-n[0] // 512)
    assert split == (units <= 1216)

    def run(prec):
        out = torch.zeros((1,) + n[::-1], dtype=torch.float64, device="cuda")
        bt.run_spectrum(batch, grid, "total", prec, [out], check_status=True)
        return out.cpu().numpy()

    got, ref = run(_lib.SR_PREC_MIXED), run(_lib.SR_PREC_DOUBLE)
    err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    strong = ref > 1e-3 * ref.max()
    worst = np.max(np.abs(got - ref)[strong] / ref[strong])
    print(mode, n, "norm %.1e point %.1e" % (err, worst))
    assert err <= TOL and worst <= TOL_POINT
