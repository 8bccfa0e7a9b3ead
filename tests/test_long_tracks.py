"""Spectra of tracks so long that they lap the transforms' circle of frequency
phases tens of thousands of times.

A perfectly periodic undulator track sampled 8 times a period, seen on
resonance on the frequencies 0.5, 1, 1.5 and 2 of the fundamental: a lap takes 16
steps and every lap adds nearly the same numbers to the same cells, so that a
plain FP32 sum rounds the same way lap after lap.  One track on few directions is
split in segments whose circles are added up; snapshots on many directions keep
whole tracks on one circle.  The reference is the FP64 kernel.

Tolerance: the FFT's FP32 rounding is that of seven stages, 7 x 6e-8 of the
amplitudes at most when they all round alike, twice that of the spectrum and
halved on average over its stages' random signs, 4e-7; the spreading kernel's
aliasing, 3e-8, and the rounding of the compensated sums are below it.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import workloads as wl  # noqa: E402

TOL = 4e-7


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("steps,n_dir,n_phi,snaps", [(1_000_000, 3, 2, 1), (400_000, 64, 114, 17)])
def test_many_laps(mode, steps, n_dir, n_phi, snaps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import _lib
    from synchrad_gb300 import batch as bt
    near, dt, g, K = mode == "near", 1.0 / 8, 200.0, 0.5
    track = wl.undulator_track(g, K, steps * dt - 2, dt, n_steps=steps, helical=near,
                               stagger=not near)
    v = np.sqrt(1 - (1 + K * K / (1 if near else 2)) / g ** 2)
    om = 2 * np.pi * np.array([0.5, 1.0, 1.5, 2.0]) * v / (1 - v)
    L = 2 * steps * dt
    pol = np.linspace(0, 1e-3 / g, n_dir)   # within the line's width
    phi = 2 * np.pi * np.arange(n_phi) / n_phi
    axes = [om, L * pol] if near else [om, np.sin(pol), np.cos(pol)]
    axes += [np.sin(phi), np.cos(phi)]
    n = (om.size, n_dir, n_phi)
    grid = bt.make_grid(mode, axes, n, torch.float64, "cuda", L_screen=L)
    batch = bt.pack_tracks([track], np.float64, snaps, dt, device="cuda")

    def run(prec):
        out = torch.zeros((snaps,) + n[::-1], dtype=torch.float64, device="cuda")
        bt.run_spectrum(batch, grid, "total", prec, [out], check_status=True)
        return out.cpu().numpy()

    got, ref = run(_lib.SR_PREC_MIXED), run(_lib.SR_PREC_DOUBLE)
    err = np.linalg.norm((got - ref).reshape(snaps, -1), axis=1) / np.linalg.norm(
        ref.reshape(snaps, -1), axis=1)
    assert err.max() <= TOL
