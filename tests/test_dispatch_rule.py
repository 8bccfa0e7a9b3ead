"""From how many steps on a batch is summed by transforms.

Short tracks stay with the term-by-term kernel: the transforms' circles cost the
same whatever a track's steps.  Which path a call takes shows in its scratch (the
transforms need more than sr_workspace_bytes_min), so the rule's lines are checked
on the host; on the GPU batches of many tracks of a few steps agree with the FP64
kernel on either side of a line.

Tolerance: terms rounded to FP32 independently, at most 8 of 6e-8 each, spectra
twice the amplitudes' error, 1e-6, and the hardware sine's 4e-7 where the sum is
taken term by term with few terms to average over: 1.5e-6.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from synchrad_gb300 import _lib  # noqa: E402

TOL = 1.5e-6


def _by_transforms(mode, n_omega, n_dirs, tracks, steps, snaps=1):
    t, g = _lib.SrTracks(), _lib.SrGrid()
    t.n_tracks, t.total_steps, t.n_snaps = tracks, tracks * steps, snaps
    g.mode = _lib.SR_MODE_FAR if mode == "far" else _lib.SR_MODE_NEAR
    g.n_omega, g.n_theta, g.n_phi = n_omega, n_dirs, 1
    L = _lib.lib()
    args = (ctypes.byref(t), ctypes.byref(g), 0, _lib.SR_PREC_MIXED)
    return L.sr_workspace_bytes(*args) > L.sr_workspace_bytes_min(*args)


@pytest.mark.parametrize("mode,n_omega,n_dirs,tracks,least", [
    ("far", 64, 1024, 64, 64), ("far", 512, 1024, 400, 64), ("far", 512, 512, 64, 128),
    ("far", 64, 8, 64, 320), ("far", 512, 8, 64, 800), ("far", 100, 8, 500, 24),
    ("far", 512, 8, 8, 640), ("far", 200, 8, 8, 200), ("far", 64, 64, 2, 320),
    ("near", 64, 1024, 64, 32), ("near", 16, 64, 64, 1280), ("near", 100, 64, 64, 400),
    ("near", 300, 64, 64, 200), ("near", 300, 8, 64, 2048), ("near", 100, 64, 8, 512)])
def test_lines(mode, n_omega, n_dirs, tracks, least):
    """The least mean steps at these sizes, each measured from both sides."""
    _lib.lib().sr_config_clear()
    assert not _by_transforms(mode, n_omega, n_dirs, tracks, least - 1)
    assert _by_transforms(mode, n_omega, n_dirs, tracks, least)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n_omega,n_dir,n_phi,n_tracks,steps", [
    (64, 3, 2, 64, 2), (300, 5, 3, 80, 12), (512, 3, 3, 70, 50), (40, 33, 30, 70, 40),
    (300, 33, 30, 70, 70), (100, 2, 4, 500, 45)])
def test_short_tracks(mode, n_omega, n_dir, n_phi, n_tracks, steps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from test_transform_sum import _spectra
    from synchrad_gb300 import workloads as wl
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=n_tracks, n_steps=steps, grid=(n_omega, n_dir, n_phi), n_periods=1)
    fast, direct, ref = _spectra(w)
    for got in (fast, direct):
        assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)
