"""What the autotuner tunes, by the path the problem takes.

Where an even axis is summed by transforms there is no shape to tune: they stay
unless the term-by-term kernel is faster, the tuned call gives the untuned bits,
and a config read back and pinned in another process takes the same path.  On an
uneven axis the points and lanes stay the default's.  Short tracks go term by
term, and their shapes are searched.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import _lib  # noqa: E402
from synchrad_gb300 import workloads as wl  # noqa: E402


def _setup(mode, axis=None, **kw):
    from oracle import host as ohost
    from synchrad_gb300 import batch as bt
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(**kw)
    a = ohost.init_args(dict(w.args, dtype="double"))
    n = tuple(int(v) for v in a["gridNodeNums"])
    axes = list(ohost.device_axes(a))
    if axis is not None:
        axes[0] = axis(axes[0])
    grid = bt.make_grid(mode, axes, n, torch.float64, "cuda", L_screen=w.L_screen or 0.0)
    return bt.pack_tracks(w.tracks, np.float64, 1, w.time_step, device="cuda"), grid, n


def _run(batch, grid, n):
    from synchrad_gb300 import batch as bt
    out = torch.zeros((1,) + n[::-1], dtype=torch.float64, device="cuda")
    ws = bt.Workspace("cuda")
    bt.run_spectrum(batch, grid, "total", _lib.SR_PREC_MIXED, [out], workspace=ws)
    return out.cpu().numpy(), ws.buf.numel()


SHAPE = ("points_per_lane", "lanes_per_direction", "steps_per_stage", "track_subsets")


@pytest.mark.parametrize("mode", ["far", "near"])
def test_transforms_stay(mode):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import batch as bt
    batch, grid, n = _setup(mode, n_tracks=24, n_steps=2000, grid=(200, 24, 24))
    _lib.lib().sr_config_clear()
    default = bt.current_config(batch, grid)
    assert default["transforms"] == 1
    plain, size = _run(batch, grid, n)
    res = bt.autotune(batch, grid, budget_ms=500.0)
    assert res["best"]["transforms"] == 1 and 0 < res["best"]["ms"] == res["default"]["ms"]
    tuned = bt.current_config(batch, grid)
    assert all(tuned[k] == default[k] for k in SHAPE + ("transforms",))
    again, size1 = _run(batch, grid, n)
    assert np.array_equal(plain, again) and size == size1
    _lib.lib().sr_config_clear()
    bt.set_config(batch, grid, transforms=bool(tuned["transforms"]), **{k: tuned[k] for k in SHAPE})
    pinned, size2 = _run(batch, grid, n)
    assert np.array_equal(plain, pinned) and size == size2
    bt.set_config(batch, grid, **{k: tuned[k] for k in SHAPE})  # without: term by term
    terms, size3 = _run(batch, grid, n)
    _lib.lib().sr_config_clear()
    assert size3 < size and not np.array_equal(plain, terms)


@pytest.mark.parametrize("mode", ["far", "near"])
def test_uneven_axis(mode):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import batch as bt
    batch, grid, n = _setup(mode, axis=lambda o: np.geomspace(o[0], o[-1], o.size), n_tracks=24,
                            n_steps=600, grid=(96, 12, 10))
    _lib.lib().sr_config_clear()
    default = bt.current_config(batch, grid)
    best = bt.autotune(batch, grid, budget_ms=300.0)["best"]
    assert best["ms"] > 0
    assert all(best[k] == default[k] for k in SHAPE[:3])
    _lib.lib().sr_config_clear()


@pytest.mark.parametrize("mode", ["far", "near"])
def test_short_tracks_are_tuned(mode):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import batch as bt
    batch, grid, n = _setup(mode, n_tracks=12, n_steps=100, grid=(96, 6, 5), n_periods=2)
    _lib.lib().sr_config_clear()
    plain, size = _run(batch, grid, n)
    best = bt.autotune(batch, grid, budget_ms=300.0)["best"]
    assert best["transforms"] == 0 and best["ms"] > 0
    tuned, _ = _run(batch, grid, n)
    _lib.lib().sr_config_clear()
    assert np.linalg.norm(tuned - plain) <= 3e-6 * np.linalg.norm(plain)
