"""The spectral sum by transforms over the steps, against term-by-term sums.

On an evenly spaced frequency axis the mixed-precision path spreads the steps
onto a circle of cells and transforms; a pinned work shape sums term by term.
Both are compared with the FP64 kernel at the places where the transforms can
go wrong: band and circle sizes (129 | 128, 257 | 256, 513 | 512 frequencies,
odd counts), directions that do not fill a warp or span many phi nodes, whole
tracks and tracks split in segments, steps cut by the |dphase| < pi rule (lists
and their overflow), axes that fall, cross zero or are not even, snapshots, and
tracks that run backwards in the retarded time.

Tolerance: the terms are FP32 products with a relative error of a few 6e-8 that
is independent from step to step, the spreading kernel's aliasing is below
3e-8 and an FFT of at most 1024 cells rounds by about 5 x 6e-8, so amplitudes
are good to ~4e-7 of their norm and spectra to ~8e-7; the term-by-term sums
round by up to 32 chained rotations (~2e-6).  3e-6 covers either.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import workloads as wl  # noqa: E402

TOL = 3e-6


def _spectra(w, comp="total", snaps=1, axis=None, f32=False, tracks=None):
    """(transform path, term by term, FP64) outputs of one workload."""
    from oracle import host as ohost
    from synchrad_gb300 import _lib
    from synchrad_gb300 import batch as bt
    mode = w.args.get("mode", "far")
    a = ohost.init_args(dict(w.args, dtype="double"))
    n = tuple(int(v) for v in a["gridNodeNums"])
    axes = list(ohost.device_axes(a))
    if axis is not None:
        axes[0] = axis(axes[0])
    tracks = w.tracks if tracks is None else tracks
    grid = bt.make_grid(mode, axes, n, torch.float64, "cuda", L_screen=w.L_screen or 0.0,
                        form_factor=np.ones(n[0]))
    batch = bt.pack_tracks(tracks, np.float32 if f32 else np.float64, snaps, w.time_step,
                           device="cuda")
    ref = bt.pack_tracks([[np.asarray(c, dtype=np.float64) for c in t[:6]] + list(t[6:])
                          for t in tracks], np.float64, snaps, w.time_step, device="cuda")
    n_out = _lib.N_OUT[_lib.COMP_IDS[comp]]

    def run(b, prec):
        out = [torch.zeros((snaps, n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
               for _ in range(n_out)]
        bt.run_spectrum(b, grid, comp, prec, out, check_status=True)
        return np.stack([o.cpu().numpy() for o in out])

    _lib.lib().sr_config_clear()
    shape = bt.current_config(batch, grid, comp)
    fast = run(batch, _lib.SR_PREC_MIXED)
    again = run(batch, _lib.SR_PREC_MIXED)
    assert np.array_equal(fast, again)
    bt.set_config(batch, grid, comp, points_per_lane=shape["points_per_lane"],
                  lanes_per_direction=shape["lanes_per_direction"])
    direct = run(batch, _lib.SR_PREC_MIXED)
    _lib.lib().sr_config_clear()
    return fast, direct, run(ref, _lib.SR_PREC_DOUBLE)


def _check(fast, direct, ref):
    norm = np.linalg.norm(ref)
    assert norm > 0
    for got in (fast, direct):
        assert np.linalg.norm(got - ref) / norm <= TOL


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n_omega,n_dir,n_phi,n_tracks", [
    (4, 3, 2, 70), (64, 1, 1, 2), (65, 33, 1, 2), (128, 2, 40, 3), (129, 5, 7, 80),
    (256, 32, 1, 2), (257, 7, 5, 3), (511, 4, 3, 66), (512, 3, 11, 2), (513, 4, 2, 3),
    (1030, 3, 3, 2)])
def test_sizes(mode, n_omega, n_dir, n_phi, n_tracks):
    """Bands, circles and warps at their edges; few tracks (segments) and many."""
    _need_gpu()
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=n_tracks, n_steps=700, grid=(n_omega, n_dir, n_phi), n_periods=10)
    _check(*_spectra(w))


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n_omega,n_tracks", [(70, 2), (70, 64), (300, 3), (700, 66)])
def test_cut_steps(mode, n_omega, n_tracks):
    """An axis from 0 on coarse tracks: the |dphase| < pi rule cuts most steps
    inside the axis, so lists fill and are emptied many times."""
    _need_gpu()
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=n_tracks, n_steps=520, grid=(n_omega, 6, 5), n_periods=70)
    g = list(w.args["grid"])
    g[0] = (0.0, g[0][1])
    w.args["grid"] = g
    _check(*_spectra(w))


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("axis", ["falling", "crossing", "uneven"])
def test_axes(mode, axis):
    """A falling axis, one that crosses zero (the included frequencies of a cut
    step are an interval inside the axis) and one that is not even."""
    _need_gpu()
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=3, n_steps=600, grid=(90, 5, 4), n_periods=40)
    f = {"falling": lambda o: np.ascontiguousarray(o[::-1]),
         "crossing": lambda o: np.linspace(-0.6 * o[-1], o[-1], o.size),
         "uneven": lambda o: np.geomspace(o[0], o[-1], o.size)}[axis]
    _check(*_spectra(w, axis=f))


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n_omega,periods", [(2, 10), (33, 10), (95, 40), (97, 10), (160, 70),
                                             (192, 10), (224, 10), (257, 40), (600, 10)])
def test_uneven_axis_sizes(mode, n_omega, periods):
    """Axes that are not even, at the frequency counts where a lane takes one
    more frequency or a warp one more tile; coarse tracks (many periods) are cut
    by the |dphase| < pi rule.  One term is a hardware sine and cosine (2e-7
    rad) of a phase good to 1e-7: 4e-7 of the amplitude's norm at most."""
    _need_gpu()
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=3, n_steps=300, grid=(n_omega, 3, 3), n_periods=periods)
    _check(*_spectra(w, snaps=2, axis=lambda o: np.sort(o[0] + (o[-1] - o[0]) * np.linspace(
        0, 1, o.size) ** 1.5)))


@pytest.mark.parametrize("mode,comp", [("far", "cartesian"), ("far", "cartesian_complex"),
                                       ("far", "spheric"), ("far", "spheric_complex"),
                                       ("near", "cartesian"), ("near", "cartesian_complex")])
@pytest.mark.parametrize("snaps", [1, 4])
def test_comps_and_snapshots(mode, comp, snaps):
    _need_gpu()
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=3, n_steps=900, grid=(140, 6, 7), n_periods=15)
    fast, direct, ref = _spectra(w, comp, snaps)
    if mode == "near" and comp.endswith("complex"):
        # exp(i omega L) of the FP64 kernel's own phase t + r carries
        # ~eps x omega L ~ 3e-8 rad
        pass
    _check(fast, direct, ref)


@pytest.mark.parametrize("mode", ["far", "near"])
def test_backwards_and_ragged(mode):
    """Tracks of uneven length, single steps among them, and tracks whose
    retarded time falls (positions in reverse) or jumps."""
    _need_gpu()
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=6, n_steps=800, grid=(150, 6, 6), n_periods=12)
    lengths = (800, 1, 2, 37, 513, 800)
    tracks = []
    for i, (t, m) in enumerate(zip(w.tracks, lengths)):
        c = [np.asarray(a)[:m].copy() for a in t[:6]]
        if i == 0:  # z overtakes the light by a little: tau falls step by step
            c[2] = c[2] + 1.6e-7 * np.arange(m)
        if i == 5:  # a gap in the retarded time
            c[2][400:] -= 0.37
        tracks.append(c + list(t[6:]))
    _check(*_spectra(w, tracks=tracks))


def test_fp32_betatron():
    _need_gpu()
    w = wl.c3_betatron_ragged(n_tracks=5, grid=(256, 7, 6), steps_range=(400, 5000))
    _check(*_spectra(w, f32=True))
