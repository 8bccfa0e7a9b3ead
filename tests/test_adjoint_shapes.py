"""Gradients on even frequency axes (sums over the frequencies by transforms)
at the sizes where those can go wrong.

Frequency counts around the bands and circles (8 is the least that is
transformed, 64 | 65 and 256 | 257 change the circle, 513 makes two bands),
one direction and counts that leave the last warp of the transforms part empty,
directions summed in one run and in several, steps cut by the |dphase| < pi rule
(one and many frequencies kept), snapshots, an axis that falls through zero, and
fields of more tracks than are held at a time.  The reference is autograd of the
float64 PyTorch restatement; snapshot k of a track is the spectrum of its first
snap_iterations[k] points.  The sizes are taken with 'cartesian_complex', whose
track gradients do not contain the saved amplitudes: those of short tracks come
from the forward's term-by-term kernel, and where the phases line up the gradient
of 'total' is the small quadrature part of A and magnifies their 2e-6.

Tolerance: the sums over the frequencies are FP32 sums by transforms, 4e-7 of
their norm each, the chain rule's products add a few 6e-8: relative L2 of 1e-6;
3e-6 is the bar of the adjoint's other tests.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import far_torch_ref as ftr  # noqa: E402
import near_torch_ref as ntr  # noqa: E402
from synchrad_gb300 import workloads as wl  # noqa: E402
from synchrad_gb300.batch import snap_iterations  # noqa: E402

TOL = 3e-6
L_SCREEN = 60.0


def _tracks(mode, periods, seed=5):
    rng = np.random.default_rng(seed)
    return [wl.undulator_track(g, 0.5, nper, 1 / 32, x0=rng.normal(0, 0.05),
                               y0=rng.normal(0, 0.05), xp=rng.normal(0, 0.01),
                               yp=rng.normal(0, 0.01), helical=mode == "near", stagger=False,
                               weight=float(rng.uniform(0.5, 2.0)))
            for g, nper in zip((10.0, 10.5, 9.5, 10.2), periods)]


def _axes(mode, n, lo, hi):
    f1 = 2 * 10.0 ** 2 / (1 + 0.5 ** 2)
    om = 2 * np.pi * f1 * np.linspace(lo, hi, n[0])
    phi = 2 * np.pi * np.arange(n[2]) / n[2]
    pol = np.linspace(0.0, 0.12, n[1] + 1)[1:]
    if mode == "far":
        return [om, np.sin(pol), np.cos(pol), np.sin(phi), np.cos(phi)]
    return [om, L_SCREEN * pol, np.sin(phi), np.cos(phi)]


def _gradients(mode, tracks, axes, n, g, snaps, comp):
    from synchrad_gb300 import autograd as sag
    lay = sag.make_layout([t[0].size for t in tracks], 1 / 32, axes, n, mode=mode,
                          L_screen=L_SCREEN if mode == "near" else 0.0, n_snaps=snaps,
                          form_factor=np.ones(n[0]) if mode == "far" else None)
    ts = [torch.tensor(np.concatenate([t[c] for t in tracks]), device="cuda", requires_grad=True)
          for c in range(6)]
    w = torch.tensor([t[6] for t in tracks], dtype=torch.float64, device="cuda",
                     requires_grad=True)
    fn = sag.far_spectrum if mode == "far" else sag.near_spectrum
    sum((S * torch.tensor(gk, device="cuda").reshape(S.shape)).sum()
        for S, gk in zip(fn(*ts, w, lay, comp), g)).backward()
    return [t.grad.cpu().numpy() for t in ts] + [w.grad.cpu().numpy()]


def _reference(mode, tracks, axes, g, snaps):
    ax = [torch.tensor(a, device="cuda") for a in axes]
    out = [[] for _ in range(6)]
    for t in tracks:
        c = [torch.tensor(t[k], device="cuda", requires_grad=True) for k in range(6)]
        w = torch.tensor([t[6]], dtype=torch.float64, device="cuda", requires_grad=True)
        for k, m in enumerate(snap_iterations((0, t[0].size), snaps)):
            part = [v[:int(m)] for v in c]
            args = (*part, w, [0, int(m)], 1 / 32, *ax)
            S = (ftr.far_comps_torch(*args, comp="cartesian_complex") if mode == "far" else
                 ntr.near_cartesian_complex_torch(*args, L_SCREEN))
            (S * torch.tensor(g[:, k], device="cuda")).sum().backward()
        for o, v in zip(out, c):
            o.append(v.grad.cpu().numpy())
    return [np.concatenate(o) for o in out]


def _rel(a, b):
    return float(np.linalg.norm(np.concatenate(a) - np.concatenate(b)) /
                 np.linalg.norm(np.concatenate(b)))


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n,lo,hi,periods,snaps", [
    ((8, 1, 1), 0.3, 2.6, (4, 6, 3), 1),
    ((64, 5, 3), 0.3, 2.6, (4, 6, 3), 1),
    ((65, 33, 1), 0.3, 2.6, (20,), 1),
    ((129, 6, 6), 2.6, -1.1, (4, 6, 3), 1),
    ((256, 3, 3), 0.3, 2.6, (9, 2), 1),
    ((257, 4, 1), 0.3, 9.0, (4, 6, 3), 1),
    ((513, 3, 2), 0.3, 2.6, (4, 6, 3), 1),
    ((90, 7, 4), 0.3, 30.0, (4, 6, 3), 1),
    ((600, 3, 2), 10.0, 22.0, (4, 6), 1),
    ((100, 4, 3), 0.3, 2.6, (40, 35, 30, 45), 3),
])
def test_gradient_sizes(mode, n, lo, hi, periods, snaps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    tracks, axes = _tracks(mode, periods), _axes(mode, n, lo, hi)
    g = np.random.default_rng(7).uniform(0.5, 1.5, size=(6, snaps, n[2], n[1], n[0]))
    got = _gradients(mode, tracks, axes, n, g, snaps, "cartesian_complex")
    ref = _reference(mode, tracks, axes, g, snaps)
    e = [_rel(got[:3], ref[:3]), _rel(got[3:6], ref[3:6])]
    print(mode, n, snaps, "positions %.1e momenta %.1e" % tuple(e))
    assert max(e) <= TOL


@pytest.mark.parametrize("mode,n_tracks", [("far", 150), ("near", 70)])
def test_more_tracks_than_are_held(mode, n_tracks):
    """A track's gradients do not depend on its neighbours: 2 GiB of cells are
    fewer than these tracks, so the last ones come from a second batch."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = (300, 22, 22)
    three = _tracks(mode, (2, 3, 2))
    axes = _axes(mode, n, 0.3, 2.6)
    g = np.random.default_rng(8).uniform(0.5, 1.5, size=(1, 1, n[2], n[1], n[0]))
    few = _gradients(mode, three, axes, n, g, 1, "total")
    many = _gradients(mode, [three[i % 3] for i in range(n_tracks)], axes, n, g, 1, "total")
    total = sum(t[0].size for t in three)
    last = many[0].size // total * total
    for k in range(6):
        for at in (0, last - total):
            assert _rel([many[k][at:at + total]], [few[k]]) <= TOL
    assert _rel([many[6][:3]], [few[6]]) <= TOL
