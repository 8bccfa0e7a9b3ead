"""How much scratch the sums by transforms take, and calls that get less.

The circles of the transforms take gigabytes at the largest grids.  Every entry
point also runs with the scratch of its term-by-term kernel, which is what an
uneven axis asks for and what a caller falls back to when the memory is not
there.

Bound: at most 4 GiB of circles or twice the resident warps' slices, 2 x 152 x 8
near-field slices of 3.8 MB = 8.7 GiB (the larger), and 1 GiB of partial spectra.
"""
import ctypes
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from synchrad_gb300 import _lib  # noqa: E402
from synchrad_gb300 import workloads as wl  # noqa: E402
from synchrad_gb300.batch import Workspace, even_axis  # noqa: E402

BOUND = 9.7 * 2 ** 30


@pytest.mark.parametrize("mode", [_lib.SR_MODE_FAR, _lib.SR_MODE_NEAR])
def test_bounds(mode):
    """Reads sizes on the host only."""
    L = _lib.lib()
    largest = 0
    for n_omega, n_dir, tracks, steps, snaps in itertools.product(
            (100, 512, 1500), (33, 4096), (1, 30, 5000), (3000, 100000), (1, 5)):
        t, g = _lib.SrTracks(), _lib.SrGrid()
        t.n_tracks, t.total_steps, t.n_snaps = tracks, tracks * steps, snaps
        g.mode, g.n_omega, g.n_theta, g.n_phi = mode, n_omega, n_dir, 1
        tp, gp = ctypes.byref(t), ctypes.byref(g)
        for prec in ([_lib.SR_PREC_MIXED] + ([_lib.SR_PREC_DF] if mode == _lib.SR_MODE_FAR else [])):
            full, least = (f(tp, gp, 0, prec) for f in (L.sr_workspace_bytes,
                                                        L.sr_workspace_bytes_min))
            # double-float: also a word of cut steps per 32 steps and directions
            words = (t.total_steps // 32 + tracks) * (-(-n_dir // 32) * -(-n_omega // 512))
            assert 0 < least <= full <= least + BOUND + (4 * words if prec == _lib.SR_PREC_DF else 0)
            largest = max(largest, full - least)
        name = "far" if mode == _lib.SR_MODE_FAR else "near"
        full, least = (getattr(L, f"sr_{name}_backward_workspace_bytes{s}")(tp, gp)
                       for s in ("", "_min"))
        # 2 GiB of cells, the tables and up to 15 more sets of 9 gradients per step
        assert 0 < least <= full <= least + 2 ** 31 + 2 ** 20 + 15 * 72 * t.total_steps
    assert largest > 2 ** 30  # the sweep reaches the sizes that the bound is about


def test_falls_back_when_the_memory_is_not_there(monkeypatch):
    ws = Workspace("cpu")
    taken, empty = [], torch.empty

    def short_of_memory(n, **kw):
        taken.append(n)
        if n > 1000:
            raise torch.OutOfMemoryError("no memory")
        return empty(n, **kw)

    monkeypatch.setattr(torch, "empty", short_of_memory)
    buf, size = ws.get_for(lambda: 5000, lambda: 600)
    assert size == 600 and buf.numel() == 600 and taken == [5000, 600]
    with pytest.raises(torch.OutOfMemoryError):
        ws.get_for(lambda: 5000, lambda: 5000)
    assert ws.get_for(lambda: 5000, lambda: 500, even=False)[1] == 500
    with pytest.raises(_lib.SynchRadError):
        ws.get_for(lambda: -1, lambda: -1)


def test_even_axis():
    o = np.linspace(2e3, 2e5, 301)
    assert even_axis(o) and even_axis(o[::-1]) and even_axis(-o) and even_axis(o[:1])
    assert not even_axis(np.geomspace(1.0, 2.0, 9))
    assert not even_axis(np.where(np.arange(301) == 7, o * (1 + 1e-11), o))
    assert not even_axis(np.full(4, 3.0)) and not even_axis(np.array([1.0, np.nan, 3.0]))


def _problem(mode, axis=None):
    from oracle import host as ohost
    from synchrad_gb300 import batch as bt
    make = wl.c2_far_mixed if mode == "far" else wl.c5_near_helical
    w = make(n_tracks=4, n_steps=900, grid=(96, 6, 5), n_periods=14)
    a = ohost.init_args(dict(w.args, dtype="double"))
    n = tuple(int(v) for v in a["gridNodeNums"])
    axes = list(ohost.device_axes(a))
    if axis is not None:
        axes[0] = axis(axes[0])
    grid = bt.make_grid(mode, axes, n, torch.float64, "cuda", L_screen=w.L_screen or 0.0)
    return bt.pack_tracks(w.tracks, np.float64, 1, w.time_step, device="cuda"), grid, n, axes, w


def _raw(batch, grid, n, prec, size):
    """sr_spectrum with `size` bytes of scratch."""
    L = _lib.lib()
    out = torch.zeros((1,) + n[::-1], dtype=torch.float64, device="cuda")
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    ts, gs = batch.c_struct(), grid.c_struct()
    outs = (ctypes.c_void_p * 6)(out.data_ptr())
    rc = L.sr_spectrum(ctypes.byref(ts), ctypes.byref(gs), 0, prec, outs, ws.data_ptr(),
                       ctypes.c_size_t(size),
                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return rc, out.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("mode,prec", [("far", "mixed"), ("near", "mixed"), ("far", "df")])
def test_least_scratch(mode, prec):
    """With the least scratch the sum is the term-by-term one (to the bit, where
    a shape can be pinned), with a byte less the call is refused, and nothing is
    written behind the least."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import batch as bt
    batch, grid, n, _, _ = _problem(mode)
    L = _lib.lib()
    L.sr_config_clear()
    pid = _lib.SR_PREC_MIXED if prec == "mixed" else _lib.SR_PREC_DF
    ts, gs = batch.c_struct(), grid.c_struct()
    args = (ctypes.byref(ts), ctypes.byref(gs), 0, pid)
    full, least = L.sr_workspace_bytes(*args), L.sr_workspace_bytes_min(*args)
    assert least < full
    rc, fast = _raw(batch, grid, n, pid, full)
    assert rc == _lib.SR_OK
    rc, short = _raw(batch, grid, n, pid, full - 1)
    assert rc == _lib.SR_OK
    rc, direct = _raw(batch, grid, n, pid, least)
    assert rc == _lib.SR_OK and np.array_equal(direct, short)
    assert 0 < np.linalg.norm(fast - direct) <= 3e-6 * np.linalg.norm(fast)
    rc, none = _raw(batch, grid, n, pid, least - 1)
    assert rc == -4 and not none.any() and b"workspace" in L.sr_last_error()
    if prec == "mixed":
        shape = bt.current_config(batch, grid)
        bt.set_config(batch, grid, points_per_lane=shape["points_per_lane"],
                      lanes_per_direction=shape["lanes_per_direction"],
                      steps_per_stage=shape["steps_per_stage"],
                      track_subsets=shape["track_subsets"])
        assert L.sr_workspace_bytes(*args) == least
        assert np.array_equal(_raw(batch, grid, n, pid, least)[1], direct)
        L.sr_config_clear()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["far", "near"])
def test_gradient_with_least_scratch(mode, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import autograd as sag
    _, grid, n, axes, w = _problem(mode)

    def gradients(least):
        lay = sag.make_layout([900] * 4, w.time_step, axes, n, mode=mode,
                              L_screen=w.L_screen or 0.0)
        if least:
            get = lay.workspace.get_for
            lay.workspace.get_for = lambda need, need_min, even=True: get(need_min, need_min)
        ts = [torch.tensor(np.concatenate([t[k] for t in w.tracks]), device="cuda",
                           requires_grad=True) for k in range(6)]
        wt = torch.ones(4, dtype=torch.float64, device="cuda", requires_grad=True)
        sag.total_spectrum_fn(mode)(*ts, wt, lay).sum().backward()
        return [t.grad.cpu().numpy() for t in ts + [wt]], lay.workspace.buf.numel()

    (a, big), (b, small) = gradients(False), gradients(True)
    assert small < big
    for part in (slice(0, 3), slice(3, 6), slice(6, 7)):
        x, y = np.stack(a[part]), np.stack(b[part])
        # the adjoint's bar, 3e-6, on either side
        assert 0 < np.linalg.norm(x - y) <= 6e-6 * np.linalg.norm(y)


def _uneven(o):
    return np.geomspace(o[0], o[-1], o.size)


@pytest.mark.gpu
@pytest.mark.parametrize("mode,prec", [("far", "mixed"), ("near", "mixed"), ("far", "df")])
def test_uneven_axis_takes_the_least(mode, prec):
    """... and given everything (a caller that does not know its axis) the kernels
    find it uneven and sum the same way, to the bit."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import batch as bt
    batch, grid, n, _, _ = _problem(mode, axis=_uneven)
    pid = _lib.SR_PREC_MIXED if prec == "mixed" else _lib.SR_PREC_DF
    L = _lib.lib()
    ts, gs = batch.c_struct(), grid.c_struct()
    args = (ctypes.byref(ts), ctypes.byref(gs), 0, pid)
    ws = Workspace("cuda")
    out = torch.zeros((1,) + n[::-1], dtype=torch.float64, device="cuda")
    bt.run_spectrum(batch, grid, "total", pid, [out], workspace=ws)
    assert ws.buf.numel() == L.sr_workspace_bytes_min(*args) < L.sr_workspace_bytes(*args)
    assert np.array_equal(out.cpu().numpy(),
                          _raw(batch, grid, n, pid, L.sr_workspace_bytes(*args))[1])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["far", "near"])
def test_gradient_on_an_uneven_axis(mode):
    """As above, for the saved forward and the backward."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from synchrad_gb300 import autograd as sag
    _, _, n, axes, w = _problem(mode, axis=_uneven)

    def gradients(known):
        lay = sag.make_layout([900] * 4, w.time_step, axes, n, mode=mode,
                              L_screen=w.L_screen or 0.0)
        assert not lay.grid.even
        lay.grid.even = not known
        ts = [torch.tensor(np.concatenate([t[k] for t in w.tracks]), device="cuda",
                           requires_grad=True) for k in range(6)]
        wt = torch.ones(4, dtype=torch.float64, device="cuda", requires_grad=True)
        sag.total_spectrum_fn(mode)(*ts, wt, lay).sum().backward()
        return [t.grad.cpu().numpy() for t in ts + [wt]], lay.workspace.buf.numel()

    (a, small), (b, big) = gradients(True), gradients(False)
    assert small < big
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
