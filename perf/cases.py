"""The workloads whose speed this repository answers for.

A case is one call of a user's program: a batch of electron tracks, a spectral
grid and an option set, evaluated through ``SynchRad.calculate_spectrum`` (host
tracks in, host spectra out) or through the differentiable spectra of
``synchrad_gb300.autograd`` (device tensors in, spectrum and gradients out).

``listed`` gives the named cases, ``draw`` more of the same ranges.  ``exact``
restates the radiation integrals in plain torch at 64 bits.
"""
import contextlib
import io
import math

import numpy as np
import torch

from synchrad_gb300 import autograd as sag
from synchrad_gb300 import workloads as wl
from synchrad_gb300.calc import SynchRad

VEC = {"total": ("total",), "cartesian": ("x", "y", "z"),
       "cartesian_complex": ("xre", "xim", "yre", "yim", "zre", "zim")}


def _case(name, **kw):
    c = dict(kind="spectrum", mode="far", dtype="mixed", comp="total", motion="undulator",
             tracks=1, steps_lo=1000, steps_hi=1000, periods=20, gamma=200.0, K=0.5,
             track_f32=False, n_omega=64, n_dir=16, n_phi=16, w_lo=0.5, w_hi=1.5,
             dir_max=1.5, axis="uniform", snaps=1)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: the analytic-undulator check's few short tracks on a coarse grid
        _case("small_call", tracks=3, steps_lo=193, steps_hi=193, periods=6, gamma=100.0, K=0.1,
              n_omega=64, n_dir=8, n_phi=6, w_lo=0.5, w_hi=1.5, dir_max=2.0),
        # the reference's default precision on one electron: the single-undulator configuration
        _case("one_electron_double", dtype="double", tracks=1, steps_lo=1408, steps_hi=1408,
              periods=20, gamma=100.0, K=0.1, n_omega=256, n_dir=32, n_phi=32, dir_max=1.0),
        # a sample of the undulator bunch over the first three harmonics, the headline grid
        _case("bunch_mixed", tracks=32, steps_lo=4000, steps_hi=4000, periods=60, gamma=400.0,
              K=1.0, n_omega=512, n_dir=64, n_phi=64, w_lo=0.5, w_hi=3.5, dir_max=2.0),
        # uneven FP32 betatron tracks from a particle-in-cell run; the sampling limit
        # |dphase| < pi cuts through the frequency axis
        _case("ragged_betatron", motion="betatron", tracks=16, steps_lo=500, steps_hi=20000,
              track_f32=True, n_omega=256, n_dir=48, n_phi=48),
        # helical electrons on a near-field screen at 20 undulator lengths
        _case("screen_mixed", mode="near", motion="helical", tracks=16, steps_lo=8000,
              steps_hi=8000, periods=50, gamma=300.0, n_omega=256, n_dir=64, n_phi=64),
        # coherent time-resolved amplitudes on odd sizes
        _case("coherent_snapshots", comp="cartesian_complex", tracks=23, steps_lo=700,
              steps_hi=2301, periods=25, gamma=300.0, K=0.8, n_omega=301, n_dir=21, n_phi=33,
              w_lo=0.6, w_hi=1.4, snaps=5),
        # a logarithmic frequency axis (broadband radiation), polarisation resolved
        _case("log_axis", comp="cartesian", tracks=17, steps_lo=1900, steps_hi=2000, periods=30,
              n_omega=201, n_dir=24, n_phi=25, w_lo=0.2, w_hi=2.0, axis="logGrid"),
        # FP64-class spectra for a misfit loss
        _case("misfit_double_float", dtype="double-float", tracks=32, steps_lo=2000,
              steps_hi=2000, periods=30, n_omega=128, n_dir=32, n_phi=32),
        # a few tracks on a small screen in the reference's FP64
        _case("screen_double", dtype="double", mode="near", motion="helical", tracks=5,
              steps_lo=1500, steps_hi=1500, periods=16, gamma=100.0, n_omega=64, n_dir=20,
              n_phi=24),
        # the reference's FP32 mode
        _case("undulator_float", dtype="float", tracks=16, steps_lo=1201, steps_hi=1201,
              periods=16, gamma=30.0, K=0.3, n_omega=150, n_dir=32, n_phi=32, dir_max=1.0),
        # a gradient step on a far-field spectrum: forward and backward
        _case("far_gradient", kind="gradient", tracks=128, steps_lo=2000, steps_hi=2000,
              periods=30, n_omega=128, n_dir=32, n_phi=32),
        # a gradient step on a screen spectrum: forward and backward
        _case("screen_gradient", kind="gradient", mode="near", motion="helical", tracks=24,
              steps_lo=2500, steps_hi=3000, periods=20, gamma=300.0, n_omega=128, n_dir=24,
              n_phi=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _points(c):
    return c["n_omega"] * c["n_dir"] * c["n_phi"] * c["tracks"] * (c["steps_lo"] + c["steps_hi"]) / 2


# point-steps above which a drawn case of a family would cost more than the largest listed one
_CAP = {"far mixed": 3e11, "near mixed": 1.5e11, "double": 4e8, "double-float": 8e9, "float": 3e9,
        "far gradient": 3.4e10, "near gradient": 8e9, "log": 4e9}


def draw(rng):
    """One more case: a family of the listed ones at other sizes."""
    fam = rng.choice(["far mixed", "far mixed", "betatron", "near mixed", "log", "double",
                      "double-float", "float", "far gradient", "near gradient"])
    near = fam.startswith("near") or (fam == "double" and rng.random() < 0.5)
    c = _case(None, mode="near" if near else "far", motion="helical" if near else "undulator",
              gamma=rng.uniform(100.0, 400.0), K=rng.uniform(0.1, 1.0))
    steps = _log_int(rng, 150, 8000)
    c.update(tracks=_log_int(rng, 1, 200), steps_lo=max(150, int(steps * rng.uniform(0.4, 1.0))),
             steps_hi=steps, n_omega=_log_int(rng, 24, 700), n_dir=_log_int(rng, 2, 80),
             n_phi=_log_int(rng, 1, 80), w_lo=rng.uniform(0.0, 0.9), w_hi=rng.uniform(1.1, 3.5))
    c["steps_lo"] = min(c["steps_lo"], c["steps_hi"])
    c["periods"] = max(4, steps // 64)
    if fam == "far mixed":
        c["comp"] = rng.choice(["total", "cartesian", "cartesian_complex"])
        c["snaps"] = rng.choice([1, 1, 2, 9])
    elif fam == "near mixed":
        c["comp"] = rng.choice(["total", "cartesian"])
    elif fam == "betatron":
        c.update(motion="betatron", track_f32=rng.random() < 0.5,
                 steps_hi=max(500, 2 * c["steps_hi"]), n_omega=_log_int(rng, 64, 400))
    elif fam == "log":
        c["axis"] = rng.choice(["logGrid", "wavelengthGrid"])
        c["w_lo"] = rng.uniform(0.1, 0.6)
    elif fam in ("double", "double-float", "float"):
        c["dtype"] = fam
        if fam == "float":  # FP32 phases: short tracks of low energy
            c.update(gamma=rng.uniform(15.0, 40.0), periods=min(c["periods"], 20))
    else:
        c["kind"] = "gradient"
    cap = _CAP["far mixed" if fam == "betatron" else fam]
    while _points(c) > cap:  # shrink towards the family's largest listed case
        k = rng.choice(["tracks", "n_dir", "n_phi"])
        c[k] = max(2 if k == "n_dir" else 1, int(c[k] * 0.7))
        if c["tracks"] == 1 and c["n_dir"] == 2 and c["n_phi"] == 1:
            break
    return c


# ------------------------------------------------------------------ inputs
def _tracks(c, seed):
    rng = np.random.default_rng(seed)
    f = np.float32 if c["track_f32"] else np.float64
    # the lengths belong to the case: every seed's batch has the same shape
    lengths = np.random.default_rng(c["tracks"] * 100003 + c["steps_hi"]).integers(
        c["steps_lo"], c["steps_hi"] + 1, c["tracks"])
    out = []
    if c["motion"] == "betatron":
        dt = 1.0 / 64
        for n in map(int, lengths):
            ph = rng.uniform(0, 2 * np.pi, 2)
            out.append(wl.betatron_track(
                rng.uniform(200, 800), rng.uniform(0.5, 3.0) / wl.UM_PER_BETATRON_PERIOD, ph[0],
                n, dt, amp_y=0.3 * rng.uniform(0.5, 3.0) / wl.UM_PER_BETATRON_PERIOD,
                phase_y=ph[1], weight=rng.uniform(0.5, 1.5), dtype=f))
        return out, dt
    g0 = c["gamma"]
    dt = (c["periods"] + 2.0) / c["steps_hi"]
    sig = 2.0 / wl.UM_PER_UNDULATOR_PERIOD
    for n in map(int, lengths):
        x0, y0 = sig * rng.standard_normal(2)
        xp, yp = (0.05 / g0) * rng.standard_normal(2)
        out.append(wl.undulator_track(
            g0 * (1 + 0.01 * rng.standard_normal()), c["K"], c["periods"], dt, n_steps=n, x0=x0,
            y0=y0, xp=xp, yp=yp, helical=c["motion"] == "helical",
            stagger=c["mode"] == "far", weight=rng.uniform(0.5, 1.5), dtype=f))
    return out, dt


def _screen(c):
    return 20.0 * c["periods"]


def _args(c):
    if c["motion"] == "betatron":
        om, top = (2e3, 2e5), 0.025
    else:
        w1 = 2 * c["gamma"] ** 2 / (1 + c["K"] ** 2 / (1 if c["motion"] == "helical" else 2))
        om, top = (c["w_lo"] * w1, c["w_hi"] * w1), c["dir_max"] / c["gamma"]
    if c["mode"] == "near":
        top *= _screen(c)
    a = {"grid": [om, (0.0, top), (0.0, 2 * np.pi), (c["n_omega"], c["n_dir"], c["n_phi"])],
         "mode": c["mode"], "dtype": c["dtype"]}
    if c["axis"] != "uniform":
        a["Features"] = [c["axis"]]
    return a


def _calc(c):
    with contextlib.redirect_stdout(io.StringIO()):
        return SynchRad(_args(c))


def prepare(case, seed):
    tracks, dt = _tracks(case, seed)
    calc = _calc(case)
    st = {"case": case, "dt": dt, "L": _screen(case) if case["mode"] == "near" else None}
    if case["kind"] == "spectrum":
        st.update(calc=calc, tracks=tracks)
        return st
    n = (case["n_omega"], case["n_dir"], case["n_phi"])
    st["layout"] = sag.make_layout([len(t[0]) for t in tracks], dt, calc._host_axes, n,
                                   mode=case["mode"], L_screen=st["L"] or 0.0)
    st["coords"] = [torch.tensor(np.concatenate([t[k] for t in tracks]), dtype=torch.float64,
                                 device="cuda", requires_grad=True) for k in range(6)]
    st["weight"] = torch.tensor([t[6] for t in tracks], dtype=torch.float64, device="cuda",
                                requires_grad=True)
    st["upstream"] = _upstream(case, seed, "cuda")
    return st


def _upstream(c, seed, device):
    """dL/dS of a weighted energy loss: smooth positive weights over the grid."""
    rng = np.random.default_rng(seed + 77)
    w = [1.0 + 0.5 * np.sin(np.linspace(0, 3, k) + rng.uniform(0, 6))
         for k in (c["n_phi"], c["n_dir"], c["n_omega"])]
    return torch.tensor(w[0][:, None, None] * w[1][None, :, None] * w[2], device=device)


def run(state):
    c = state["case"]
    if c["kind"] == "spectrum":
        calc = state["calc"]
        calc.calculate_spectrum([list(t) for t in state["tracks"]], timeStep=state["dt"],
                                comp=c["comp"], L_screen=state["L"], nSnaps=c["snaps"],
                                verbose=False)
        return {k: _kept(c, calc.Data["radiation"][k]) for k in VEC[c["comp"]]}
    fn = sag.far_total_spectrum if c["mode"] == "far" else sag.near_total_spectrum
    spec = fn(*state["coords"], state["weight"], state["layout"])
    grads = torch.autograd.grad(spec, state["coords"] + [state["weight"]],
                                grad_outputs=state["upstream"])
    return {"spectrum": spec.detach().float(), "gradients": [g.float() for g in grads]}


def _kept(c, spectrum):
    """What the program keeps of a spectrum: the 32-bit precisions' results,
    which come widened, are stored as the 32-bit values they are good for."""
    return spectrum.astype(np.float32) if c["dtype"] in ("mixed", "float") else spectrum


def work(case):
    """Inputs once, outputs once; per track, direction and step the retarded
    phase and the amplitude (about 60 flops), and the sum over steps at every
    frequency: term by term at the 64-bit and 32-bit port and on uneven axes,
    by a transform over the steps (about 100 flops a step and 5 N log2 N for
    each component) where the frequencies are evenly spaced."""
    steps = case["tracks"] * (case["steps_lo"] + case["steps_hi"]) / 2
    n_o, n_d = case["n_omega"], case["n_dir"] * case["n_phi"]
    n_out = len(VEC[case["comp"]]) * case["snaps"]
    real = 4 if (case["track_f32"] or case["dtype"] == "float") else 8
    b = 6 * real * steps + 8.0 * n_out * n_o * n_d
    comps = 2 if case["mode"] == "far" else 6
    term_by_term = case["dtype"] in ("double", "float") or case["axis"] != "uniform"
    if term_by_term:
        fl = steps * n_d * (60.0 + n_o * (8.0 + 4.0 * comps))
    else:
        fl = steps * n_d * (60.0 + 50.0 * comps)
        fl += case["tracks"] * case["snaps"] * n_d * comps * 10.0 * n_o * math.log2(2 * n_o)
    if case["kind"] == "gradient":
        b = 2 * b + 8.0 * 7 * steps
        fl *= 3
    return {"bytes": b, "flops": fl}


# ------------------------------------------------------------------ 64 bits
def _axes64(c):
    (o0, o1), (d0, d1), (p0, p1), (no, nd, nph) = _args(c)["grid"]
    f = np.float32 if c["dtype"] == "float" else np.float64
    if c["axis"] == "logGrid":
        om = o0 * np.exp(np.log(o1 / o0) / (no - 1.0) * np.arange(no))
    elif c["axis"] == "wavelengthGrid":
        om = 1.0 / np.linspace(1.0 / o1, 1.0 / o0, no)
    else:
        om = np.linspace(o0, o1, no)
    d = np.linspace(d0, d1, nd).astype(f)
    ph = (p0 + (p1 - p0) / nph * np.arange(nph)).astype(f)
    return om.astype(f), d, ph


def _phase_sum(tau, dtau, om, amps, uniform):
    """sum_s amp_s exp(i om_j tau_s) over the steps with om_j |dtau_s| < pi.

    tau, dtau [D, S]; amps: list of real [D, S]; returns complex [D, N] each.
    Frequencies j = a B + b on an even axis: exp(i om_aB tau) exp(i b dom tau),
    contracted over the steps; a block of B frequencies that the limit cuts is
    summed term by term."""
    n = om.numel()
    blk = max(1, int(math.sqrt(n))) if uniform else 1
    na = -(-n // blk)
    dom = (om[-1] - om[0]) / (n - 1) if uniform else om.new_zeros(())
    first = om[torch.arange(na, device=om.device) * blk]
    last = om[torch.clamp(torch.arange(na, device=om.device) * blk + blk - 1, max=n - 1)]
    biggest = torch.maximum(first.abs(), last.abs())
    adt = dtau.detach().abs()
    whole = biggest * adt[..., None] < math.pi                       # [D, S, na]
    Q = torch.exp(1j * (torch.arange(blk, device=om.device, dtype=om.dtype) * dom) * tau[..., None])
    E = torch.exp(1j * first * tau[..., None]) * whole
    k, D = len(amps), tau.shape[0]
    amp = torch.stack(amps, dim=-1)                                   # [D, S, k]
    A = torch.matmul((E[..., None, :] * amp[..., None]).flatten(2).transpose(1, 2), Q)
    A = A.reshape(D, k, na * blk)[:, :, :n].transpose(1, 2).reshape(D * n, k)
    if blk > 1:
        smallest = torch.minimum(first.abs(), last.abs())
        cut = (~whole) & (smallest * adt[..., None] < math.pi)
        d, s, a = torch.nonzero(cut, as_tuple=True)
        for lo in range(0, d.numel(), 2_000_000):
            dd, ss, aa = d[lo:lo + 2_000_000], s[lo:lo + 2_000_000], a[lo:lo + 2_000_000]
            j = aa[:, None] * blk + torch.arange(blk, device=om.device)
            oj = om[torch.clamp(j, max=n - 1)]
            ok = (j < n) & (oj.abs() * adt[dd, ss][:, None] < math.pi)
            e, b = torch.nonzero(ok, as_tuple=True)
            z = torch.exp(1j * oj[e, b] * tau[dd[e], ss[e]])
            A = A.index_add(0, dd[e] * n + j[e, b], z[:, None] * amp[dd[e], ss[e]])
    out = [v.reshape(D, n) for v in A.unbind(1)]
    return out


def _track_amplitudes(c, x, y, z, ux, uy, uz, dt, om, dir64, ph64, L, upto):
    """Complex Cartesian amplitudes [D, N] of one track, D = n_phi * n_dir."""
    P, D = torch.meshgrid(ph64, dir64, indexing="ij")
    P, D = P.reshape(-1, 1), D.reshape(-1, 1)
    n = x.numel() - 1
    t = torch.arange(n, device=x.device, dtype=torch.float64) * dt
    g2 = 1 + ux * ux + uy * uy + uz * uz
    g = torch.sqrt(g2)
    b = [ux / g, uy / g, uz / g]
    one_m_bz = (1 + ux * ux + uy * uy) / (g * (g + uz))
    uniform = c["axis"] == "uniform" and om.numel() > 3
    sl = slice(0, upto)
    if c["mode"] == "far":
        nx, ny, nz = torch.sin(D) * torch.cos(P), torch.sin(D) * torch.sin(P), torch.cos(D)
        omc = 2 * torch.sin(0.5 * D) ** 2
        tau = (t - z[:-1]) + omc * z[:-1] - nx * x[:-1] - ny * y[:-1]
        plain = tau
        bm = [0.5 * (v[1:] + v[:-1]) for v in b]
        a = [(v[1:] - v[:-1]) / dt for v in b]
        den = 0.5 * (one_m_bz[1:] + one_m_bz[:-1]) + omc * bm[2] - nx * bm[0] - ny * bm[1]
        c2 = 1 / den
        c1 = (nx * a[0] + ny * a[1] + nz * a[2]) * c2 * c2
        amps = [c1 * (nk - bk) - c2 * ak for nk, bk, ak in zip((nx, ny, nz), bm, a)]
    else:
        X, Y = D * torch.cos(P), D * torch.sin(P)
        dx, dy, dz = X - x[:-1], Y - y[:-1], L - z[:-1]
        rho2 = dx * dx + dy * dy
        r = torch.sqrt(rho2 + dz * dz)
        tau = (t - z[:-1]) + rho2 / (r + dz)                          # t + r - L
        plain = tau + L
        nk = (dx / r, dy / r, dz / r)
        one_m_nz = rho2 / (r * (r + dz))
        bn = (b[0][:-1] - nk[0], b[1][:-1] - nk[1], one_m_nz - one_m_bz[:-1])
        amps = [v / r for v in bn] + [v / (r * r) for v in nk]
    dtau = torch.cat([plain[:, :1], tau[:, 1:] - tau[:, :-1]], dim=1)
    s = _phase_sum(tau[:, sl], dtau[:, sl], om, [v[:, sl] for v in amps], uniform)
    if c["mode"] == "near":
        s = [s[3 + k] + 1j * om * s[k] for k in range(3)]
    return s


def exact(case, seed):
    c = case
    if not torch.cuda.is_available():
        return None
    tracks, dt = _tracks(c, seed)
    steps = sum(len(t[0]) for t in tracks)
    pts = c["n_omega"] * c["n_dir"] * c["n_phi"] * float(steps) * c["snaps"]
    if pts * (6 if c["mode"] == "near" else 3) * (3 if c["kind"] == "gradient" else 1) > 1.25e12:
        return None
    if c["axis"] != "uniform" and pts > 1.5e10:
        return None
    dev = torch.device("cuda")
    om_h, dir_h, ph_h = _axes64(c)
    # a 32-bit call's grid and step are its 32-bit values
    f = np.float32 if c["dtype"] == "float" else np.float64
    om = torch.tensor((f(2 * np.pi) * om_h).astype(np.float64), device=dev)
    ph64 = torch.tensor(ph_h.astype(np.float64), device=dev)
    dt = float(f(dt))
    grad = c["kind"] == "gradient"
    nd, npk, no = c["n_dir"], c["n_phi"], c["n_omega"]
    keys = VEC[c["comp"]]
    out = {k: torch.zeros(c["snaps"], npk * nd, no, dtype=torch.float64, device=dev) for k in keys}
    up = _upstream(c, seed, dev).reshape(npk * nd, no) if grad else None
    grads = [[] for _ in range(7)]
    longest = max(len(t[0]) for t in tracks)
    rows = max(1, int(3e9 / (16.0 * longest * 6 * (2 * math.sqrt(no) + 8 if c["axis"] == "uniform"
                                                  else 3 * no))))
    per = max(1, rows // npk)
    for tr in tracks:
        co = [torch.tensor(np.asarray(v).astype(f).astype(np.float64), device=dev) for v in tr[:6]]
        w = torch.tensor(float(tr[6]), dtype=torch.float64, device=dev)
        if grad:
            co = [v.requires_grad_(True) for v in co]
            w.requires_grad_(True)
        acc = [torch.zeros_like(v) for v in co + [w]]
        n = len(tr[0])
        cuts = np.linspace(0, n, c["snaps"] + 1).astype(np.uint32)[1:]
        for d0 in range(0, nd, per):
            d64 = torch.tensor(dir_h[d0:d0 + per].astype(np.float64), device=dev)
            k = d64.numel()
            rows_at = (torch.arange(npk, device=dev)[:, None] * nd + d0
                       + torch.arange(k, device=dev)).reshape(-1)
            for i, cut in enumerate(cuts):
                if cut < 2:
                    continue
                A = _track_amplitudes(c, *co, dt, om, d64, ph64, _screen(c), int(cut) - 1)
                if c["comp"] == "total":
                    S = w * dt * dt * sum(v.real ** 2 + v.imag ** 2 for v in A)
                    out["total"][i].index_add_(0, rows_at, S.detach())
                    if grad:
                        g = torch.autograd.grad(S, co + [w], grad_outputs=up[rows_at])
                        acc = [p + q for p, q in zip(acc, g)]
                elif c["comp"] == "cartesian":
                    for key, v in zip(keys, A):
                        out[key][i].index_add_(0, rows_at, w * dt * dt * (v.real ** 2 + v.imag ** 2))
                else:
                    for key, v in zip(("x", "y", "z"), A):
                        out[key + "re"][i].index_add_(0, rows_at, torch.sqrt(w) * dt * v.real)
                        out[key + "im"][i].index_add_(0, rows_at, torch.sqrt(w) * dt * v.imag)
        if grad:
            for lst, v in zip(grads, acc):
                lst.append(v.reshape(-1))
    if grad:
        return {"spectrum": out["total"][0].reshape(npk, nd, no),
                "gradients": [torch.cat(v) for v in grads]}
    return {k: v.reshape(c["snaps"], npk, nd, no).transpose(-1, -3).contiguous().cpu().numpy()
            for k, v in out.items()}
