"""The FP64 and FP32 kernels at the sizes where their work split can go wrong.

A warp takes 32 / L directions and L x K consecutive frequencies; what depends
on (direction, step) alone is computed once per 32 steps and shared.  Checked
against the CPU oracle (the reference kernels' arithmetic): frequency counts
around the tiles, one direction and directions that leave a warp partly filled,
steps around a multiple of 32, even and uneven axes (rotations, or a sine and a
cosine per point), phases small and large, and steps that the |dphase| < pi rule
cuts.

Tolerances as in the golden-vector tests: FP64 1e-12 relative L2 (the phases
round alike; sin and cos differ in the last bits: ~1e-15 per term against a
cancellation of up to ~1e3 in the weak points of these grids), FP32 1e-5.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from synchrad_gb300 import workloads as wl  # noqa: E402

TOL = {"double": 1e-12, "float": 1e-5}


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("dtype", ["double", "float"])
@pytest.mark.parametrize("features", [[], ["logGrid"]])
@pytest.mark.parametrize("n_omega,n_dir,n_phi,n_steps,comp", [
    (1, 1, 1, 2, "total"), (7, 3, 1, 33, "cartesian"), (8, 1, 5, 65, "total"),
    (33, 5, 3, 96, "total"), (65, 2, 7, 97, "cartesian_complex"), (257, 3, 3, 64, "total"),
    (300, 33, 2, 40, "cartesian")])
def test_sizes(mode, dtype, features, n_omega, n_dir, n_phi, n_steps, comp):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import host
    from synchrad_gb300.calc import SynchRad
    rng = np.random.default_rng(n_omega)
    g0, K, dt = 40.0, 0.7, 1.0 / 24
    w1 = wl.fundamental(g0, K)
    # the axis reaches past the sampling limit: the rule cuts steps
    top = 0.02 if mode == "far" else 1.0
    f = np.float64 if dtype == "double" else np.float32
    tracks = [wl.undulator_track(g0 * (1 + 0.01 * rng.standard_normal()), K, 4, dt,
                                 n_steps=n_steps + 3 * i, stagger=mode == "far",
                                 weight=rng.uniform(0.5, 1.5), dtype=f) for i in range(3)]
    args = {"grid": [(0.1 * w1, 4.0 * w1), (0.0, top), (0.0, 2 * np.pi), (n_omega, n_dir, n_phi)],
            "mode": mode, "dtype": dtype, "Features": features}
    call = dict(comp=comp, nSnaps=2 if n_steps > 2 else 1, L_screen=50.0 if mode == "near" else None)
    ref, *_ = host.calculate_spectrum(dict(args), [list(t) for t in tracks], dt, **call)
    calc = SynchRad(dict(args))
    if features:  # the axis by np.exp: its last bit differs between platforms
        a = host.init_args(dict(args))
        calc.Args["omega"] = np.asarray(a["omega"]).astype(calc.dtype)
        calc._init_data()
    calc.calculate_spectrum([list(t) for t in tracks], timeStep=dt, verbose=False, **call)
    got = np.concatenate([calc.Data["radiation"][k].ravel() for k in sorted(ref)])
    exp = np.concatenate([ref[k].ravel() for k in sorted(ref)])
    norm = np.linalg.norm(exp)
    if norm == 0:
        assert not got.any()
        return
    assert np.linalg.norm(got - exp) / norm <= TOL[dtype]
