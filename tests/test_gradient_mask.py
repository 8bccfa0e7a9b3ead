"""Far-field gradients of steps within a thousandth of the |dphase| < pi limit,
seen from a direction far off the beam axis.

A track along a direction theta_0 with gamma theta_0 = 150, observed along
itself: the terms of the retarded time's step, dt theta_0^2 / 2 each, cancel to
dt / (2 gamma^2), so that FP32 differences of them are wrong by half a per cent.
The frequencies span the limit's +-0.3 %: which of them a step includes decides
half of its gradient, and the gradient has to take the ones that the forward
took.  An axis that is uneven by 1e-9 goes term by term, with the mask of every
point from double-float times.

Tolerance: both ways round 1 - n.beta to FP32 before it cancels, at most
4 x 2^-24 (gamma theta)^2 / 2 = 2.7e-3, the gradient contains it cubed at most:
8e-3 on either side, 1.6e-2 between them.  A step taken whole changes by order
one.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1.6e-2
DT, N, K = 1.0 / 64, 257, 0.3


def _gradients(uneven):
    from synchrad_gb300 import autograd as sag
    th0 = 0.086
    g = 150.0 / th0
    t = DT * np.arange(N)
    beta = 1 - (1 + K * K / 2) / (2 * g * g)     # mean velocity along theta_0
    uy = K * np.cos(2 * np.pi * t)
    up = np.sqrt(g * g - 1 - uy * uy)
    coords = [beta * t * np.sin(th0), K / (2 * np.pi * g) * np.sin(2 * np.pi * t),
              beta * t * np.cos(th0), up * np.sin(th0), uy, up * np.cos(th0)]
    limit = np.pi / (DT * (1 + K * K / 2) / (2 * g * g))
    om = limit * np.linspace(0.997, 1.003, 64)
    if uneven:
        om[1::2] *= 1 + 1e-9
    th = np.array([th0, th0 + 0.02 / g])
    axes = [om, np.sin(th), np.cos(th), np.zeros(1), np.ones(1)]
    lay = sag.make_layout([N], DT, axes, (64, 2, 1), mode="far")
    ts = [torch.tensor(c, device="cuda", requires_grad=True) for c in coords]
    S = sag.far_total_spectrum(*ts, torch.ones(1, dtype=torch.float64, device="cuda"), lay)
    S.sum().backward()
    return S.detach().cpu().numpy(), [t.grad.cpu().numpy() for t in ts]


def test_steps_at_the_limit():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    s0, even = _gradients(False)
    s1, walked = _gradients(True)
    assert np.linalg.norm(s0 - s1) <= TOL * np.linalg.norm(s1)
    for part in (slice(0, 3), slice(3, 6)):
        a, b = np.stack(even[part]), np.stack(walked[part])
        assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)
