"""The FP64 kernel on few frequencies and many directions, where a direction takes
one, two or four lanes of a warp (a point each) and a warp up to 32 directions:
counts that leave the last warp partly filled, steps around a multiple of 32, cut
steps and snapshots.  Against the CPU oracle, with the tolerance of
test_port_shapes.py and for its reasons.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_port_shapes import test_sizes as _against_the_oracle  # noqa: E402


@pytest.mark.parametrize("mode", ["far", "near"])
@pytest.mark.parametrize("n_omega,n_dir,n_phi,n_steps,comp,features", [
    (1, 71, 67, 33, "total", []), (2, 61, 53, 64, "cartesian", []),
    (2, 35, 30, 31, "total", ["logGrid"]), (3, 47, 23, 40, "cartesian_complex", []),
    (4, 71, 67, 32, "total", ["logGrid"])])
def test_few_frequencies(mode, n_omega, n_dir, n_phi, n_steps, comp, features):
    _against_the_oracle(mode, "double", features, n_omega, n_dir, n_phi, n_steps, comp)
