"""The GPU set-up outside the usual ranges, against the host set-up."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200.molecule import DEFAULT_PHYSICS  # noqa: E402
from multigrid_b200.problem import kappa  # noqa: E402
from test_gpu_boundary import both  # noqa: E402


def salty(salt):
    physics = dict(DEFAULT_PHYSICS, ionic_strength=salt)
    return physics, kappa(physics)[0]


def one_atom(n, h, radius):
    """Near the corner (0, 0, 0), a positive charge."""
    return np.array([[1.0, 1.0, 1.0, radius, 0.7]])


@pytest.mark.parametrize("h", [1e2, 1e5, 1e7, 1e12])
def test_boundary_exponent_far_below_the_smallest_double(h):
    """exp(-kappa d) of arguments to -10^3 .. -10^13: the host's zeros are
    zeros (the exponent's index has more than 32 bits from kappa d = 2.3e7
    on)."""
    n = 9
    physics, k = salty(1e4)
    assert k * h * (n - 1) > 1e3
    dev, host = both(n, h, one_atom(n, h, 1.5), physics)
    x0, d = host["x0"].ravel(), dev["x0"]
    assert (x0 == 0.0).any() and (x0 > 0.0).any()
    assert np.array_equal(d == 0.0, x0 == 0.0)
    assert np.abs(d - x0).max() <= 1e-14 * np.abs(x0).max()


def test_boundary_subnormal_values():
    """exp's arguments between -745 and -700. The argument's rounding (a few
    2^-53 of 745: below 1e-12 of the value) and half an ulp of a subnormal
    exp times the atom's factor over the distance (below 2^-1069 here)."""
    n = 33
    physics, k = salty(1e4)
    h = 800.0 / k / (n - 1)
    dev, host = both(n, h, one_atom(n, h, 1.5), physics)
    x0, d = host["x0"].ravel(), dev["x0"]
    sub = (x0 > 0.0) & (x0 < 2.2250738585072014e-308)
    assert sub.sum() > 20
    assert (np.abs(d - x0)[sub] <= 1e-12 * x0[sub] + 2.0 ** -1069).all()


def test_boundary_beyond_the_largest_double():
    """Deep inside an atom exp overflows: infinite where the host's is."""
    n, h = 9, 4.0
    physics, k = salty(1e4)
    assert k * 60.0 > 720.0
    dev, host = both(n, h, one_atom(n, h, 60.0), physics)
    x0, d = host["x0"].ravel(), dev["x0"]
    big = np.isinf(x0)
    assert big.any() and not big.all()
    assert np.array_equal(np.isinf(d), big)
    fine = ~big
    assert (np.abs(d - x0)[fine] <= 1e-12 * x0[fine]).all()
