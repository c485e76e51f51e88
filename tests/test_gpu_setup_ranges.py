"""The GPU set-up outside the usual ranges, against the host set-up."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200.molecule import DEFAULT_PHYSICS  # noqa: E402
from multigrid_b200 import _lib  # noqa: E402
from multigrid_b200.problem import (kappa, physics_struct,  # noqa: E402
                                    setup_fine)

KEYS = ("oC", "oE", "oN", "uC", "f", "x0")


def setup_on_gpu(n, h, atoms, physics):
    out = {k: torch.full((n ** 3,), 7.0, dtype=torch.float64, device="cuda")
           for k in KEYS}
    atoms = np.ascontiguousarray(atoms, dtype=np.float64)
    _lib.check("pmg_setup_fine_d", _lib.lib.pmg_setup_fine_d(
        n, h, atoms.ctypes.data_as(_lib.PD), len(atoms),
        ctypes.byref(physics_struct(physics)),
        *[ctypes.c_void_p(out[k].data_ptr()) for k in KEYS], None))
    torch.cuda.synchronize()
    return {k: out[k].cpu().numpy() for k in KEYS}


def both(n, h, atoms, physics):
    return setup_on_gpu(n, h, atoms, physics), setup_fine(n, h, atoms,
                                                          physics)


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


def test_more_than_2_31_coordinates_of_kept_probe_centres():
    """7.5 million atoms that do not touch keep all their 96 probe centres:
    723 million rows of three coordinates. The masks at the few grid points
    depend on the atoms near them alone, which the host sets up."""
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    n, h, per_axis = 9, 200.0, 196
    g = (np.arange(per_axis) + 0.5) * (h * (n - 1) / per_axis)
    physics = dict(DEFAULT_PHYSICS)
    atoms = np.empty((per_axis ** 3, 5))
    atoms[:, :3] = np.stack(np.meshgrid(g, g, g, indexing="ij"),
                            -1).reshape(-1, 3)
    atoms[:, 3] = 1.5
    atoms[:, 4] = 0.0
    assert len(atoms) * 96 * 3 > 2 ** 31
    assert g[1] - g[0] > 2 * (1.5 + physics["probe_radius"])
    # faces lie half a spacing from the points along one axis
    off = np.abs(atoms[:, :3] / (h / 2) - np.rint(atoms[:, :3] / (h / 2)))
    near = atoms[(off * (h / 2) < 6.0).all(axis=1)]
    assert 1000 < len(near) < 50000
    out = setup_on_gpu(n, h, atoms, physics)
    host = setup_fine(n, h, near, physics)
    for k in ("oC", "oE", "oN", "uC"):
        want = host[k].ravel()
        assert len(np.unique(want)) > 1, k
        assert np.array_equal(out[k], want), k


# one sphere (every warp a part of it), a few, and as many as there are warps
# or more; spheres that reach past the grid, and of one column
@pytest.mark.parametrize("n,h,count,radius", [
    (33, 0.1, 1, 5.0), (33, 0.1, 1, 0.0), (40, 0.1, 12, 1.8),
    (65, 0.05, 3, 1.0), (33, 0.3, 150, 0.2), (33, 1.0, 400, 1.5)])
@pytest.mark.parametrize("probe", [0.0, 1.4])
def test_marks_of_few_and_many_spheres(n, h, count, radius, probe):
    rng = np.random.default_rng(count + n)
    atoms = np.column_stack([rng.uniform(0.0, (n - 1) * h, (count, 3)),
                             np.full(count, radius),
                             rng.normal(0, 0.5, count)])
    dev, host = both(n, h, atoms, dict(DEFAULT_PHYSICS, probe_radius=probe))
    for k in ("oC", "oE", "oN", "uC", "f"):
        assert np.array_equal(dev[k], host[k].ravel()), k
