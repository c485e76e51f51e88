"""The GPU set-up's Debye-Hueckel boundary at the sizes where its split over
threads changes, and at the ends of its exponential's range, against the host
set-up (CUDA's or the host's exp and sqrt are within an ulp or two; the sums
run in another order: 1e-14 of the largest value, the bound of the set-up's
other tests)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200 import _lib  # noqa: E402
from multigrid_b200.molecule import DEFAULT_PHYSICS  # noqa: E402
from multigrid_b200.problem import physics_struct, setup_fine  # noqa: E402

KEYS = ("oC", "oE", "oN", "uC", "f", "x0")


def both(n, h, atoms, physics):
    out = {k: torch.full((n ** 3,), 7.0, dtype=torch.float64, device="cuda")
           for k in KEYS}
    atoms = np.ascontiguousarray(atoms, dtype=np.float64)
    _lib.check("pmg_setup_fine_d", _lib.lib.pmg_setup_fine_d(
        n, h, atoms.ctypes.data_as(_lib.PD), len(atoms),
        ctypes.byref(physics_struct(physics)),
        *[ctypes.c_void_p(out[k].data_ptr()) for k in KEYS], None))
    torch.cuda.synchronize()
    host = setup_fine(n, h, atoms, physics)
    return {k: out[k].cpu().numpy() for k in KEYS}, host


def atoms_in(n, h, count, seed):
    rng = np.random.default_rng(seed)
    return np.column_stack([rng.uniform(0.1 * h, (n - 1.1) * h, (count, 3)),
                            rng.uniform(0.5, 2.0, count),
                            rng.normal(0, 0.5, count)])


# rows of 1 to 4 points past a multiple of the points per thread; fewer and
# more atoms than warps and than a tile
@pytest.mark.parametrize("n,count", [(3, 1), (4, 7), (5, 8), (6, 9), (7, 257),
                                     (34, 600)])
@pytest.mark.parametrize("salt", [0.0, 0.15, 30.0])
def test_boundary_sizes(n, count, salt):
    physics = dict(DEFAULT_PHYSICS, ionic_strength=salt)
    dev, host = both(n, 0.9, atoms_in(n, 0.9, count, n + count), physics)
    for k in ("oC", "oE", "oN", "uC", "f"):
        assert np.array_equal(dev[k], host[k].ravel()), k
    x0 = host["x0"].ravel()
    assert np.abs(dev["x0"] - x0).max() <= 1e-14 * np.abs(x0).max()


def test_boundary_on_a_grid_point():
    """An atom on a face point gives the host's infinity there and only
    there; terms below the smallest double leave every other value finite."""
    n, h = 9, 40.0
    at = np.array([[100.0, 120.0, 160.0, 1.5, 0.7],
                   [0.0, 2 * h, 3 * h, 1.5, -0.4]])
    dev, host = both(n, h, at, dict(DEFAULT_PHYSICS, ionic_strength=200.0))
    x0, d = host["x0"].ravel(), dev["x0"]
    fine = np.isfinite(x0)
    assert fine.sum() == x0.size - 1
    assert np.array_equal(np.isfinite(d), fine)
    assert np.array_equal(d[~fine], x0[~fine])
