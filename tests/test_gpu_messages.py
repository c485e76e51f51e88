"""Messages between the CTAs of the kernels that hold the lowest levels on
chip: their order against late warps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200 import PBELinearProblem, _lib  # noqa: E402
from multigrid_b200.molecule import Workload, level_n  # noqa: E402
from multigrid_b200.problem import setup_fine  # noqa: E402


def problem(base, nlev):
    n = level_n(base, nlev)
    w = Workload("shape", base, nlev, 0.8, 12, 0.25 * 0.8 * (n - 1), 11)
    return w, setup_fine(w.n, w.h, w.atoms(), w.physics)


def solve(w, fine, precision):
    with PBELinearProblem(w.base, w.nlev, w.box, precision, w.physics) as p:
        p.set_fine(**fine)
        p.buildmultilevelops()
        r = p.solve(tol=1e-10, max_cycles=60)
        return r.cycles, p.potential().ravel().copy()


# top levels of 9^3 and 5^3 (half of the warps hold no point) and of 13^3
@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64-fast"])
@pytest.mark.parametrize("base,nlev", [(2, 3), (1, 4), (1, 3), (3, 3)])
def test_late_warps_without_a_point(base, nlev, precision):
    """A warp that comes to its wait long after the rest of its plane (0.3 ms,
    several times the launch) still finds the phase it waits for: the same
    cycles and bits as without the delay."""
    w, fine = problem(base, nlev)
    want = solve(w, fine, precision)
    _lib.check("pmg_test_idle_warp_delay",
               _lib.lib.pmg_test_idle_warp_delay(300))
    try:
        got = solve(w, fine, precision)
    finally:
        _lib.check("pmg_test_idle_warp_delay",
                   _lib.lib.pmg_test_idle_warp_delay(0))
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
