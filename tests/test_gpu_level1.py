"""Level 1 of the one-launch lowest levels: by its inverse, by the CG where the
inverse does not exist, and the modes that change nothing there."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200 import PBELinearProblem  # noqa: E402
from multigrid_b200.molecule import Workload, level_n  # noqa: E402
from multigrid_b200.problem import setup_fine  # noqa: E402


def problem(base, nlev):
    n = level_n(base, nlev)
    w = Workload("shape", base, nlev, 0.8, 12, 0.25 * 0.8 * (n - 1), 11)
    return w, setup_fine(w.n, w.h, w.atoms(), w.physics)


def solve(w, fine, precision, trilinear=False, throughput=False):
    with PBELinearProblem(w.base, w.nlev, w.box, precision, w.physics,
                          hierarchy="reference") as p:
        p.set_throughput_mode(throughput)
        p.set_fine(**fine)
        p.buildmultilevelops(trilinear)
        r = p.solve(tol=1e-10, max_cycles=60)
        return r, p.potential().ravel().copy()


# level 1 of 1, 27 and 125 unknowns
@pytest.mark.parametrize("precision", ["mixed", "fp64-fast"])
@pytest.mark.parametrize("base,nlev", [(1, 4), (2, 4), (3, 3)])
def test_no_inverse_of_a_negative_definite_level(base, nlev, precision):
    """The whole system with its sign changed has the same solution. Its level
    1 has no positive pivot, so the CG solves it (to 1e-4 of its residual); the
    potentials agree as far as the solves' tolerance carries (1e-8)."""
    w, fine = problem(base, nlev)
    minus = {k: v if k == "x0" else -v for k, v in fine.items()}
    r, x = solve(w, fine, precision, trilinear=True)
    s, y = solve(w, minus, precision, trilinear=True)
    assert r.relres < 1e-10 and s.relres < 1e-10
    assert abs(s.cycles - r.cycles) <= 2
    assert np.linalg.norm(y - x) <= 1e-8 * np.linalg.norm(x)


@pytest.mark.parametrize("precision", ["mixed", "fp64-fast", "fp64"])
def test_throughput_mode_gives_the_same_bits(precision):
    w, fine = problem(2, 4)
    r, x = solve(w, fine, precision)
    s, y = solve(w, fine, precision, throughput=True)
    assert s.cycles == r.cycles
    assert np.array_equal(x, y)
