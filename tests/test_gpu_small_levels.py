"""The kernels that hold a small level on chip, at the sizes where their split
over threads and CTAs changes, against the CPU restatement.

Sums run in another order than the restatement's, so iterates agree to
rounding amplified by the iteration (1e-12 of the largest value, the bound
the other CG tests use) and the iteration counts are equal.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200 import pmgc  # noqa: E402

DEV = torch.device("cuda:0")


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64,
                           device=DEV)


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def level(nx, ny, nz, kind, seed):
    """A symmetric, strictly diagonally dominant operator with random
    couplings, a cc, a right-hand side and a start with a nonzero shell."""
    rng = np.random.default_rng(seed)
    n3 = nx * ny * nz
    ops = [np.full(n3, float(kind))] + [rng.uniform(0.0, 1.0, n3) for _ in
                                        range(3 if kind == 7 else 13)]
    return (ops, rng.uniform(0.0, 0.1, n3), rng.normal(size=n3),
            rng.normal(size=n3) * 0.1)


# one point; one CTA at its limit (343 unknowns) and just above it; one and
# two planes per CTA, fewer planes than CTAs; the largest; the general path
SHAPES = [(3, 3, 3), (9, 9, 9), (10, 9, 9), (17, 3, 17), (5, 17, 10),
          (17, 17, 9), (17, 17, 11), (17, 17, 17), (18, 9, 9)]


@pytest.mark.parametrize("kind", [7, 27])
@pytest.mark.parametrize("shape", SHAPES)
def test_vcghs_shapes(restatement, shape, kind):
    nx, ny, nz = shape
    ops, cc, f, x0 = level(nx, ny, nz, kind, nx + 31 * ny + 7 * nz + kind)
    xo = x0.copy()
    it_o, ro = restatement.cghs(nx, ny, nz, ops, cc, f, xo, 400, 1e-10)
    work = [torch.full((nx * ny * nz,), 3.0, dtype=torch.float64, device=DEV)
            for _ in range(3)]
    work[1].zero_()
    work[2].zero_()
    x = T(x0)
    it = pmgc.Vcghs(nx, ny, nz, T(np.stack(ops)), T(cc), T(f), x, *work, 400,
                    1e-10)
    assert it == it_o and 0 < it < 400
    assert rel(x.cpu().numpy(), xo) <= 1e-12
    # the residual it leaves, against the first one
    r0 = np.linalg.norm(f)
    assert np.linalg.norm(work[2].cpu().numpy() - ro) <= 1e-12 * r0
    # the direction's shell is zero whatever the array held
    p = work[0].cpu().numpy().reshape(nz, ny, nx).copy()
    p[1:-1, 1:-1, 1:-1] = 0.0
    assert not p.any()


@pytest.mark.parametrize("n", [3, 4, 9, 10, 11, 15, 17])
def test_class_cg_sizes(restatement, n):
    ops, _, f, x0 = level(n, n, n, 27, n)
    # the restatement's CG of the class reads a zero-shell start
    x0 = x0.reshape(n, n, n)
    shell = np.ones((n, n, n), bool)
    shell[1:-1, 1:-1, 1:-1] = False
    x0[shell] = 0.0
    xo = x0.ravel().copy()
    it_o = restatement.cg(n, ops, f, xo)
    x = T(x0.ravel())
    it = pmgc.cg_level(n, n, n, [T(a) for a in ops], T(f), x)
    assert it == it_o > 0
    assert rel(x.cpu().numpy(), xo) <= 1e-12


# hierarchies whose levels of up to 17^3 run in one launch: 9^3 over 5^3, two
# and three levels below the top, a 3^3 coarsest level, 13^3 over 7^3 (125
# unknowns), 17^3 over 9^3 (343 unknowns); and whose level 1 (13^3, 19^3) runs
# by itself, on chip and not
@pytest.mark.parametrize("base,nlev", [(2, 3), (2, 4), (1, 5), (3, 3), (4, 3),
                                       (6, 2), (9, 2)])
def test_low_levels_of_the_cycle(restatement, base, nlev):
    """FP64 against the restated class: the same cycles, the potential to
    1e-12 (sums in another order); the refinement paths to 1e-8 of it."""
    from multigrid_b200 import PBELinearProblem
    from multigrid_b200.molecule import Workload, level_n
    from multigrid_b200.problem import setup_fine
    n = level_n(base, nlev)
    w = Workload("shape", base, nlev, 0.8, 12, 0.25 * 0.8 * (n - 1), 11)
    fine = setup_fine(w.n, w.h, w.atoms(), w.physics)
    xo, co, _ = restatement.solve(base, nlev, fine, tol=1e-10, max_cycles=100)
    for prec, tol in (("fp64", 1e-12), ("fp64-fast", 1e-8), ("mixed", 1e-8)):
        with PBELinearProblem(base, nlev, w.box, prec, w.physics,
                              hierarchy="reference") as p:
            p.set_fine(**fine)
            p.buildmultilevelops()
            r = p.solve(tol=1e-10, max_cycles=100)
            x = p.potential().ravel()
        assert r.relres < 1e-10, (prec, r.cycles, r.relres)
        assert np.linalg.norm(x - xo) <= tol * np.linalg.norm(xo), prec
        if prec == "fp64":
            assert r.cycles == co


def band(n, m, seed):
    """LINPACK upper band storage of a symmetric positive definite matrix
    (diagonally dominant), column-major with lda = m + 1."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, m + 1))  # row j: column j of the band
    for j in range(n):
        k0 = max(0, m - j)
        a[j, k0:m] = rng.uniform(-1.0, 0.0, m - k0)
    a[:, m] = 2.0 * m + rng.uniform(1.0, 2.0, n)
    return a.ravel()


# one unknown; half widths 0, around LINPACK's unrolling by five and at a
# warp; a 9^3 level's 27-point band; one that does not fit on chip
@pytest.mark.parametrize("n,m", [(1, 0), (4, 0), (6, 1), (27, 13), (40, 31),
                                 (60, 17), (343, 57), (400, 100)])
def test_band_sizes_bit_for_bit(restatement, n, m):
    a = band(n, m, n + m)
    want = a.copy()
    assert restatement.dpbfa(want, m + 1, n, m) == 0
    g = T(a)
    assert pmgc.Vdpbfa(g, m + 1, n, m) == 0
    assert np.array_equal(g.cpu().numpy(), want)
    b = np.random.default_rng(m).normal(size=n)
    xo = b.copy()
    restatement.dpbsl(want, m + 1, n, m, xo)
    x = T(b)
    pmgc.Vdpbsl(g, m + 1, n, m, x)
    assert np.array_equal(x.cpu().numpy(), xo)


@pytest.mark.parametrize("bad", [1, 5, 27])
def test_band_bad_pivot_leaves_later_columns(restatement, bad):
    n, m = 27, 13
    a = band(n, m, 3)
    a[(bad - 1) * (m + 1) + m] = -1.0
    want = a.copy()
    assert restatement.dpbfa(want, m + 1, n, m) == bad
    g = T(a)
    assert pmgc.Vdpbfa(g, m + 1, n, m) == bad
    assert np.array_equal(g.cpu().numpy(), want)
