"""Messages between the CTAs of the kernels that hold the lowest levels on
chip: their order against late warps, and what a caller sees when one does
not arrive (every wait expects 16 bytes more than are sent and runs out)."""
import contextlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200 import PBELinearProblem, _lib, pmgc  # noqa: E402
from multigrid_b200._lib import PmgError  # noqa: E402
from multigrid_b200.molecule import Workload, level_n  # noqa: E402
from multigrid_b200.problem import setup_fine  # noqa: E402
from test_oracle import apbs_maps, apbs_params  # noqa: E402


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


@contextlib.contextmanager
def messages_lost():
    _lib.check("pmg_test_message_short_delivery",
               _lib.lib.pmg_test_message_short_delivery(16))
    try:
        yield
    finally:
        _lib.check("pmg_test_message_short_delivery",
                   _lib.lib.pmg_test_message_short_delivery(0))


def reports_lost(call):
    with pytest.raises(PmgError) as e:
        call()
    assert e.value.status == _lib.PMG_ERR_TIMEOUT
    assert b"did not arrive" in _lib.lib.pmg_last_error()


def dominant(n, seed):
    rng = np.random.default_rng(seed)
    ops = [np.full(n ** 3, 27.0)] + [rng.uniform(0.0, 1.0, n ** 3)
                                     for _ in range(13)]
    return (torch.as_tensor(np.stack(ops), device="cuda"),
            torch.as_tensor(rng.normal(size=n ** 3), device="cuda"))


# one and two planes per CTA
@pytest.mark.parametrize("n", [10, 17])
def test_lost_message_of_the_cg_is_reported(n):
    ops, f = dominant(n, n)

    def cg():
        x = torch.zeros_like(f)
        it = pmgc.cg_level(n, n, n, list(ops), f, x)
        return it, x

    def vcghs():
        x = torch.zeros_like(f)
        work = [torch.zeros_like(f) for _ in range(3)]
        it = pmgc.Vcghs(n, n, n, ops, torch.zeros_like(f), f, x, *work, 200,
                        1e-10)
        return it, x

    for call in (cg, vcghs):
        want = call()
        with messages_lost():
            reports_lost(call)
        got = call()
        assert got[0] == want[0] and torch.equal(got[1], want[1])


# levels 5^3 to 17^3, 5^3 and 9^3 and 7^3 and 13^3 in one launch; a level 1 of
# 11^3 by itself
@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64-fast"])
@pytest.mark.parametrize("base,nlev", [(2, 4), (2, 3), (3, 3), (5, 2)])
def test_lost_message_of_a_solve_is_reported(base, nlev, precision):
    w, fine = problem(base, nlev)
    want = solve(w, fine, precision)
    with messages_lost():
        reports_lost(lambda: solve(w, fine, precision))
    got = solve(w, fine, precision)
    assert got[0] == want[0] and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("kw", [dict(nlev=2), dict(nlev=1),
                                dict(nlev=2, mgsmoo=4, itmax=3)])
def test_lost_message_of_the_driver_is_reported(kw):
    """The driver queues its coarsest CG (17^3 here) and, with mgsmoo 4, the
    smoother's without reading them back; the stop test's norm brings the
    loss."""
    n = 33 if kw["nlev"] == 2 else 17
    maps = apbs_maps(n, n)
    iparm, rparm = apbs_params(n, **kw)
    dev = [torch.as_tensor(np.ascontiguousarray(maps[k]), device="cuda",
                           dtype=torch.float64)
           for k in ("xf", "yf", "zf", "gxcf", "gycf", "gzcf", "a1cf", "a2cf",
                     "a3cf", "ccf", "fcf")]

    def drive():
        u = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
        return pmgc.Vmgdriv(iparm, rparm, u, *dev), u

    want = drive()
    with messages_lost():
        reports_lost(drive)
    got = drive()
    assert got[0] == want[0] and torch.equal(got[1], want[1])


@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64-fast"])
@pytest.mark.parametrize("base,nlev", [(2, 4), (5, 2)])
def test_lost_message_of_a_pcg_solve_is_reported(base, nlev, precision):
    w, fine = problem(base, nlev)

    def pcg():
        with PBELinearProblem(w.base, w.nlev, w.box, precision,
                              w.physics) as p:
            p.set_fine(**fine)
            p.buildmultilevelops()
            r = p.pcg_solve(tol=1e-10, max_iters=60)
            return r.cycles, p.potential().ravel().copy()

    want = pcg()
    with messages_lost():
        reports_lost(pcg)
    got = pcg()
    assert got[0] == want[0] and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("base,nlev", [(2, 4), (5, 2)])
def test_lost_message_of_a_caller_s_cycles_is_reported(base, nlev):
    """Cycles queued one by one: the next call that waits for the stream
    reports the loss, and only that one."""
    w, fine = problem(base, nlev)

    def run(end):
        with PBELinearProblem(w.base, w.nlev, w.box, "fp64",
                              w.physics) as p:
            p.set_fine(**fine)
            p.buildmultilevelops()
            for _ in range(3):
                p.v_cycle()
            return end(p)

    def residual(p):
        return p.compute_residual_2()

    def potential(p):
        return p.potential().ravel().copy()

    want = run(residual), run(potential)
    for end in (residual, potential):
        with messages_lost():
            reports_lost(lambda: run(end))

            def told_once(p):
                reports_lost(lambda: end(p))
                return end(p)

            run(told_once)
    assert run(residual) == want[0]
    assert np.array_equal(run(potential), want[1])


def test_cycles_after_a_solve_that_reported_a_loss():
    w, fine = problem(2, 4)
    with PBELinearProblem(w.base, w.nlev, w.box, "fp64", w.physics) as p:
        p.set_fine(**fine)
        p.buildmultilevelops()
        with messages_lost():
            reports_lost(lambda: p.solve(tol=1e-10, max_cycles=60))
        p.v_cycle()
        assert np.isfinite(p.compute_residual_2())
