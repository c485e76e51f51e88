"""The 27-point sweep where its tiles of 8 and 16 are cut: one point, exactly
one tile, one point more, ragged edges, and tiles of 16 on each side of full.

In double the update order fixes every bit. In float each of a point's 27
terms rounds once: with a diagonal above twice the row's couplings a sweep
amplifies by at most 2, so float and double differ by at most
28 * 2^-24 * 2 = 3.4e-6 of the largest value a sweep; 1e-5 for two.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from multigrid_b200 import pmgc  # noqa: E402

SHAPES = [(3, 3, 3), (10, 10, 4), (11, 9, 5), (19, 34, 6), (50, 50, 5),
          (51, 49, 4), (66, 67, 5)]


def T(a, dtype):
    return torch.as_tensor(a, dtype=dtype, device="cuda:0")


@pytest.mark.parametrize("iadjoint", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_gs27_tile_edges(restatement, shape, iadjoint):
    nx, ny, nz = shape
    n3 = nx * ny * nz
    rng = np.random.default_rng(nx + 7 * ny + 31 * nz)

    def rnd(lo, hi):  # float-rounded, so both precisions see the same inputs
        return rng.uniform(lo, hi, n3).astype(np.float32).astype(np.float64)

    # 26 couplings below 1: twice their sum is below 52
    ops = [rnd(52.0, 60.0)] + [rnd(0.0, 1.0) for _ in range(13)]
    f, x0 = rnd(-52.0, 52.0), rnd(-1.0, 1.0)
    xo = x0.copy()
    dp = ctypes.POINTER(ctypes.c_double)
    ptrs = (dp * 14)(*[a.ctypes.data_as(dp) for a in ops])
    restatement.lib.pmgo_gsrb27x(
        nx, ny, nz, ptrs, np.zeros(n3).ctypes.data_as(dp),
        f.ctypes.data_as(dp), xo.ctypes.data_as(dp), 2, iadjoint, 0)
    for dtype in (torch.float64, torch.float32):
        x = T(x0, dtype)
        pmgc.Vgsrb27x(nx, ny, nz, [T(a, dtype) for a in ops], None,
                      T(f, dtype), x, itmax=2, iadjoint=iadjoint)
        got = x.cpu().numpy().astype(np.float64)
        if dtype == torch.float64:
            assert np.array_equal(got, xo)
        else:
            assert np.abs(got - xo).max() <= 1e-5 * np.abs(xo).max()
