"""The divide by corrections of a product with a kept reciprocal
(csrc/row_stencil.cuh div_by_recip) has the bits of the divide for every
numerator and divisor: on the host (tests/cpp/div_by_recip.cu), and on the GPU
where a whole problem is scaled to the ends of the exponent range."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_class_of_operand_on_the_host(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "div_by_recip")
    subprocess.run([nvcc, "-std=c++17", "-O2", "--fmad=false", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "multigrid_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "div_by_recip.cu"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


# float: numerators of the colour passes whose residuals underflow, subnormal
# ones, and ones beyond the corrected range; double: both sides of its ends
# (beyond them the damping's products underflow and nothing is left to see; the
# class's cycle, whose coarse CG stops below 1e-8, cannot be scaled down)
@pytest.mark.gpu
@pytest.mark.parametrize("precision,exponent", [
    ("fp64", 490), ("fp64-fast", -500), ("fp64-fast", 490),
    ("mixed", -100), ("mixed", -125), ("mixed", 80)])
def test_scaled_problem_streamed_and_not(precision, exponent):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from multigrid_b200 import PBELinearProblem, WORKLOADS
    from multigrid_b200.problem import set_finest_streaming, setup_fine
    w = WORKLOADS["pb65"]
    fine = setup_fine(w.n, w.h, w.atoms(), w.physics)
    fine["f"] = np.ldexp(fine["f"], exponent)
    fine["x0"] = np.ldexp(fine["x0"], exponent)
    out = {}
    try:
        for on in (True, False):
            set_finest_streaming(on)
            with PBELinearProblem(w.base, w.nlev, w.box, precision,
                                  w.physics) as p:
                p.set_fine(**fine)
                p.buildmultilevelops()
                assert p.finest_streamed() == on
                p.solve(tol=0.0, max_cycles=3)
                out[on] = p.potential().ravel().copy()
    finally:
        set_finest_streaming(True)
    assert np.isfinite(out[True]).all() and out[True].any()
    assert np.array_equal(out[True], out[False])
