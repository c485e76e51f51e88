"""Limits of the GPU set-up that the host checks before any device call."""
import ctypes

import pytest

from multigrid_b200 import _lib
from multigrid_b200.molecule import DEFAULT_PHYSICS
from multigrid_b200.problem import physics_struct


@pytest.mark.parametrize("natoms", [22369622, 2 ** 31 - 1])
def test_more_probe_positions_than_an_int_counts_are_refused(natoms):
    """96 probe positions per atom are counted in 32 bits; the atoms are not
    read for the refusal (the array here holds none)."""
    assert natoms * 96 >= 2 ** 31
    some = (ctypes.c_double * 8)()
    rc = _lib.lib.pmg_setup_fine_d(
        9, 0.5, some, natoms, ctypes.byref(physics_struct(DEFAULT_PHYSICS)),
        *[ctypes.cast(some, ctypes.c_void_p)] * 6, None)
    assert rc == _lib.PMG_ERR_ARG
    assert b"probe positions" in _lib.lib.pmg_last_error()
