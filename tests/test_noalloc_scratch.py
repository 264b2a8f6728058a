"""The no-allocation energy does not depend on what its fixed scratch holds when the call starts
(its sum counts arriving blocks there, and overlapping calls of other threads, themselves
undefined, may leave any count behind)."""
import ctypes as C

import numpy as np
import pytest

import rbmongpu_gb300 as rg
from rbmongpu_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [3, 12])   # one block of the sum, and sixteen
@pytest.mark.parametrize("byte", [0x01, 0xff])
def test_leftovers(N, byte):
    rng = np.random.default_rng(N)
    M = 2 * N
    psi = rg.Psi(np.zeros(N), np.zeros(N), rng.normal(0, 0.05, M) + 0j, rng.normal(0, 0.05, (N, M)) + 0j)
    op = rg.Operator(*rg.operators.tfim_chain(N, 1.0, 0.7))
    lib, got = _lib.lib(), []
    for fill in (0, byte, None):
        if fill is not None:
            assert lib.rbmg_noalloc_scratch_fill(fill) == _lib.RBMG_OK
        out = (C.c_double * 2)()
        assert lib.rbmg_ev_value_exact_noalloc(psi._h, op._h, N, out) == _lib.RBMG_OK
        got.append((out[0], out[1]))
    assert got[0] == got[1] == got[2] and got[0][0] != 0.0
