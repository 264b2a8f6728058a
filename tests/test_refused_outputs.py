"""An exact summation over a log psi that is not finite is refused and leaves the caller's arrays
as they were (through the C ABI: the Python calls return fresh arrays)."""
import ctypes as C

import numpy as np
import pytest

import rbmongpu_gb300 as rg
from rbmongpu_gb300 import _lib

pytestmark = pytest.mark.gpu


def doubles(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture
def call():
    N, M = 6, 4
    psi = rg.Psi(np.zeros(N), np.zeros(N), 1e308 * np.ones(M), np.zeros((N, M)))
    return N, psi, rg.Operator(*rg.operators.tfim_chain(N)), rg.ExactSummation(N), _lib.lib()


@pytest.mark.parametrize("name", ["rbmg_ev_gradient", "rbmg_ev_eloc_gradient", "rbmg_ev_fluctuation_gradient"])
def test_gradients(call, name):
    N, psi, op, ens, lib = call
    grad, value = np.full(2 * psi.num_params, 7.0), np.full(2, 7.0)
    args = [psi._h, op._h, ens._h] + ([1] if "eloc" in name else []) + [doubles(grad), doubles(value)]
    assert getattr(lib, name)(*args) == _lib.RBMG_ENAN
    assert (grad == 7.0).all() and (value == 7.0).all()


def test_samples(call):
    N, psi, op, ens, lib = call
    spins = np.full(1 << N, 7, np.uint64)
    lp, e = np.full(2 << N, 7.0), np.full(2 << N, 7.0)
    assert lib.rbmg_ensemble_samples(ens._h, psi._h, op._h, spins.ctypes.data_as(C.POINTER(C.c_uint64)), doubles(lp),
                                     doubles(e)) == _lib.RBMG_ENAN
    assert (spins == 7).all() and (lp == 7.0).all() and (e == 7.0).all()


def test_s_matrix():
    """Of 8 MB and more, whose pages are made present while the GPU works."""
    N, M = 8, 80
    psi, lib = rg.Psi(np.zeros(N), np.zeros(N), 1e308 * np.ones(M), np.zeros((N, M))), _lib.lib()
    out = np.full(2 * psi.num_params ** 2, 7.0)
    assert out.nbytes >= 8 << 20
    assert lib.rbmg_s_matrix(psi._h, rg.ExactSummation(N)._h, 0, doubles(out)) == _lib.RBMG_ENAN
    assert (out == 7.0).all()
