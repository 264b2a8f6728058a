"""The weights, means and gradients of exact summation are formed on the device from end to
end: one block and 512 of them, one chunk of 65536 states and several, a sector with one state.

Tolerances: energies are FP64 weighted sums of the local energies that rg.local_energies
returns for the same states, 1e-12; gradients are FP32 sums of up to 32 terms added in FP64, whose terms
carry a relative error below 2^-22 and exceed the result by at most 40, 1e-5 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lc(z):
    """The activation and its derivative (include/quantum_state/psi_functions.hpp:49-57)."""
    s = np.where(z.real > 0, 1.0, -1.0)
    u = s * z
    D = 9.19376335670885 + u * (10.2180213465 + u * (7.771429504240965 + u * (3.746646023906276 + u)))
    dD = 10.2180213465 + u * (2 * 7.771429504240965 + u * (3 * 3.746646023906276 + u * 4))
    n = 5.49914721954 - 2.16564366435 * u
    return 0.9003320053750442 * u + n / D - 0.598139, s * (0.9003320053750442 + (-2.16564366435 * D - n * dD) / (D * D))


def rbm(N, M):
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(N)
    b = rng.normal(0, 0.1, M) + 1j * rng.normal(0, 0.1, M)
    W = rng.normal(0, 0.1, (N, M)) + 1j * rng.normal(0, 0.1, (N, M))
    return rg.Psi(np.zeros(N), np.zeros(N), b, W, 1.0, False, True), b, W


@pytest.mark.parametrize("N, M, sector", [(1, 1, None), (2, 3, 2), (3, 40, None), (9, 12, None), (17, 5, None), (18, 3, 0)])
def test_gradient_against_numpy(N, M, sector):
    import rbmongpu_gb300 as rg
    psi, b, W = rbm(N, M)
    ens = rg.ExactSummation(N)
    states = np.arange(1 << N, dtype=np.uint64)
    s = np.where((states[:, None] >> np.arange(N, dtype=np.uint64)) & np.uint64(1), 1.0, -1.0)
    if sector is not None:
        ens.set_total_z_symmetry(sector)
        keep = s.sum(1) == sector
        states, s = states[keep], s[keep]
    op = rg.Operator(*rg.operators.heisenberg_chain(N) if sector is not None else rg.operators.tfim_chain(N, 1.0, 0.7))
    f, T = lc(b + s @ W)
    lp = f.sum(1)
    w = np.exp(2 * (lp.real - lp.real.max()))
    z = w.sum()
    assert abs(np.log(psi.norm(ens)) - (lp.real.max() + 0.5 * np.log(z))) < 1e-9
    psi.normalize(ens)
    w /= z
    E = rg.local_energies(psi, op, states[:, None])
    g, _ = rg.ExpectationValue().gradient(psi, op, ens)
    value = rg.ExpectationValue()(psi, op, ens)   # of the same local energies; the gradient's come from its own pass
    mean = (w * E).sum()
    assert abs(value - mean) <= 1e-9 * np.abs(E).max()   # the numpy weights' own rounding
    # <E O*> + conj<E_k> - 2 <E><O*>, E_k = sum_n e_n O_k(s'_n); for these Hermitian operators
    # <E_k> = <E O>* over all states, up to psi's FP32 parameters
    d, _ = rg.ExpectationValue().eloc_gradient(psi, op, ens, True)
    O = np.concatenate([T, (s[:, :, None] * T[:, None, :]).reshape(len(s), -1)], 1)
    cov = (w[:, None] * (E - mean)[:, None] * O.conj()).sum(0)
    if sector is None:
        assert np.linalg.norm(g[2 * N:] - 2 * cov) <= 1e-5 * np.linalg.norm(cov) + 1e-6
        assert np.linalg.norm(d[2 * N:] - 2 * cov) <= 1e-5 * np.linalg.norm(cov) + 1e-6
    assert not g[:2 * N].any() and not d[:2 * N].any()


def test_non_finite_states_stay_refused():
    import rbmongpu_gb300 as rg
    psi = rg.Psi(np.zeros(3), np.zeros(3), np.full(4, 1.5e308 + 0j), np.zeros((3, 4), complex), 1.0, False, True)
    ens = rg.ExactSummation(3)
    op = rg.Operator(*rg.operators.tfim_chain(3, 1.0, 1.0))
    for call in (lambda: psi.norm(ens), lambda: rg.ExpectationValue().gradient(psi, op, ens),
                 lambda: rg.ExpectationValue()(psi, op, ens)):
        with pytest.raises(Exception, match="non-finite log psi"):
            call()
    good, _, _ = rbm(3, 4)   # and the next call finds its scratch as it should be
    assert np.isfinite(good.norm(ens))
