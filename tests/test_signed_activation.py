"""Chains with hidden angles whose real part is an exact zero of either sign, or small and of
both signs: the packed activation folds the sign of Re theta in with the sign bits, and the
spins and accept counts equal the CPU restatement's, which multiplies by +-1, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, M, chains", [(8, 20, 5), (16, 64, 33), (20, 90, 9), (12, 250, 7), (10, 400, 3)])
@pytest.mark.parametrize("real", [0.0, 0.0625])
def test_chains_at_zero_real_angles(N, M, chains, real):
    import rbmongpu_gb300 as rg
    from oracle import pyoracle as po
    rng = np.random.default_rng(N * M)
    sign = lambda *s: rng.choice([-1.0, 1.0], s)
    # real parts +-real: sums over an even number of spins are multiples of 2 real, often zero
    b = real * (1 + sign(M)) + 0.4j * rng.normal(size=M)
    W = real * sign(N, M) + 0.2j * rng.normal(size=(N, M))
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W, 1.0, False, True)
    mc = rg.MonteCarloLoop(chains * 3, 1, 2, chains, seed=5)
    sp, _, _ = mc.samples(psi)
    spins, _, _, acc, _ = po.mc_run(po.RBM(b, W, 1.0), None, chains, 3, 1, 2, seed=5, want_eloc=False)
    assert np.array_equal(sp.reshape(3, chains, -1), spins)
    assert int(mc.acceptance()[0]) == int(acc.sum()) > 0
