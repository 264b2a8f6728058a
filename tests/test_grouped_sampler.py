"""Chains of the sampler with several walkers per warp: walker counts that leave a warp's last
groups empty, every group width, one to four spin words, magnetisation sectors, and streams
that continue from call to call, against the CPU replay bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as po

gpu = pytest.mark.gpu


def rbm(N, M):
    rng = np.random.default_rng(1000 * N + M)
    return (0.1 * (rng.normal(size=M) + 1j * rng.normal(size=M)),
            0.1 * (rng.normal(size=(N, M)) + 1j * rng.normal(size=(N, M))))


@gpu
@pytest.mark.parametrize("N,M,chains,sector", [
    (3, 1, 1, None), (12, 32, 2, None), (12, 24, 3, None), (64, 17, 5, None), (20, 33, 1, None), (65, 64, 9, None),
    (130, 60, 3, None), (30, 75, 7, None), (200, 128, 2, None), (128, 100, 5, None), (9, 200, 2049, None),
    (8, 10, 5, 0), (10, 40, 3, 4), (36, 75, 9, 0), (64, 100, 3, -6), (6, 150, 2050, 2)])
def test_chains_equal_the_replay(N, M, chains, sector):
    import rbmongpu_gb300 as rg
    b, W = rbm(N, M)
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W)
    steps, sweeps, therm, seed = 3, 2, 3, 41
    mc = rg.MonteCarloLoop(chains * steps, sweeps, therm, chains, seed=seed)
    if sector is not None:
        mc.set_total_z_symmetry(sector)
    spins, _, _ = mc.samples(psi, log_psi=False)
    ref, _, _, acc, rej = po.mc_run(po.RBM(b, W, 1.0), None, chains, steps, sweeps, therm, seed=seed, want_eloc=False,
                                    total_z=sector is not None, sector=sector or 0)
    assert np.array_equal(spins.reshape(steps, chains, -1), ref)
    got, props, per = mc.acceptance(per_chain=True)
    assert np.array_equal(per, np.asarray(acc, np.uint64)) and props == int((acc + rej).sum())


@gpu
@pytest.mark.parametrize("N,M,walkers", [(24, 20, 6), (24, 40, 3), (70, 90, 5), (11, 130, 2051)])
def test_streams_continue(N, M, walkers):
    """Five sweeps of a persistent chain in one call and in calls of 1, 3 and 1 sweeps."""
    import rbmongpu_gb300 as rg
    b, W = rbm(N, M)
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W)
    one, many = rg.Chain(psi, walkers, seed=9), rg.Chain(psi, walkers, seed=9)
    one.sweep_async(psi, None, 5)
    for n in (1, 3, 1):
        many.sweep_async(psi, None, n)
    a, c = one.checkpoint(), many.checkpoint()
    for k in a:
        assert np.array_equal(a[k], c[k]), k
