"""The deep-net sampler and adjoint with two configurations per packed operation against the
kernels that take one configuration a block: identical spins, energies and gradients for layer
sizes around the tiles (one unit, fewer than a warp, more than a block), one to three layers,
connections that repeat or rotate, walker and neighbour counts that leave halves empty, and
weights rewritten by the device optimiser."""
import os

import numpy as np
import pytest

import rbmongpu_gb300 as rg

gpu = pytest.mark.gpu


def net(N, sizes, seed, conn=None):
    """Dense layers, or per layer the input of connection c of unit j by conn(l, c, j, fan)."""
    rng = np.random.default_rng(seed)
    b, cn, W, fan = [], [], [], N
    for l, m in enumerate(sizes):
        sd = np.sqrt(0.3 / fan / 2)
        b.append(rng.normal(0, sd, m) + 1j * rng.normal(0, sd, m))
        cn.append(np.array([[c if conn is None else conn(l, c, j, fan) for j in range(m)] for c in range(fan)]))
        W.append(rng.normal(0, sd, (fan, m)) + 1j * rng.normal(0, sd, (fan, m)))
        fan = m
    return rg.PsiDeep(np.zeros(N), np.zeros(N), b, cn, W, 1 + 0.2j * rng.normal(size=sizes[-1]))


def with_env(name, value, f):
    old = os.environ.get(name)
    os.environ[name] = str(value)
    try:
        return f()
    finally:
        if old is None:
            del os.environ[name]
        else:
            os.environ[name] = old


def same(psi, op, walkers):
    def chain():
        mc = rg.MonteCarloLoop(2 * walkers, 1, 2, walkers, seed=6)
        sp, lp, _ = mc.samples(psi)
        return sp, lp, mc.acceptance(per_chain=True)[2]

    def gradient():
        return rg.ExpectationValue().eloc_gradient(psi, op, rg.MonteCarloLoop(walkers, 1, 2, walkers, seed=7))
    a, b = chain(), with_env("RBMG_DEEP_WALKERS_PER_BLOCK", 1, chain)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    (g, E), (h, F) = gradient(), with_env("RBMG_DEEP_ADJOINT_BATCH", 1, gradient)
    assert np.array_equal(g, h) and E == F


@gpu
@pytest.mark.parametrize("N,sizes,walkers", [(3, (1,), 1), (9, (5,), 7), (12, (130, 3), 9), (17, (31, 65, 2), 8),
                                             (70, (64, 63), 17), (20, (129, 128, 127), 3), (5, (2, 200), 10)])
def test_layer_sizes(N, sizes, walkers):
    same(net(N, sizes, N), rg.Operator(*rg.operators.tfim_chain(N, 1.0, 0.9)), walkers)


@gpu
@pytest.mark.parametrize("kind", ["repeated", "rotated"])
def test_connections(kind):
    conn = {"repeated": lambda l, c, j, fan: (c // 2 + j) % fan,
            "rotated": lambda l, c, j, fan: (c + 2 * j) % fan}[kind]
    same(net(14, (20, 9, 6), 3, conn), rg.Operator(*rg.operators.heisenberg_chain(14)), 11)


@gpu
def test_weights_of_the_device_optimiser():
    N = 12
    psi = net(N, (20, 10), 5)
    op = rg.Operator(*rg.operators.tfim_chain(N, 1.0, 0.9))
    rg.Optimizer("vanilla", psi.num_params, eta=0.05).step(psi, op, rg.MonteCarloLoop(64, 1, 2, 64, seed=1))
    moved = rg.MonteCarloLoop(64, 1, 2, 64, seed=2).samples(psi)[0]
    fresh = psi.copy()     # the same parameters through the host
    assert np.array_equal(moved, rg.MonteCarloLoop(64, 1, 2, 64, seed=2).samples(fresh)[0])
    same(psi, op, 13)
