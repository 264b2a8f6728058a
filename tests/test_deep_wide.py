"""Deep nets whose layers are so wide that a block's shared memory holds fewer configurations than
the kernels take otherwise: the same energies and gradients as the kernels that take one
configuration a block, bit for bit (every configuration's arithmetic is theirs)."""
import numpy as np
import pytest

import rbmongpu_gb300 as rg
import test_deep_fp64
from test_deep_pairs import net, with_env

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(720, 720, 720), (900, 900), (600, 800, 800)])
def test_adjoint(sizes):
    """Eight neighbours a pass need more than the 227 KB of a block, four do not."""
    N = 6
    psi, op = net(N, sizes, 3), rg.Operator(*rg.operators.tfim_chain(N, 1.0, 0.9))
    words = np.random.default_rng(1).integers(0, 2 ** N, (5, 1)).astype(np.uint64)

    def gradient():
        return rg.ExpectationValue().eloc_gradient(psi, op, rg.FixedSamples(N, words))
    (g, E), (h, F) = gradient(), with_env("RBMG_DEEP_ADJOINT_BATCH", 1, gradient)
    assert np.array_equal(g, h) and E == F


@pytest.mark.parametrize("walkers,sizes,per_block", [
    (7300, (40, 20), 8),       # seven blocks an SM: 128 threads
    (3700, (180, 90), 8),      # four: 256
    (3700, (260, 30), 8),      # four, more units than 256: 512
    (1300, (300, 5, 3), 8),    # two: 512
    (5, (1000, 40), 8),        # one: 1024
    (5, (7,), 8),
    (5, (600, 30), 4), (3, (600, 30), 2),
])
def test_sampler_threads(walkers, sizes, per_block):
    """Threads of a block by the blocks an SM holds (152 SMs): the chains of one walker a block."""
    N = 5
    psi = net(N, sizes, 4)

    def chain():
        mc = rg.MonteCarloLoop(2 * walkers, 1, 1, walkers, seed=6)
        sp, lp, _ = mc.samples(psi)
        return sp, lp, mc.acceptance(per_chain=True)[2]
    for x, y in zip(with_env("RBMG_DEEP_WALKERS_PER_BLOCK", per_block, chain),
                    with_env("RBMG_DEEP_WALKERS_PER_BLOCK", 1, chain)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("samples,sizes,batch", [
    (700, (40, 20), 8), (500, (180, 90), 8), (500, (260, 30), 8), (200, (300, 5, 3), 8), (5, (600, 600, 600), 8),
    (5, (7,), 8), (5, (600, 30), 4), (700, (40, 20), 2), (3, (600, 30), 2),
])
def test_adjoint_threads(samples, sizes, batch):
    N = 6
    psi, op = net(N, sizes, 3), rg.Operator(*rg.operators.tfim_chain(N, 1.0, 0.9))
    words = np.random.default_rng(1).integers(0, 2 ** N, (samples, 1)).astype(np.uint64)

    def gradient():
        return rg.ExpectationValue().eloc_gradient(psi, op, rg.FixedSamples(N, words))
    (g, E), (h, F) = (with_env("RBMG_DEEP_ADJOINT_BATCH", q, gradient) for q in (batch, 1))
    assert np.array_equal(g, h) and E == F


@pytest.mark.parametrize("sizes", [(128, 10), (129, 10), (10, 129, 3)])
def test_estimator_threads(sizes):
    """The FP64 estimator takes 128 threads a block up to 128 units and 512 above."""
    test_deep_fp64.test_estimator(9, sizes, 17, False)
