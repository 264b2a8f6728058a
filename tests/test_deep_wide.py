"""Deep nets whose layers are so wide that a block's shared memory holds fewer configurations than
the kernels take otherwise: the same energies and gradients as the kernels that take one
configuration a block, bit for bit (every configuration's arithmetic is theirs)."""
import numpy as np
import pytest

import rbmongpu_gb300 as rg
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
