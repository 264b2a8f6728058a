"""The sampler's choice between whole warps and groups of lanes, by the blocks that an SM gets (152
SMs): walker w's chain on both sides of every limit."""
import numpy as np
import pytest

from test_sampler_lanes import psi, run

pytestmark = pytest.mark.gpu


# walkers in blocks of 608: up to 3 on whole warps (K = 1: 2, K = 3: 1); from K = 8 on (250, 400 units)
# odd numbers up to 13 too; 300 units have no groups
@pytest.mark.parametrize("N, M, walkers", [(9, 20, (33, 1216, 1217)), (12, 64, (33, 1824, 1825)), (10, 80, (33, 608, 609)),
                                           (70, 128, (33, 1824, 1825)), (11, 150, (33, 1824, 1825)), (13, 190, (33, 1825)),
                                           (12, 250, (33, 1825, 2433, 3041, 8513)), (9, 300, (33, 1825, 9000)),
                                           (10, 400, (33, 1825, 2432, 2433, 3041))])
def test_a_walkers_chain(N, M, walkers):
    p = psi(N, M)
    first = run(p, walkers[0])
    for w in walkers[1:]:
        np.testing.assert_array_equal(run(p, w), first)
