"""The gradient's scratch follows the samples of the call: a few configurations of a large net hold
what these need."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_few_samples_of_a_large_net():
    """Of 40 samples the sums have two splits of (1 + N) M entries of 16 bytes, 14 MB for the three
    of a gradient; the other buffers are below 40 MB.  A thread has a scratch of its own."""
    import torch
    import rbmongpu_gb300 as rg
    N, M = 256, 576
    rng = np.random.default_rng(1)
    psi = rg.Psi(np.zeros(N), np.zeros(N), rng.normal(0, 0.05, M) + 0j, rng.normal(0, 0.05, (N, M)) + 0j)
    words = rng.integers(0, 2 ** 63, (40, 4)).astype(np.uint64)
    ens, op = rg.FixedSamples(N, words), rg.Operator(*rg.operators.tfim_chain(N))
    rg.ExpectationValue().gradient(psi, op, ens)   # the kernels are loaded
    held = []

    def call():
        before = torch.cuda.mem_get_info()[0]
        for f in (rg.ExpectationValue().gradient, rg.ExpectationValue().eloc_gradient):
            f(psi, op, ens)
        held.append(before - torch.cuda.mem_get_info()[0])
    t = threading.Thread(target=call)
    t.start()
    t.join()
    assert 0 <= held[0] < 256 << 20
