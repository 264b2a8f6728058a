"""The FP64 local energy and gradient estimator of deep nets, neighbours in batches, against sums
put together in numpy from log psi and O_k of single configurations: layer sizes that change the
batch, numbers of strings around it, strings of several flips, repeated connections."""
import numpy as np
import pytest

import rbmongpu_gb300 as rg

gpu = pytest.mark.gpu


def net(N, sizes, seed, repeat=False):
    rng = np.random.default_rng(seed)
    b, cn, W, fan = [], [], [], N
    for m in sizes:
        sd = np.sqrt(0.3 / fan / 2)
        b.append(rng.normal(0, sd, m) + 1j * rng.normal(0, sd, m))
        cn.append(np.array([[(c // 2 + j) % fan if repeat else c for j in range(m)] for c in range(fan)]))
        W.append(rng.normal(0, sd, (fan, m)) + 1j * rng.normal(0, sd, (fan, m)))
        fan = m
    return rg.PsiDeep(np.zeros(N), np.zeros(N), b, cn, W, 1 + 0.3j * rng.normal(size=sizes[-1])), rng


@gpu
@pytest.mark.parametrize("N,sizes,strings,repeat", [(3, (1,), 1, False), (6, (9, 4), 15, False), (8, (33, 6, 2), 16, True),
                                                    (9, (20, 30), 17, False), (10, (300, 40), 35, False),
                                                    (7, (500, 400, 300), 5, False)])
def test_estimator(N, sizes, strings, repeat):
    psi, rng = net(N, sizes, N, repeat)
    rows = [[(3, 0), (3, N - 1)]]
    for n in range(strings):
        k = int(rng.integers(1, min(4, N)))
        rows.append([(int(rng.integers(1, 3)) if q == 0 else int(rng.integers(1, 4)), int(i))
                     for q, i in enumerate(rng.choice(N, k, replace=False))])
    coef = rng.normal(size=len(rows)) + 0.2j * rng.normal(size=len(rows))
    op = rg.Operator(*rg.operators.table(rows, coef))
    conf = rng.integers(0, 1 << N, 6).astype(np.uint64)
    lp = lambda x: psi.log_psi_s(int(x))                         # noqa: E731
    O = lambda x: rg.psi_O_k_vector(psi, int(x))                 # noqa: E731
    E, Ek, Os = [], [], []
    for x in conf:
        e, ek = 0, 0
        for c, row in zip(coef, rows):
            y, ph = int(x), c
            for t, i in row:
                s = 1 if (int(x) >> i) & 1 else -1
                if t == 2:
                    ph = ph * (-1j * s)
                if t == 3:
                    ph = ph * s
                if t in (1, 2):
                    y ^= 1 << i
            term = ph * np.exp(lp(y) - lp(x))
            e, ek = e + term, ek + term * O(y)
        E.append(e)
        Ek.append(ek)
        Os.append(O(x))
    E, Ek, Os = np.array(E), np.array(Ek), np.array(Os)
    assert np.abs(rg.local_energies(psi, op, conf) - E).max() < 1e-12 * np.abs(E).max()
    ref = (E[:, None] * Os.conj()).mean(0) + Ek.mean(0).conj() - 2 * E.mean() * Os.mean(0).conj()
    g, got = rg.ExpectationValue().gradient(psi, op, rg.FixedSamples(N, conf))
    assert abs(got - E.mean()) < 1e-12 * np.abs(E).max()
    # three sums that cancel: relative to their terms
    size = (np.abs(E)[:, None] * np.abs(Os)).mean(0).max() + np.abs(Ek).mean(0).max()
    assert np.abs(g - ref).max() < 1e-11 * size
