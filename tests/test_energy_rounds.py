"""Local energies, a lane of the kernel taking two strings a round: numbers of off-diagonal strings
around a round's 8 and 16, two-site flips beside single ones in one round, several spin words.

Further strings with coefficient zero add exact zeros (also to a compensated sum: only the split
between its two parts may move), but make the last strings share their round with others, or take
the branch for several flips: the energies stay the same bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, M, strings, pairs", [(9, 20, 1, 0), (9, 40, 7, 0), (9, 70, 8, 0), (12, 100, 9, 0), (20, 130, 16, 0),
                                                  (20, 170, 17, 0), (30, 200, 24, 0), (40, 260, 25, 3), (70, 400, 33, 16),
                                                  (130, 500, 60, 9), (200, 30, 1, 8)])
def test_zero_strings_in_the_same_round_change_nothing(N, M, strings, pairs):
    import rbmongpu_gb300 as rg
    from rbmongpu_gb300 import operators as o
    rng = np.random.default_rng(N + strings)
    noise = lambda *s: rng.normal(0, 0.05, s) + 1j * rng.normal(0, 0.05, s)
    psi = rg.Psi(np.zeros(N), np.zeros(N), noise(M), noise(N, M))
    flips = [[int(i)] for i in rng.permutation(N)[:strings]]
    for k in range(pairs):
        flips.insert(int(rng.integers(0, len(flips) + 1)), [int(i) for i in rng.choice(N, 2, replace=False)])
    up = rng.integers(0, 2, (7, N)).astype(bool)
    words = np.zeros((7, (N + 63) // 64), np.uint64)
    for i in range(N):
        words[:, i // 64] |= up[:, i].astype(np.uint64) << np.uint64(i % 64)
    coef = noise(len(flips)) * 20

    def energies(zeros):
        rows = [[(o.X, i) for i in sites] for sites in flips + zeros]
        return rg.local_energies(psi, rg.Operator(*o.table(rows, np.append(coef, np.zeros(len(zeros))))), words)

    alone = energies([])
    assert np.abs(alone).min() > 0
    for zeros in ([[0]] * 8, [[0]] * 9, [[0, N - 1]], [[1]] * 7 + [[0, N - 1]]):
        np.testing.assert_array_equal(energies(zeros), alone)
