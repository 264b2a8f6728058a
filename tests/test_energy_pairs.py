"""Local energies by the form that takes two strings a lane and round (more than eight strings of one
or two flips, in runs) against the form of one string a round: a string of three flips with
coefficient zero, which adds exact zeros, sends an operator there.  Bit for bit: rounds that are and
are not full, both kinds in one round, several spin words, all numbers of units per lane."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, M, ones, twos", [(9, 20, 9, 0), (9, 40, 0, 9), (10, 70, 0, 16), (12, 100, 0, 17), (20, 130, 16, 16),
                                              (20, 170, 18, 15), (30, 200, 30, 40), (40, 260, 0, 65), (70, 300, 64, 70),
                                              (70, 400, 3, 45), (130, 500, 0, 130), (200, 30, 100, 200)])
def test_against_one_string_a_round(N, M, ones, twos):
    import rbmongpu_gb300 as rg
    from rbmongpu_gb300 import operators as o
    rng = np.random.default_rng(N + ones + twos)
    noise = lambda *s: rng.normal(0, 0.05, s) + 1j * rng.normal(0, 0.05, s)   # noqa: E731
    psi = rg.Psi(np.zeros(N), np.zeros(N), noise(M), noise(N, M))
    rows = [[(o.X, int(rng.integers(N)))] for _ in range(ones)]
    rows += [[(int(rng.integers(1, 3)), int(i)) for i in rng.choice(N, 2, replace=False)] for _ in range(twos)]
    rows.insert(1, [(o.Z, 0), (o.Z, 1)])
    coef = 20 * noise(len(rows))
    up = rng.integers(0, 2, (9, N)).astype(bool)
    words = np.zeros((9, (N + 63) // 64), np.uint64)
    for i in range(N):
        words[:, i // 64] |= up[:, i].astype(np.uint64) << np.uint64(i % 64)
    two = rg.local_energies(psi, rg.Operator(*o.table(rows, coef)), words)
    one = rg.local_energies(psi, rg.Operator(*o.table(rows + [[(o.X, 0), (o.X, 1), (o.X, 2)]], np.append(coef, 0))), words)
    assert np.abs(two).min() > 0
    np.testing.assert_array_equal(two, one)
