"""The serving kernel takes two strings, and in its sums two rows, per packed operation.
Checked where the pairing has remainders: off-diagonal strings alone between diagonal ones
and in odd numbers, single flips beside two-site flips in one pair, rows in odd numbers, a
site that no string flips, and every compiled number of hidden units per lane (M = 17, 42,
100, 200, 400 and 560: 1, 2, 4, 8, 13 and 18).

Tolerances are those of the served gradients in tests/test_serving.py: energies within 1e-6
and gradients within 1e-5 of the largest entry of the single-network pass on the same
configurations (FP32 terms of the same sums), and the same bits for both tile heights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def interleaved(N):
    """A diagonal string, then one, two or three off-diagonal ones in turn; site N - 1 is
    flipped by none, site 4 by three strings, site 6 by a two-site string only."""
    import rbmongpu_gb300 as rg
    X, Y, Z = rg.operators.X, rg.operators.Y, rg.operators.Z
    flips = [[(X, i)] for i in range(N - 1) if i != 6]
    flips += [[(X, 4), (X, 6)], [(Y, 4), (Z, 1)]]
    strings, q = [], 0
    for i in range(N):
        strings.append([(Z, i), (Z, (i + 1) % N)])
        strings += flips[q:q + 1 + i % 3]
        q += 1 + i % 3
    strings += flips[q:]
    coef = [(-0.9 + 0.01 * n) * (1.0 if s[0][0] != Y else 1j) for n, s in enumerate(strings)]
    return rg.operators.table(strings, coef)


@pytest.mark.parametrize("N, M, walkers", [(17, 17, 33), (21, 42, 64), (33, 100, 257), (37, 200, 31), (50, 400, 40),
                                           (31, 560, 20)])
def test_served_gradient_with_remainders(N, M, walkers):
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(N)
    noise = lambda *s: rng.normal(0, 0.05, s) + 1j * rng.normal(0, 0.05, s)
    psi = rg.Psi(np.zeros(N), np.zeros(N), noise(M), noise(N, M), 1.0, False, True)
    op = rg.Operator(*interleaved(N))
    results = []
    for rows in (8, 16):
        batch = rg.Batch([(psi, op, walkers, 11)])
        batch.set_shape(4, rows)
        batch.run(5, 1)
        results.append(batch.result(0, want_eloc=True))
    E, g, eloc = results[0]
    g_ref, E_ref = rg.ExpectationValue().gradient(psi, op, rg.FixedSamples(N, batch.spins(0)))
    assert abs(E - eloc.mean()) <= 1e-13 * np.abs(eloc).max()
    assert abs(E - E_ref) <= 1e-6 * abs(E_ref)
    assert not g[:2 * N].any()
    assert np.abs(g - g_ref).max() <= 1e-5 * np.abs(g_ref).max()
    assert results[1][0] == E
    np.testing.assert_array_equal(results[1][1], g)
