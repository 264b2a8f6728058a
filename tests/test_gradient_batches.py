"""The gradient of a transverse-field operator takes several chunks of samples per launch and sums
within each chunk's own 32-sample groups: chunks that are and are not whole groups, a last chunk
shorter than the others, more units of work than blocks.

Against the form that stores every string's terms, a plain chunk per launch: the same FP32 sums up
to where its chunks end and the rounding of the centring energy; 1e-5 of the norm, as the other
estimator tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, M, count", [(64, 128, 7942), (64, 128, 7943), (64, 128, 20000), (140, 250, 9001), (200, 30, 25000)])
def test_batches_against_the_stored_form(N, M, count):
    """A second string of coefficient zero on a flipped site takes the general form, one plain
    chunk at a time with every string's terms stored."""
    import rbmongpu_gb300 as rg
    from rbmongpu_gb300 import operators as o
    rng = np.random.default_rng(count)
    psi = rg.Psi(np.zeros(N), np.zeros(N), rng.normal(0, 0.05, M) + 1j * rng.normal(0, 0.05, M),
                 rng.normal(0, 0.05, (N, M)) + 1j * rng.normal(0, 0.05, (N, M)))
    rows = [[(o.Z, i), (o.Z, (i + 1) % N)] for i in range(N)] + [[(o.X, i)] for i in range(N)]
    coef = np.append(-np.ones(N), -0.7 * np.ones(N))
    words = rng.integers(0, 2 ** 63, (count, (N + 63) // 64)).astype(np.uint64)
    if N % 64:
        words[:, -1] &= np.uint64((1 << (N % 64)) - 1)
    fs = rg.FixedSamples(N, words)
    ev = rg.ExpectationValue()
    for f in (ev.gradient, ev.eloc_gradient):
        g, E = f(psi, rg.Operator(*o.table(rows, coef)), fs)
        h, F = f(psi, rg.Operator(*o.table(rows + [[(o.X, 0)]], np.append(coef, 0.0))), fs)
        assert abs(E - F) <= 1e-12 * abs(F)
        assert np.linalg.norm(g - h) <= 1e-5 * np.linalg.norm(h)
