"""The energy gradient of a transverse-field operator (each off-diagonal string one site's own)
at the sizes where its passes can go wrong: remainders of the eight- and 32-sample groups and of
the eight strings of a block, several 32-sample chunks, more spins than a row tile, weights."""
import numpy as np
import pytest

gpu = pytest.mark.gpu


def rbm(N, M, seed):
    rng = np.random.default_rng(seed)
    b = rng.normal(0, 0.1, M) + 1j * rng.normal(0, 0.1, M)
    return b, rng.normal(0, 0.1, (N, M)) + 1j * rng.normal(0, 0.1, (N, M)), rng


def words(up):
    w = np.zeros((len(up), (up.shape[1] + 63) // 64), np.uint64)
    for i in range(up.shape[1]):
        w[:, i // 64] |= up[:, i].astype(np.uint64) << np.uint64(i % 64)
    return w


def field_operator(N, rng):
    """zz bonds and x / y fields with complex coefficients, in a random order."""
    from rbmongpu_gb300 import operators as o
    rows = [[(o.Z, i), (o.Z, (i + 1) % N)] for i in range(N)] + [[(int(rng.integers(1, 3)), i)] for i in range(N - 1)]
    coef = rng.normal(size=len(rows)) + 0.3j * rng.normal(size=len(rows))
    order = rng.permutation(len(rows))
    return [rows[k] for k in order], coef[order]


@gpu
@pytest.mark.parametrize("N,M,count", [(2, 1, 1), (5, 33, 7), (9, 31, 63), (17, 64, 64), (12, 40, 65), (20, 129, 520),
                                       (33, 20, 4097), (65, 70, 300), (6, 300, 130), (10, 500, 66), (8, 32, 16400)])
def test_single_flip_form_equals_the_general_form(N, M, count):
    """A second string on an already flipped site, with coefficient 0, adds zeros to every sum
    and takes the general form.  The sums are the same FP32 sums; a local energy may move by
    its last FP64 bits and then a sample's FP32 coefficient by one rounding, 2^-24."""
    import rbmongpu_gb300 as rg
    b, W, rng = rbm(N, M, N + M)
    rows, coef = field_operator(N, rng)
    site = next(r[0] for r in rows if r[0][0] != 3)
    fs = rg.FixedSamples(N, words(rng.integers(0, 2, (count, N)).astype(bool)))
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W)
    ev = rg.ExpectationValue()
    single = rg.Operator(*rg.operators.table(rows, coef))
    general = rg.Operator(*rg.operators.table(rows + [[site]], np.append(coef, 0.0)))
    for f in (ev.gradient, ev.eloc_gradient):
        g, E = f(psi, single, fs)
        h, F = f(psi, general, fs)
        assert abs(E - F) <= 1e-12 * abs(F)
        assert np.abs(g - h).max() <= 2.0 ** -23 * np.abs(h).max()


@gpu
def test_weights_over_several_chunks():
    """2^17 enumerated states: chunks of 65536, 128 samples a warp, the ensemble's weights."""
    import rbmongpu_gb300 as rg
    N, M = 17, 6
    b, W, rng = rbm(N, M, 4)
    rows, coef = field_operator(N, rng)
    site = next(r[0] for r in rows if r[0][0] != 3)
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W)
    es = rg.ExactSummation(N)
    psi.normalize(es)
    ev = rg.ExpectationValue()
    g, E = ev.gradient(psi, rg.Operator(*rg.operators.table(rows, coef)), es)
    h, F = ev.gradient(psi, rg.Operator(*rg.operators.table(rows + [[site]], np.append(coef, 0.0))), es)
    assert abs(E - F) <= 1e-12 * abs(F)
    assert np.abs(g - h).max() <= 2.0 ** -23 * np.abs(h).max()


def lc(z):
    s = np.where(z.real > 0, 1.0, -1.0)
    u = s * z
    D = 9.19376335670885 + u * (10.2180213465 + u * (7.771429504240965 + u * (3.746646023906276 + u)))
    dD = 10.2180213465 + u * (2 * 7.771429504240965 + u * (3 * 3.746646023906276 + u * 4))
    n = 5.49914721954 - 2.16564366435 * u
    return 0.9003320053750442 * u + n / D, s * (0.9003320053750442 + (-2.16564366435 * D - n * dD) / (D * D))


@gpu
@pytest.mark.parametrize("N,M", [(67, 20), (68, 33), (135, 40), (140, 9)])
def test_row_tiles_against_numpy(N, M):
    """N + 1 = 68, 69, 136 and 141 rows against row tiles of at most 68, in FP64 numpy; FP32
    sums of 40 samples are held to the 1e-5 of the other estimator tests."""
    import rbmongpu_gb300 as rg
    b, W, rng = rbm(N, M, 3 * N)
    count = 40
    up = rng.integers(0, 2, (count, N)).astype(bool)
    s = np.where(up, 1.0, -1.0)
    h = 0.7
    th = b + s @ W
    f, T = lc(th)
    E = -(s * np.roll(s, -1, 1)).sum(1).astype(complex)
    O = np.concatenate([T, (s[:, :, None] * T[:, None, :]).reshape(count, -1)], 1)
    Ek = E[:, None] * O
    for i in range(N):
        fi, Ti = lc(th - 2 * s[:, i:i + 1] * W[i])
        e = -h * np.exp((fi - f).sum(1))
        si = s.copy()
        si[:, i] *= -1
        E = E + e
        Ek = Ek + e[:, None] * np.concatenate([Ti, (si[:, :, None] * Ti[:, None, :]).reshape(count, -1)], 1)
    ref = (E[:, None] * O.conj()).mean(0) + Ek.mean(0).conj() - 2 * E.mean() * O.mean(0).conj()
    g, got = rg.ExpectationValue().gradient(rg.Psi(np.zeros(N), np.zeros(N), b, W),
                                            rg.Operator(*rg.operators.tfim_chain(N, 1.0, h)),
                                            rg.FixedSamples(N, words(up)))
    assert abs(got - E.mean()) < 1e-5 * abs(E.mean())
    assert np.linalg.norm(g[2 * N:] - ref) < 1e-5 * np.linalg.norm(ref)
