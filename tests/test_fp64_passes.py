"""The FP64 passes of the complex RBM at the sizes where their groups can go wrong: angles
from spin-group sums (six spins a group, across word boundaries, above and below the size
where the table is used) and local energies taken eight and 32 strings at a time."""
import numpy as np
import pytest

gpu = pytest.mark.gpu
EPS = 2.0 ** -53


def lc(z):
    s = np.where(z.real > 0, 1.0, -1.0)
    u = s * z
    D = 9.19376335670885 + u * (10.2180213465 + u * (7.771429504240965 + u * (3.746646023906276 + u)))
    return 0.9003320053750442 * u + (5.49914721954 - 2.16564366435 * u) / D - 0.598139


def words(up):
    count, N = up.shape
    w = np.zeros((count, (N + 63) // 64), np.uint64)
    for i in range(N):
        w[:, i // 64] |= up[:, i].astype(np.uint64) << np.uint64(i % 64)
    return w


def rbm(rng, N, M, sigma=0.1):
    b = rng.normal(0, sigma, M) + 1j * rng.normal(0, sigma, M)
    return b, rng.normal(0, sigma, (N, M)) + 1j * rng.normal(0, sigma, (N, M))


@gpu
@pytest.mark.parametrize("N,M,count", [(5, 1, 1), (6, 31, 2048), (7, 33, 2047), (23, 32, 2048), (24, 75, 3),
                                       (64, 30, 40), (65, 64, 5), (70, 33, 9), (127, 20, 4), (130, 576, 2), (256, 7, 3)])
def test_log_psi_against_numpy(N, M, count):
    """Each angle is a sum of N + 1 terms and log psi one of M: a rounding error of at most
    EPS times the terms' magnitudes per addition, 60 operations an activation."""
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(100 * N + M)
    b, W = rbm(rng, N, M)
    W[0] = 0.0
    b[0] = 1j * b[0].imag
    if M == 1:
        W[:] = 1j * W.imag            # Re theta = 0 exactly
    up = rng.integers(0, 2, (count, N)).astype(bool)
    s = np.where(up, 1.0, -1.0)
    f = lc(b + s @ W)
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W)
    got = psi.log_psi_batch(words(up))
    size = np.abs(b).sum() + np.abs(W).sum() + M
    assert np.abs(got - f.sum(1)).max() <= EPS * (N + M + 60) * size


def local_energies(op, lp):
    """E_loc of every basis state from the amplitudes, string by string."""
    coef, types, idx = op
    x = np.arange(len(lp))
    E = np.zeros(len(lp), np.complex128)
    for c, ty, ix in zip(coef, types, idx):
        y, ph = x.copy(), np.full(len(lp), c, np.complex128)
        for t, i in zip(ty, ix):
            if i < 0:
                break
            sgn = np.where((x >> i) & 1, 1.0, -1.0)
            if t == 2:
                ph = ph * (-1j * sgn)
            if t == 3:
                ph = ph * sgn
            if t in (1, 2):
                y = y ^ (1 << i)
        E += ph * np.exp(lp[y] - lp)
    return E


@gpu
@pytest.mark.parametrize("N,M,strings", [(5, 9, 1), (7, 33, 7), (8, 24, 9), (9, 40, 33), (11, 17, 70)])
def test_distance_of_mixed_operators(N, M, strings):
    """HilbertSpaceDistance of random strings of 0 to 3 factors (diagonal, several flips, Y
    phases) against numpy: the terms are formed in FP64, so the squared distance, a difference
    of two numbers near 1, is held to 2^-53 times the operations of a term (about 1e4)."""
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(strings)
    rows = []
    for n in range(strings):
        k = 1 if n == 0 else int(rng.integers(0, 4))
        rows.append([(int(rng.integers(1, 4)) if n else 1, int(i)) for i in rng.choice(N, k, replace=False)])
    coef = 0.1 * (rng.normal(size=strings) + 1j * rng.normal(size=strings))
    op = rg.operators.table(rows, coef)
    b, W = rbm(rng, N, M)
    db, dW = rbm(rng, N, M, 0.05)
    s = np.where((np.arange(1 << N)[:, None] >> np.arange(N)) & 1, 1.0, -1.0)
    lp, lq = lc(b + s @ W).sum(1), lc(b + db + s @ (W + dW)).sum(1)
    w = np.exp(2 * (lp.real - lp.real.max()))
    w /= w.sum()
    E, dl = local_energies(op, lp), lq - lp
    om, pr, nn = np.exp(dl.conj()) * E, np.exp(2 * dl.real), np.abs(E) ** 2
    ref = 1 - abs((w * om).sum()) ** 2 / ((w * nn).sum() * (w * pr).sum())
    z = np.zeros(N)
    d = rg.HilbertSpaceDistance(N, 2 * N + M + N * M)(rg.Psi(z, z, b, W), rg.Psi(z, z, b + db, W + dW),
                                                       rg.Operator(*op), True, rg.ExactSummation(N))
    assert abs(d * d - ref) <= 1e4 * EPS
