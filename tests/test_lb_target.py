"""The locally balanced training target against FP64 numpy, for every width of a lane's hidden
units, odd and even numbers of seeds, seeds that wrap around, one to three spin words."""
import numpy as np
import pytest


def lc(z):
    s = np.where(z.real > 0, 1.0, -1.0)
    u = s * z
    D = 9.19376335670885 + u * (10.2180213465 + u * (7.771429504240965 + u * (3.746646023906276 + u)))
    return 0.9003320053750442 * u + (5.49914721954 - 2.16564366435 * u) / D


@pytest.mark.gpu
@pytest.mark.parametrize("N,M,count", [(9, 5, 3), (10, 40, 1), (33, 100, 5), (64, 250, 2), (101, 400, 3), (130, 500, 2)])
def test_against_numpy(N, M, count):
    """Re Delta is a sum of M FP32 differences of values of about one: 2^-24 (M + 64) times a few
    operations a difference, relative on p* and on q."""
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(N)
    b = 0.1 * (rng.normal(size=M) + 1j * rng.normal(size=M))
    W = 0.1 * (rng.normal(size=(N, M)) + 1j * rng.normal(size=(N, M)))
    up = rng.integers(0, 2, (count, N)).astype(bool)
    words = np.zeros((count, (N + 63) // 64), np.uint64)
    for i in range(N):
        words[:, i // 64] |= up[:, i].astype(np.uint64) << np.uint64(i % 64)
    logits = rng.normal(size=(count, N + 8)).astype(np.float32)
    psi = rg.Psi(np.zeros(N), np.zeros(N), b, W)
    got = rg.Proposal(N, seed=1).lb_target(psi, words, logits) * count
    s = np.where(up, 1.0, -1.0)
    th = b + s @ W
    delta = np.zeros((count, N, 8))
    for i in range(N):
        t = th.copy()
        for q in range(8):
            c = (i + q) % N
            t -= 2 * s[:, c:c + 1] * W[c]
            delta[:, i, q] = (lc(t) - lc(th)).real.sum(1)
    p = np.exp(delta - delta.max(axis=(1, 2), keepdims=True))
    p /= p.sum(axis=(1, 2), keepdims=True)
    soft = lambda x: np.exp(x) / np.exp(x).sum(1, keepdims=True)   # noqa: E731
    x = logits.astype(np.float64)
    q = np.concatenate([soft(x[:, :N]), soft(x[:, N:])], 1)
    ps = np.concatenate([p.sum(2), p.sum(1)], 1)
    assert np.all(np.abs(got - (q - ps)) <= 2.0 ** -24 * 16 * (M + 64) * (q + ps))
