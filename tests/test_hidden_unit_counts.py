"""Each compiled number of hidden units per lane at the edges of its range: a network gives the
same walkers, local energies and gradients as with further units of weight zero, which take it to
the next number (their terms are exact zeros and the order of the sums is the same)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def networks(N, M, more):
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(M)
    b = rng.normal(0, 0.1, M) + 1j * rng.normal(0, 0.1, M)
    W = rng.normal(0, 0.1, (N, M)) + 1j * rng.normal(0, 0.1, (N, M))
    z = np.zeros(N)
    return (rg.Psi(z, z, b, W, 1.0, False, True),
            rg.Psi(z, z, np.append(b, np.zeros(more - M)), np.append(W, np.zeros((N, more - M)), axis=1), 1.0, False, True))


@pytest.mark.parametrize("M, more", [(65, 128), (96, 97), (97, 160), (129, 192), (160, 161), (161, 193), (192, 256),
                                     (257, 416), (320, 321)])
@pytest.mark.parametrize("total_z", [False, True])
def test_zero_units_change_nothing(M, more, total_z):
    import rbmongpu_gb300 as rg
    N = 12
    op = rg.Operator(*(rg.operators.heisenberg_chain(N) if total_z else rg.operators.tfim_chain(N, 1.0, 0.8)))
    out = []
    for psi in networks(N, M, more):
        mc = rg.MonteCarloLoop(66, 1, 3, 33, seed=7)
        if total_z:
            mc.set_total_z_symmetry(0)
        spins, _, eloc = mc.samples(psi, op)
        g, E = rg.ExpectationValue().gradient(psi, op, rg.FixedSamples(N, spins))
        batch = rg.Batch([(psi, op, 5, 3)])
        batch.run(2, 1)
        e, h, _ = batch.result(0)
        grads = [np.concatenate([v[2 * N:2 * N + M], v[2 * N + psi.M:].reshape(N, psi.M)[:, :M].ravel()]) for v in (g, h)]
        out.append([spins, eloc, E, e, batch.spins(0)] + grads)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_networks_of_one_range_still_pair():
    """The energy difference of two networks of 90 and 120 units (three and four per lane) is that
    with both at 120; 90 and 150 stay refused.  The zero units' log psi, f(0) = 2e-8 each, and the
    FP32 log psi leave 1e-5."""
    import rbmongpu_gb300 as rg
    N = 10
    op = rg.Operator(*rg.operators.tfim_chain(N, 1.0, 0.8))
    a, wide = networks(N, 90, 120)
    b, _ = networks(N, 120, 121)
    ev, ens = rg.ExpectationValue(), rg.ExactSummation(N)
    got, ref = (np.asarray(ev.difference(x, b, [op], ens)) for x in (a, wide))
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    far, _ = networks(N, 150, 151)
    with pytest.raises(Exception):
        ev.difference(a, far, [op], ens)
