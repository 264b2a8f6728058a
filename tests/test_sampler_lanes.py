"""The Metropolis sampler puts a walker on a whole warp or on a group of lanes, by the number of
walkers: walker w's chain is the same either way, at every number of hidden units per lane, in a
magnetisation sector, and over several spin words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def psi(N, M):
    import rbmongpu_gb300 as rg
    rng = np.random.default_rng(N + M)
    return rg.Psi(np.zeros(N), np.zeros(N), rng.normal(0, 0.1, M) + 1j * rng.normal(0, 0.1, M),
                  rng.normal(0, 0.1, (N, M)) + 1j * rng.normal(0, 0.1, (N, M)), 1.0, False, True)


def run(p, walkers, sector=None):
    import rbmongpu_gb300 as rg
    mc = rg.MonteCarloLoop(2 * walkers, 1, 2, walkers, seed=21)
    if sector is not None:
        mc.set_total_z_symmetry(sector)
    spins, _, _ = mc.samples(p, rg.Operator(*rg.operators.tfim_chain(p.N, 1.0, 1.0)), log_psi=False)
    return spins.reshape(2, walkers, -1)[:, :33]


# walkers: below and above each limit of the rule (33 on whole warps; 1217, 1537 and 609 in groups
# below 256 units, from there on 1537 and 6145 with whole warps between)
@pytest.mark.parametrize("N, M, walkers", [(9, 20, (33, 1216, 1217)), (12, 64, (33, 1536, 1537)), (10, 80, (33, 608, 609)),
                                           (70, 128, (33, 1537)), (11, 150, (33, 1537)), (13, 190, (33, 1537)),
                                           (140, 250, (33, 1537, 3583, 3584)), (12, 320, (33, 1537, 6144, 6145)),
                                           (65, 400, (33, 1537, 3584)), (200, 40, (33, 1537)), (16, 576, (33, 2000))])
def test_a_walkers_chain_does_not_depend_on_its_lanes(N, M, walkers):
    p = psi(N, M)
    first = run(p, walkers[0])
    assert len(np.unique(first, axis=1)) > 0 and (first[0] != first[1]).any()
    for w in walkers[1:]:
        np.testing.assert_array_equal(run(p, w), first)


@pytest.mark.parametrize("N, M, sector, many", [(8, 20, 0, 1217), (36, 75, 0, 609), (21, 30, 19, 1217), (64, 100, -60, 1537),
                                                (12, 64, 12, 1537), (10, 300, 2, 1537)])
def test_the_same_in_a_magnetisation_sector(N, M, sector, many):
    """Sectors with one or two spins the other way need many draws for a flip's partner: more than
    the group's lanes test at once.  (12, 12): no partner but the site itself."""
    p = psi(N, M)
    few = run(p, 33, sector)
    up = sum(np.bitwise_count(few[..., k]).astype(int) for k in range(few.shape[-1]))
    assert (2 * up - N == sector).all()
    np.testing.assert_array_equal(run(p, many, sector), few)
