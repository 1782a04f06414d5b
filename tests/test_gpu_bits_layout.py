"""States and bond signs taken into bit planes and back by wide loads (lines of
a multiple of 8 sites, split rows) against the launch-per-step path: last
words of 8, 16, 24 and 32 sites, one and two words per thread, with bonds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(lat, ham, beta, resident, nc):
    import marqov_b200 as M
    with M.makeCore(lat, M.Config(seed=31, repid=2, resident=resident), ham, beta) as c:
        c.init()
        a = c.emcs(1, nc, 1)
        b = c.emcs(3, nc, 1)
        return [a[0], b[0], c.state]


@pytest.mark.parametrize("dim,L", [(2, 8), (2, 16), (2, 40), (2, 56), (2, 72), (2, 104), (2, 168), (3, 8)])
def test_lines_of_octets(dim, L):
    import marqov_b200 as M
    lat = M.RegularHypercubic(L, dim)
    for x, y in zip(_chain(lat, M.Ising(-1.0), 0.3, None, 1), _chain(lat, M.Ising(-1.0), 0.3, False, 1)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("dim,L", [(2, 8), (2, 40), (2, 64), (3, 8), (3, 24)])
def test_bonds(dim, L):
    import marqov_b200 as M
    lat = M.RegularRandomBond(L, dim, 0.5, seed=3)
    ham = M.EdwardsAndersonIsing(-1.0)
    for x, y in zip(_chain(lat, ham, 0.9, None, 0), _chain(lat, ham, 0.9, False, 0)):
        assert np.array_equal(x, y)
