"""The bit-plane path of small Ising-type lattices (bits_emcs.cu) against the
launch-per-step path, bit for bit: sizes whose x-lines fill words, straddle
them or leave most of one empty (4 .. 180), 2D and 3D, ferro- and
antiferromagnetic couplings, +-1 bonds, high and low temperatures (every class
accepted, none), several clusters and sweeps per EMCS, batches and exchanges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(lat, ham, beta, resident, nc, nm, n=5):
    import marqov_b200 as M
    with M.makeCore(lat, M.Config(seed=21, repid=4, resident=resident), ham, beta) as c:
        c.init()
        out = [*c.emcs(n, nc, nm)]
        if nc:
            out.append(c.wolff(3))
        out += [*c.emcs(2, 0, 1), c.state, np.array(c.counters)]
        return out


def same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("dim,L", [(2, L) for L in (4, 6, 30, 32, 34, 48, 62, 64, 66, 96, 128, 180)]
                         + [(3, L) for L in (4, 6, 10, 16, 20, 24, 32)])
@pytest.mark.parametrize("nc,nm", [(0, 2), (1, 1), (2, 0)])
def test_ising(dim, L, nc, nm):
    import marqov_b200 as M
    beta = 0.44068679 if dim == 2 else 0.2216546
    lat = M.RegularHypercubic(L, dim)
    same(chain(lat, M.Ising(-1.0), beta, None, nc, nm), chain(lat, M.Ising(-1.0), beta, False, nc, nm))


@pytest.mark.parametrize("dim,L", [(2, 36), (3, 12)])
@pytest.mark.parametrize("J,beta", [(1.0, 0.4), (-1.0, 0.0), (-1.0, 8.0), (-0.3, 1.1), (1.0, 40.0)])
def test_couplings(dim, L, J, beta):
    import marqov_b200 as M
    lat = M.RegularHypercubic(L, dim)
    same(chain(lat, M.Ising(J), beta, None, 0, 2), chain(lat, M.Ising(J), beta, False, 0, 2))
    if J < 0:
        h = M.Ising(J, "int8")
        same(chain(lat, h, beta, None, 1, 1), chain(lat, h, beta, False, 1, 1))


@pytest.mark.parametrize("dim,L", [(2, 18), (2, 64), (3, 8), (3, 18), (3, 32)])
def test_spin_glass(dim, L):
    import marqov_b200 as M
    lat = M.RegularRandomBond(L, dim, 0.5, seed=3)
    same(chain(lat, M.EdwardsAndersonIsing(-1.0), 0.9, None, 0, 2), chain(lat, M.EdwardsAndersonIsing(-1.0), 0.9, False, 0, 2))
    same(chain(lat, M.Ising(-1.0), 0.4, None, 1, 1), chain(lat, M.Ising(-1.0), 0.4, False, 1, 1))


def test_bonds_other_than_unit_stay_on_the_per_site_path():
    import marqov_b200 as M
    lat = M.RegularRandomBond(8, 3, 0.5, seed=3)
    lat.bonds = (2 * lat.bonds).astype(np.int8)
    same(chain(lat, M.EdwardsAndersonIsing(-1.0), 0.4, None, 0, 1), chain(lat, M.EdwardsAndersonIsing(-1.0), 0.4, False, 0, 1))


def members(resident, glass=False):
    import marqov_b200 as M
    cfg = [M.Config(seed=5, repid=i, resident=resident) for i in range(6)]
    if glass:
        return [(M.RegularRandomBond(L, 3, 0.5, seed=i), c, M.EdwardsAndersonIsing(-1.0), 0.9)
                for i, (L, c) in enumerate(zip((8, 16, 10, 32, 40, 16), cfg))]
    return [(M.RegularHypercubic(L, 2), c, M.Ising(-1.0), 0.43) for L, c in zip((64, 32, 128, 48, 64, 300), cfg)]


@pytest.mark.parametrize("glass", [False, True])
def test_batch(glass):
    import marqov_b200 as M
    got = []
    for resident in (None, False):
        with M.Batch(members(resident, glass), graph_steps=3) as b:
            b.init()
            nc = 0 if glass else 2
            got.append([*b.emcs(9, nc, 2), *b.emcs(300 if glass else 70, nc, 1)] + [b.member(i).state for i in range(6)])
    same(*got)


def test_tempering():
    import marqov_b200 as M
    got = []
    for resident in (None, False):
        ladder = [(M.RegularHypercubic(32, 2), M.Config(seed=1, repid=i, resident=resident), M.Ising(-1.0), b)
                  for i, b in enumerate(np.linspace(0.40, 0.48, 8))]
        with M.Batch(ladder) as b:
            b.init()
            got.append([*b.tempering(40, 2, 1, 1, seed=3), *b.tempering(3, 1, 0, 2, seed=4)]
                       + [b.member(i).state for i in range(8)])
    same(*got)
    assert (got[0][1] == 1).any() and (got[0][1] == 0).any()
