"""Sweeps of Ising-type models on graphs in one launch (csr_sweep.cu) against
one launch per colour, bit for bit: graphs of one and of several CTAs, a last
word that is partly empty, one colour and many, degrees above what is fetched
ahead, isolated sites, integer bond weights, both signs of the coupling, and
runs that mix sweeps, clusters, measurements and samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def star_forest(n, hub):
    """Hubs of degree `hub` with leaves, and some sites without neighbours."""
    rows = [[] for _ in range(n)]
    for h in range(0, n - hub - 1, hub + 3):
        for k in range(1, hub + 1):
            rows[h].append(h + k)
            rows[h + k].append(h)
    return rows


def csr(rows, bonds=None, colours=None):
    import marqov_b200 as M
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    return M.CSRLattice(rp, np.array([j for r in rows for j in r], np.int32), bonds, colours)


def graphs():
    import marqov_b200 as M
    g = M.RandomGeometricGraph2D(5000, 12.0, seed=2)
    key = {}
    rng = np.random.default_rng(4)
    w = np.array([key.setdefault((min(i, j), max(i, j)), int(rng.integers(-3, 4)))
                  for i in range(g.n) for j in g.nbrs(0, i)], np.int8)
    weighted = M.CSRLattice(g.row_ptr, g.col_idx, w)
    complete = csr([[j for j in range(40) if j != i] for i in range(40)])
    return {"rgg_77": M.RandomGeometricGraph2D(77, 6.0, seed=1), "rgg_1024": M.RandomGeometricGraph2D(1024, 8.0, seed=1),
            "rgg_1031": M.RandomGeometricGraph2D(1031, 8.0, seed=1), "rgg_20011": M.RandomGeometricGraph2D(20011, 8.0, seed=3),
            "weighted": weighted, "square": M.RegularHypercubic(64, 2).to_csr(), "stars": csr(star_forest(3001, 40)),
            "complete": complete, "isolated": csr([[] for _ in range(70)])}


def chain(lat, ham, beta, per_colour):
    import marqov_b200 as M
    with M.makeCore(lat, M.Config(seed=8, repid=3, per_colour=per_colour), ham, beta) as c:
        c.init()
        out = [*c.emcs(3, 0, 2)]
        c.metropolis(3)
        out += [*c.emcs(2, 0, 0), *c.emcs(4, 0, 1), c.state, np.array(c.counters)]
        if ham.wolff:
            out += [c.wolff(3), *c.emcs(3, 1, 2), np.array(c.measure()), c.state]
        return out


@pytest.mark.parametrize("name", ["rgg_77", "rgg_1024", "rgg_1031", "rgg_20011", "weighted", "square", "stars", "complete",
                                  "isolated"])
@pytest.mark.parametrize("J,beta", [(-1.0, 0.5), (1.0, 0.3), (-1.0, 0.0)])
def test_one_launch_equals_launch_per_colour(name, J, beta):
    import marqov_b200 as M
    lat = graphs()[name]
    ham = M.EdwardsAndersonIsing(J) if name == "weighted" else M.Ising(J, "int8")
    if J > 0:
        ham.wolff = False
    for x, y in zip(chain(lat, ham, beta, False), chain(lat, ham, beta, True)):
        assert np.array_equal(x, y)


def test_many_sites():
    import marqov_b200 as M
    lat = M.RandomGeometricGraph2D(200003, 8.0, seed=6)
    a, b = (chain(lat, M.Ising(-1.0, "int8"), 0.5, p) for p in (False, True))
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
