"""Ising-type lattices whose bond weights are not just +-1, against the oracle:
neighbourhood sums up to the sum of a site's |weights| index the acceptance
table on every path (one launch on a cluster, launches per colour, one CTA,
batches), with the largest int8 weights, zeros and degrees above what is fetched
ahead."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

WEIGHTS = {"small": np.arange(-3, 4), "two": np.array([-2, 2]), "extreme": np.array([-128, -127, 127]),
           "mixed": np.array([-100, -1, 0, 1, 50])}


def graph(name, which):
    import marqov_b200 as M
    rng = np.random.default_rng(7)
    if name == "rgg":
        g = M.RandomGeometricGraph2D(5000, 12.0, seed=2)
    else:  # hubs of 40 neighbours
        rows = [[] for _ in range(600)]
        for h in range(0, 550, 43):
            for k in range(1, 41):
                rows[h].append(h + k)
                rows[h + k].append(h)
        g = M.CSRLattice(np.r_[0, np.cumsum([len(r) for r in rows])], np.concatenate([np.array(r, int) for r in rows]))
    w = {}
    bonds = [w.setdefault((min(i, j), max(i, j)), int(rng.choice(WEIGHTS[which]))) for i in range(g.n) for j in g.nbrs(0, i)]
    return M.CSRLattice(g.row_ptr, g.col_idx, np.array(bonds, np.int8))


def square(L, dim, which):
    import marqov_b200 as M
    lat = M.RegularRandomBond(L, dim, 0.5, seed=3)
    w = np.random.default_rng(8).choice(WEIGHTS[which], (lat.npoints, dim))
    nbr = lat.to_csr().col_idx.reshape(-1, 2 * dim)
    for d in range(dim):
        lat.bonds[:, 2 * d] = w[:, d]
        lat.bonds[:, 2 * d + 1] = w[nbr[:, 2 * d + 1], d]
    return lat


def oracle_run(orc, lat, s, beta, seed, repid, sweeps):
    csr = lat.to_csr() if hasattr(lat, "to_csr") else lat
    col = csr.colours if csr.colours is not None else csr.greedy_colours()
    order = np.argsort(col, kind="stable")
    g = O.Graph(csr.row_ptr, csr.col_idx, np.r_[0, np.cumsum(np.bincount(col))], order, csr.bonds)
    m = O.OrcModel(kind=O.EA, J=-1.0)
    s, obs = s.copy(), []
    for t in range(sweeps):
        orc.sweep_int8(m, g, s, beta, seed, repid, t)
        obs.append(orc.measure_int8(m, g, s)[:2])
    return s, np.array(obs)


LATTICES = [("rgg", None), ("hubs", None), ("square", (12, 2)), ("square", (8, 3)), ("square", (18, 3))]


@pytest.mark.parametrize("kind,shape", LATTICES)
@pytest.mark.parametrize("which", list(WEIGHTS))
def test_paths_equal_the_oracle(orc, kind, shape, which):
    import marqov_b200 as M
    lat = square(*shape, which) if shape else graph(kind, which)
    beta = 0.6 / np.abs(WEIGHTS[which]).max()
    paths = [dict(), dict(per_colour=True), dict(resident=True), dict(resident=False)]
    want = None
    for path in paths:
        with M.makeCore(lat, M.Config(seed=5, repid=1, **path), M.EdwardsAndersonIsing(-1.0), beta) as c:
            c.init()
            if want is None:
                want = oracle_run(orc, lat, c.state, beta, 5, 1, 6)
            obs, _ = c.emcs(6, 0, 1)
            assert np.array_equal(c.state, want[0]), path
            assert np.array_equal(obs[:, :2], want[1]), path
    with M.Batch([(lat, M.Config(seed=5, repid=1, resident=r), M.EdwardsAndersonIsing(-1.0), beta) for r in (None, True)]) as b:
        b.init()
        obs, _ = b.emcs(6, 0, 1)
        for i in range(2):
            assert np.array_equal(b.member(i).state, want[0])
            assert np.array_equal(obs[:, i, :2], want[1])


def test_weights_beyond_the_table_are_refused():
    import marqov_b200 as M
    leaves = 140_000
    rp = np.r_[0, leaves + np.arange(leaves + 1)]
    ci = np.r_[1 + np.arange(leaves), np.zeros(leaves, int)]
    for w, ok in ((1, True), (127, False)):
        lat = M.CSRLattice(rp, ci, np.full(2 * leaves, w, np.int8))
        if ok:
            M.makeCore(lat, M.Config(seed=1), M.EdwardsAndersonIsing(-1.0), 0.1).close()
        else:
            with pytest.raises(M.MarqovError):
                M.makeCore(lat, M.Config(seed=1), M.EdwardsAndersonIsing(-1.0), 0.1)
