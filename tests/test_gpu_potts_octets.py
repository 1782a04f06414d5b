"""Potts sweeps and measurements by octets of an x-line against the per-site
kernels of the same lattice as a graph, bit for bit: the smallest and odd
multiples of 8, two and three dimensions, few states, more than the counted
ones, the most; frozen and free couplings; a batch of uneven members."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(M, L, dim):
    n = L ** dim
    i = np.arange(n)
    nbrs = []
    for d in range(dim):
        x = (i // L ** d) % L
        nbrs += [i + np.where(x == L - 1, -(L - 1), 1) * L ** d, i + np.where(x == 0, L - 1, -1) * L ** d]
    colours = sum((i // L ** d) % L for d in range(dim)) % 2
    return M.CSRLattice(np.arange(0, n * 2 * dim + 1, 2 * dim, dtype=np.int32), np.stack(nbrs, 1).astype(np.int32).reshape(-1),
                        colours=colours.astype(np.int32))


def _run(M, lat, q, beta, k):
    cfg = M.Config(seed=21, repid=k, ncluster=0, nmetro=1, resident=False)
    with M.makeCore(lat, cfg, M.Potts(q, -1.0), beta) as c:
        c.init()
        obs, _ = c.emcs(4, ncluster=0, nmetro=1)
        return np.array(obs), c.state.copy()


@pytest.mark.parametrize("beta", [0.0, 1.0, 1e6])
@pytest.mark.parametrize("q", [2, 3, 8, 9, 64])
@pytest.mark.parametrize("L,dim", [(8, 2), (24, 2), (64, 2), (8, 3), (24, 3)])
def test_octets_match_per_site_kernels(L, dim, q, beta):
    import marqov_b200 as M
    a = _run(M, M.RegularHypercubic(L, dim), q, beta, 3)
    b = _run(M, _graph(M, L, dim), q, beta, 3)
    assert (a[1] == b[1]).all()
    assert (a[0] == b[0]).all()


@pytest.mark.parametrize("sizes", [(8, 40, 64, 200), (8, 12, 64)])  # 12 has no octets: the whole batch goes by sites
def test_batch_of_uneven_members(sizes):
    import marqov_b200 as M
    members = [(M.RegularHypercubic(L, 2), M.Config(seed=21, repid=k, ncluster=0, nmetro=1), M.Potts(3 + k, -1.0), 0.9)
               for k, L in enumerate(sizes)]
    with M.Batch(members) as b:
        b.init()
        obs, _ = b.emcs(4, 0, 1)
        got = [b.member(k).state.copy() for k in range(len(sizes))]
    for k, L in enumerate(sizes):
        o, s = _run(M, _graph(M, L, 2), 3 + k, 0.9, k)
        assert (s == got[k]).all()
        assert (np.array(obs)[:, k] == o).all()
