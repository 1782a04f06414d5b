"""Batches of small uneven int8 Ising lattices on the graph path (members that
would otherwise be held as bit planes): breadth first and labelling in bit
tiles grow the clusters of the members' own handles, also between exchanges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def members(dim, sizes, ham, betas):
    import marqov_b200 as M
    return [(M.RegularHypercubic(L, dim), M.Config(seed=3, repid=i, resident=False), ham, b)
            for i, (L, b) in enumerate(zip(sizes, betas))]


@pytest.mark.parametrize("dim,sizes,kind", [(2, (32, 34, 64, 128), "int"), (2, (6, 48, 100, 36), "int8"), (3, (8, 10, 18, 32), "int"),
                                            (2, (64,) * 5, "int8")])
def test_clusters_of_graph_members(dim, sizes, kind):
    import marqov_b200 as M
    beta = 0.44068679 if dim == 2 else 0.2216546
    mem = members(dim, sizes, M.Ising(-1.0, kind), [beta] * len(sizes))
    want = []
    for lat, cfg, ham, b in mem:
        with M.makeCore(lat, cfg, ham, b) as c:
            c.set_wolff("bfs")
            c.init()
            c.emcs(4, 0, 1)
            want.append((*c.emcs(7, 2, 1), c.state))
    for algo in ("bfs", "label"):
        with M.Batch(mem, graph_steps=3) as b:
            b.set_wolff(algo)
            b.init()
            b.emcs(4, 0, 1)
            obs, mc = b.emcs(7, 2, 1)
            assert b.wolff == algo
            for i, (o, m, s) in enumerate(want):
                assert np.array_equal(obs[:, i], o) and np.array_equal(mc[:, i], m) and np.array_equal(b.member(i).state, s)


def test_exchanges_of_graph_members():
    import marqov_b200 as M
    got = []
    for algo in ("bfs", "label"):
        with M.Batch(members(2, (48,) * 8, M.Ising(-1.0), np.linspace(0.40, 0.48, 8))) as b:
            b.set_wolff(algo)
            b.init()
            got.append([*b.tempering(30, 2, 1, 1, seed=3)] + [b.member(i).state for i in range(8)])
    for x, y in zip(*got):
        assert np.array_equal(x, y)
    assert (got[0][1] == 1).any() and (got[0][1] == 0).any()
