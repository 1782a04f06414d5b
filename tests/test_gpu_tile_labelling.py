"""Clusters labelled in bit tiles against breadth-first growth, on the GPU:
single handles and batches, sizes below, at and beyond the tiles' edges
(words of 32 sites, 64 and 128 rows, 8 x 8 and 8 x 16 units in 3D), the four
launch shapes (by the number of units), int8 and float models."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA = 0.44068679


def models():
    import marqov_b200 as M
    return {"ising": (M.Ising(-1.0), BETA), "embed": (M.Ising(-1.0, "int8"), BETA), "potts": (M.Potts(3, -1.0), 1.05),
            "ising3": (M.Ising(-1.0), 0.23), "heis": (M.Heisenberg(-1.0), 0.9), "phi4": (M.Phi4(0.4, 1.1), 0.4)}


CASES = [("ising", 2, L) for L in (4, 30, 32, 34, 64, 66, 128, 130)] + [("embed", 2, 48), ("potts", 2, 36), ("potts", 2, 96)] \
    + [("ising3", 3, L) for L in (4, 8, 10, 18, 34)] + [("heis", 3, 6), ("heis", 3, 18), ("phi4", 3, 16), ("phi4", 3, 34), ("phi4", 2, 40)]


@pytest.mark.parametrize("model,dim,L", CASES)
def test_single_handle(model, dim, L):
    import marqov_b200 as M
    ham, beta = models()[model]
    got = []
    for algo in ("bfs", "label"):
        with M.makeCore(M.RegularHypercubic(L, dim), M.Config(seed=9, repid=2, resident=False), ham, beta) as c:
            c.set_wolff(algo)
            c.init()
            a = c.wolff(4)
            c.metropolis(8)
            b = c.wolff(8)
            obs, mc = c.emcs(3, 2, 1)
            got.append((a, b, mc, c.state))
    for x, y in zip(*got):
        assert (x == y).all()


@pytest.mark.parametrize("model,dim,sizes", [("ising", 2, (32, 34, 64, 128)), ("potts", 2, (64, 256, 512, 512, 512, 512)),
                                             ("ising", 2, (1024,)), ("ising", 2, (1024,) * 4), ("ising", 2, (2048, 2048)), ("phi4", 3, (6, 16, 20)), ("heis", 3, (40, 40, 64))])
def test_batch(model, dim, sizes):
    import marqov_b200 as M
    ham, beta = models()[model]
    got = []
    for algo in ("bfs", "label"):
        with M.Batch([(M.RegularHypercubic(L, dim), M.Config(seed=3, repid=i), ham, beta) for i, L in enumerate(sizes)],
                     graph_steps=3) as b:
            b.set_wolff(algo)
            b.init()
            b.emcs(4, 0, 1)
            obs, mc = b.emcs(7, 2, 1)
            got.append((obs, mc, [b.member(i).state for i in range(len(sizes))]))
    assert (got[0][1] == got[1][1]).all()
    assert np.allclose(got[0][0], got[1][0], rtol=1e-12, atol=1e-13)  # float sums differ in order only
    for x, y in zip(got[0][2], got[1][2]):
        assert (x == y).all()
