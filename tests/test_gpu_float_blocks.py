"""Float stencil sweeps by blocks of a colour (one or two sites per thread, the
decision screened in FP32) against the per-site sweep of the same lattice as a
graph, which computes every cut exactly: the same states, bit for bit, at
couplings from none to ones that freeze the lattice, on ragged sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(M, L, dim):
    lat = M.RegularHypercubic(L, dim)
    n = L ** dim
    i = np.arange(n)
    nbrs = []
    for d in range(dim):
        x = (i // L ** d) % L
        nbrs += [i + np.where(x == L - 1, -(L - 1), 1) * L ** d, i + np.where(x == 0, L - 1, -1) * L ** d]
    col = np.stack(nbrs, 1).astype(np.int32)
    colours = sum((i // L ** d) % L for d in range(dim)) % 2
    return lat, M.CSRLattice(np.arange(0, n * 2 * dim + 1, 2 * dim, dtype=np.int32), col.reshape(-1),
                             colours=colours.astype(np.int32))


@pytest.mark.parametrize("beta", [0.0, 0.37, 4.0, 1e9])
@pytest.mark.parametrize("L,dim", [(6, 3), (10, 2), (22, 3)])
@pytest.mark.parametrize("model", ["phi4", "smallcap", "fresh", "xxz"])
def test_blocks_match_the_exact_decision(model, L, dim, beta):
    import marqov_b200 as M
    ham = {"phi4": lambda: M.Phi4(max(beta, 0.1), 1.1), "smallcap": lambda: M.Heisenberg(-1.0, "smallcap", -0.9697),
           "fresh": lambda: M.Heisenberg(-1.0, "fresh"), "xxz": lambda: M.XXZAntiferro(0.8, 0.2, "smallcap", -0.5)}[model]
    out = []
    for lat in _graph(M, L, dim):
        with M.makeCore(lat, M.Config(seed=5, repid=2, ncluster=0, nmetro=1), ham(), beta) as c:
            c.init()
            c.metropolis(6)
            out.append((c.state.copy(), c.measure()))
    assert (out[0][0] == out[1][0]).all()
    # the energy's terms are added in another order: a few 2^-53 of their sum of magnitudes (O(1) per site)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12, atol=1e-12)


def test_two_sites_per_thread_match_one():
    """Five chains of 50^3 together fill the chip (two sites per thread); alone they do not."""
    import marqov_b200 as M

    def member(i):
        return M.RegularHypercubic(50, 3), M.Config(seed=3, repid=i, ncluster=0, nmetro=1), M.Phi4(0.37 + 0.01 * i, 1.1)

    with M.Batch([(*member(i), 0.37 + 0.01 * i) for i in range(5)]) as b:
        b.init()
        b.emcs(3, 0, 1)
        got = [b.member(i).state.copy() for i in range(5)]
    for i in range(5):
        lat, cfg, ham = member(i)
        with M.makeCore(lat, cfg, ham, 0.37 + 0.01 * i) as c:
            c.init()
            c.metropolis(3)
            assert (c.state == got[i]).all()
