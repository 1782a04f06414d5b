"""The description of a handle names the paths its runs take: clusters and sweeps
of one lattice may differ where clusters do not fit a CTA's shared memory."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,clusters", [(64, "label-smem"), (174, "label-smem"), (176, "bfs"), (180, "bfs"), (182, "label")])
def test_paths_of_2d_lattices(L, clusters):
    import marqov_b200 as M
    with M.makeCore(M.RegularHypercubic(L, 2), M.Config(seed=1), M.Ising(-1.0), 0.44) as c:
        words = dict(w.split("=", 1) for w in c.describe().split())
        assert words["clusters"] == clusters
        assert (words["path"] == "resident-smem") == (L <= 180)
        c.init()
        before = c.launches
        c.wolff(3)
        # resident: one launch for all three; else several per cluster
        assert (c.launches - before == 1) == (clusters == "label-smem")
