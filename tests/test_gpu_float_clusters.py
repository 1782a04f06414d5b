"""Float handles choose labelling or breadth-first growth by the clusters last
reported: the same chain as either one alone, whichever is taken when."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,L,beta", [("heis", 24, 0.8), ("heis", 24, 0.2), ("phi4", 24, 0.45), ("phi4", 20, 0.3)])
def test_auto_matches_breadth_first(model, L, beta):
    import marqov_b200 as M
    got = []
    for algo in ("bfs", "auto"):
        ham = M.Phi4(beta, 1.1) if model == "phi4" else M.Heisenberg(-1.0, "smallcap", -0.9697)
        with M.makeCore(M.RegularHypercubic(L, 3), M.Config(seed=4, repid=1, ncluster=1, nmetro=3), ham, beta) as c:
            c.set_wolff(algo)
            c.init()
            obs, mc, kinds = [], [], set()
            for _ in range(12):
                o, m = c.emcs(4, 1, 3)
                obs += list(o)
                mc += list(m)
                kinds.add("clusters=label" in c.describe())
            sizes = c.wolff(5)
            got.append((np.array(mc), sizes, c.state, np.array(obs)))
        if algo == "auto":
            assert (True in kinds) == (max(mc) > 1500)  # grown past the line, or never near it
    for x, y in zip(got[0][:3], got[1][:3]):
        assert (x == y).all()
    np.testing.assert_allclose(got[0][3], got[1][3], rtol=1e-12, atol=1e-12)  # atomic sums differ in order only
