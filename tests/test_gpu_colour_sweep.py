"""The colour kernels of the 2D Ising sweep (one launch per colour, in place),
forced one at a time against the oracle: one word column (L = 64, every edge
neighbour is the row itself), an odd number of columns, the couplings' two
signs, measurements fused into the sweep, and a batch of sweeps without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.44068679, 0.05, 3.0])
@pytest.mark.parametrize("J", [-1.0, 1.0])
@pytest.mark.parametrize("L", [64, 192, 320])
@pytest.mark.parametrize("rows", [1, 2, 4])
def test_colour_kernel_matches_oracle(orc, rows, L, J, beta, monkeypatch):
    import marqov_b200 as M
    monkeypatch.setenv("MARQOV_B200_SWEEP_CONFIG", f"ising2d_colour<{rows}>")
    cfg = M.Config(seed=77, repid=5, ncluster=0, nmetro=1, resident=False)
    with M.makeCore(M.RegularHypercubic(L, 2), cfg, M.Ising(J), beta) as c:
        c.init()
        s = c.state
        obs, _ = c.emcs(3, ncluster=0, nmetro=1)
        c.metropolis(2)
        assert c.describe().endswith(f"ising2d_colour<{rows}>")
        got, counters = c.state, c.counters
    for sweep in range(5):
        orc.ising2d_sweep(L, J, s, beta, 77, 5, sweep)
        if sweep < 3:
            g = s.reshape(L, L).astype(np.int64)
            bonds = int((g * np.roll(g, 1, 0)).sum() + (g * np.roll(g, 1, 1)).sum())
            assert obs[sweep, 0] == J * (2 * bonds) / (2 * L * L)
            assert obs[sweep, 1] == abs(float(g.sum())) / (L * L)
    assert (s == got).all()
    assert counters == (5, 0)
