"""Runs of 2D Ising sweeps on bit planes, against the oracle: one word column,
odd numbers of columns, strips of 1 to 8 rows, the couplings' two signs and
none, measurements fused into a run of EMCS, sweeps after it without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.44068679, 0.05, 3.0])
@pytest.mark.parametrize("J", [-1.0, 1.0, 0.0])
@pytest.mark.parametrize("L", [64, 192, 320])
@pytest.mark.parametrize("rows", [1, 2, 4, 8])
def test_bit_planes_match_oracle(orc, rows, L, J, beta, monkeypatch):
    import marqov_b200 as M
    monkeypatch.setenv("MARQOV_B200_SWEEP_CONFIG", f"ising2d_bits<{rows}>")
    cfg = M.Config(seed=78, repid=4, ncluster=0, nmetro=2, resident=False)
    with M.makeCore(M.RegularHypercubic(L, 2), cfg, M.Ising(J), beta) as c:
        c.init()
        s = c.state
        obs, _ = c.emcs(3, ncluster=0, nmetro=2)
        c.metropolis(1)
        assert c.describe().endswith(f"ising2d_bits<{rows}>")
        got, counters = c.state, c.counters
    for sweep in range(7):
        orc.ising2d_sweep(L, J, s, beta, 78, 4, sweep)
        if sweep < 6 and sweep % 2:
            g = s.reshape(L, L).astype(np.int64)
            bonds = int((g * np.roll(g, 1, 0)).sum() + (g * np.roll(g, 1, 1)).sum())
            assert obs[sweep // 2, 0] == J * (2 * bonds) / (2 * L * L)
            assert obs[sweep // 2, 1] == abs(float(g.sum())) / (L * L)
    assert (s == got).all()
    assert counters == (7, 0)


@pytest.mark.parametrize("L,nsweeps", [(1024, 1), (1024, 4), (1024, 5), (2112, 3), (8256, 2), (12352, 3)])
def test_default_route_matches_a_launch_per_sweep(L, nsweeps, monkeypatch):
    """Whatever route a run of sweeps takes by default, its state and observables
    are those of the same sweeps called one by one, clusters between them or not."""
    import marqov_b200 as M

    def go(split):
        cfg = M.Config(seed=9, repid=1, ncluster=1, nmetro=nsweeps)
        with M.makeCore(M.RegularHypercubic(L, 2), cfg, M.Ising(-1.0), 0.44) as c:
            c.init()
            out = []
            for nc in (0, 1):
                if split:
                    for _ in range(2):
                        if nc:
                            c.wolff(nc)
                        for _ in range(nsweeps):
                            c.metropolis(1)
                        out.append(c.measure())
                else:
                    out += list(c.emcs(2, ncluster=nc, nmetro=nsweeps)[0])
            return np.array([list(o)[:2] for o in out]), c.state, c.counters

    a, b = go(False), go(True)
    assert (a[0] == b[0]).all() and (a[1] == b[1]).all() and a[2] == b[2]
