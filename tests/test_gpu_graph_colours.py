"""One-launch sweeps of graphs whose colours are missing on some CTAs or have no
site at all (csr_sweep.cu) against one launch per colour, bit for bit, also
with several handles at work on their own streams.  A wait that is made to run
out (a word that nobody sends, a limit of 200 us) is reported, and the handle
runs on from a state that is set again."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(name):
    import marqov_b200 as M
    if name == "rgg":  # most of its greedy colours are missing on some CTAs
        return M.RandomGeometricGraph2D(16384, 8.0, seed=5)
    sq = M.RegularHypercubic(64, 2).to_csr()
    parity = np.add.outer(np.arange(64), np.arange(64)).ravel() & 1
    classes = {"gap": (0, 3), "long_gap": (7, 1500), "far": (1, 4096)}
    if name in classes:
        return M.CSRLattice(sq.row_ptr, sq.col_idx, None, np.array(classes[name], np.int32)[parity])
    # "halves": two squares side by side, each with colours of its own
    n = sq.n
    rp = np.r_[sq.row_ptr, sq.row_ptr[1:] + sq.row_ptr[-1]].astype(np.int32)
    ci = np.r_[sq.col_idx, sq.col_idx + n].astype(np.int32)
    return M.CSRLattice(rp, ci, None, np.r_[parity, 2 + 2 * parity].astype(np.int32))


def chain(lat, per_colour, repid=0):
    import marqov_b200 as M
    with M.makeCore(lat, M.Config(seed=8, repid=repid, per_colour=per_colour), M.Ising(-1.0, "int8"), 0.4) as c:
        c.init()
        out = [*c.emcs(3, 0, 2)]
        c.metropolis(40)
        return out + [*c.emcs(20, 0, 3), c.state]


@pytest.mark.parametrize("name", ["rgg", "gap", "long_gap", "far", "halves"])
def test_missing_colours(name):
    lat = graph(name)
    for x, y in zip(chain(lat, False), chain(lat, True)):
        assert np.array_equal(x, y)


def test_slices_beyond_the_graphs_size():
    import marqov_b200 as M
    hubs, leaves = 32 * np.arange(1000), 32000 + np.arange(1100)  # a hub per slice of its colour
    deg = np.zeros(33100, int)
    deg[hubs], deg[leaves] = 1100, 1000
    ci = np.r_[np.tile(leaves, 1000), np.tile(hubs, 1100)]
    lat = M.CSRLattice(np.r_[0, np.cumsum(deg)], ci)
    for x, y in zip(chain(lat, False), chain(lat, True)):
        assert np.array_equal(x, y)
    with M.makeCore(lat, M.Config(seed=8), M.Ising(-1.0, "int8"), 0.4) as c:
        c.init()
        before = c.launches
        c.metropolis(5)
        assert c.launches - before == 10  # a launch per colour


@pytest.mark.parametrize("name", ["rgg", "gap"])
@pytest.mark.parametrize("colour,nm,measure", [(2, 1, True), (2, 4, True), (7, 4, True), (3, 8, False)])
def test_wait_that_runs_out(name, colour, nm, measure):
    import marqov_b200 as M
    from marqov_b200 import _lib
    lat = graph(name)
    with M.makeCore(lat, M.Config(seed=8), M.Ising(-1.0, "int8"), 0.4) as c:
        c.init()
        s0 = c.state
        _lib.check(c._lib.mqv_selftest_inject_timeout(c.handle, colour, 200_000))
        with pytest.raises(M.MarqovError) as ei:
            if measure:
                c.emcs(3, 0, nm)
            else:
                c.metropolis(nm)
                c.synchronize()
        assert ei.value.status == _lib.ERR_TIMEOUT
        with pytest.raises(M.MarqovError) as ei:
            c.metropolis(1)
        assert ei.value.status == _lib.ERR_STATE
        c.state = s0
        before = c.counters
        got = [*c.emcs(2, 0, 1), c.state]
    with M.makeCore(lat, M.Config(seed=8, per_colour=True), M.Ising(-1.0, "int8"), 0.4) as c:
        c.state = s0
        c.counters = before
        for x, y in zip(got, [*c.emcs(2, 0, 1), c.state]):
            assert np.array_equal(x, y)


def test_handles_side_by_side():
    lats = [graph("rgg"), graph("halves"), graph("gap")] * 2
    want = [chain(g, True, i) for i, g in enumerate(lats)]
    got = [None] * len(lats)

    def work(i):
        got[i] = chain(lats[i], False, i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(lats))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
