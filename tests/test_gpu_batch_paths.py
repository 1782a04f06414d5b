"""Where a batch's Ising-type members run: as bit planes, one CTA each, or by
launches where few large ones would leave the chip idle and the batch has run a
while (256 EMCS).  The same chain either way, also in batches that change between runs with and without clusters, in
mixed batches and between exchanges; and single handles whose clusters are
labelled by launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA = {2: 0.44068679, 3: 0.2216546}


def ising(dim, sizes, **cfg):
    import marqov_b200 as M
    return [(M.RegularHypercubic(L, dim), M.Config(seed=6, repid=i, **cfg), M.Ising(-1.0), BETA[dim]) for i, L in enumerate(sizes)]


def glasses(L, n, **cfg):
    import marqov_b200 as M
    return [(M.RegularRandomBond(L, 3, 0.5, seed=i), M.Config(seed=6, repid=i, **cfg), M.EdwardsAndersonIsing(-1.0), 0.9)
            for i in range(n)]


def mixed(**cfg):
    import marqov_b200 as M
    return ising(2, (160, 32, 180, 174, 200), **cfg) + [(M.RegularHypercubic(24, 2), M.Config(seed=2, repid=9), M.Potts(3, -1.0), 1.0)]


def run(members, clusters):
    import marqov_b200 as M
    with M.Batch(members, graph_steps=3) as b:
        b.init()
        out, took = [], []
        for nc, nm, n in ((0, 2, 5), (1, 1, 245), (0, 1, 4), (2, 1, 5), (0, 1, 3)):
            before = b.launches
            out += [*b.emcs(n, nc if clusters else 0, nm)]
            took.append((b.launches - before) / n)
        return out + [b.member(i).state for i in range(len(members))], took


@pytest.mark.parametrize("make,clusters", [(lambda **c: ising(2, (160, 160), **c), True), (lambda **c: ising(2, (174,) * 28, **c), True),
                                           (lambda **c: ising(3, (32, 28, 30), **c), True), (mixed, True),
                                           (lambda **c: glasses(40, 3, **c), False), (lambda **c: glasses(36, 8, **c), False)])
def test_same_chain_on_either_path(make, clusters):
    got, _ = run(make(), clusters)
    want, _ = run(make(resident=False), clusters)
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("make,clusters,on_launches", [
    (lambda **c: ising(2, (128, 128), **c), True, [False] * 5),
    (lambda **c: ising(2, (160, 160), **c), True, [False, False, False, True, False]),
    (lambda **c: ising(2, (160,) * 24, **c), True, [False] * 5),
    (lambda **c: ising(2, (178, 178), **c), True, [False, True, False, True, False]),
    (lambda **c: ising(2, (160, 160), resident=True, **c), True, [False] * 5),
    (lambda **c: ising(2, (160, 160, 32), **c), True, [False, False, False, True, False]),
    (lambda **c: glasses(40, 3, **c), False, [False] * 3 + [True] * 2), (lambda **c: glasses(40, 12, **c), False, [False] * 5)])
def test_path_taken(make, clusters, on_launches):
    _, took = run(make(), clusters)
    # bit planes: a launch or two per call; launches: several per EMCS
    assert [t > 2 for t in took] == on_launches


def test_exchanges():
    import marqov_b200 as M
    got = []
    for resident in (None, False):
        ladder = [(lat, M.Config(seed=1, repid=i, resident=resident), h, b)
                  for i, ((lat, _, h, _), b) in enumerate(zip(ising(2, (160,) * 6), np.linspace(0.43, 0.45, 6)))]
        with M.Batch(ladder) as b:
            b.init()
            got.append([*b.tempering(125, 2, 1, 1, seed=3), *b.tempering(6, 2, 1, 1, seed=8), *b.tempering(6, 1, 0, 2, seed=4), *b.tempering(4, 1, 1, 1, seed=5)]
                       + [b.member(i).state for i in range(6)])
    for x, y in zip(*got):
        assert np.array_equal(x, y)


def test_handle_whose_clusters_are_labelled():
    import marqov_b200 as M
    got = []
    for resident, algo in ((None, "auto"), (None, "bfs"), (True, "auto"), (False, "auto")):
        (lat, cfg, ham, beta), = ising(3, (32,), resident=resident)
        with M.makeCore(lat, cfg, ham, beta) as c:
            c.set_wolff(algo)
            where = "label-smem" if resident or algo == "bfs" else "label"
            assert f"clusters={where} " in c.describe()
            assert ("path=resident-smem" in c.describe()) == (resident is not False)
            c.init()
            got.append([*c.emcs(4, 0, 2), *c.emcs(4, 2, 1), c.wolff(3), *c.emcs(3, 0, 1), c.state])
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("algo", ["bfs", "label"])
def test_mixed_batch_by_either_algorithm(algo):
    # the lattices of 160 and 174 stay on the bit planes, beside launches that
    # grow the clusters of the others
    import marqov_b200 as M
    got = []
    for resident in (None, False):
        with M.Batch(mixed(resident=resident), graph_steps=2) as b:
            b.set_wolff(algo)
            b.init()
            got.append([*b.emcs(7, 2, 1), *b.emcs(40, 3, 1), *b.emcs(250, 1, 1)] + [b.member(i).state for i in range(6)])
    for x, y in zip(*got):
        assert np.array_equal(x, y)
