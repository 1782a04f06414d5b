"""Labelled clusters of a handle recorded into a CUDA graph: the calls outside the
graph, before and after its replays, and the replays themselves grow the
clusters of a handle that was never captured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replays", [0, 2])
def test_clusters_beside_a_captured_call(replays):
    import marqov_b200 as M
    import torch
    from marqov_b200 import _lib
    lib = _lib.load()

    def make():
        c = M.makeCore(M.RegularHypercubic(256, 2), M.Config(seed=4), M.Ising(-1.0), 0.40)
        c.init()
        c.wolff(2)
        return c

    def at(h, beta, serial):
        h.set_beta(beta)
        h.counters = (h.counters[0], serial)

    with make() as c, make() as want:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        c.set_stream(stream.cuda_stream)
        at(c, 0.46, 7)
        with torch.cuda.graph(graph, stream=stream):
            _lib.check(lib.mqv_wolff(c.handle, 1, None))

        def replay():  # the recorded cluster: its own serial and coupling
            graph.replay()
            torch.cuda.synchronize()
            at(want, 0.46, 7)
            want.wolff(1)
            assert np.array_equal(c.state, want.state)

        for _ in range(replays):
            replay()
        for beta in (0.46, 0.42):
            for h in (c, want):
                at(h, beta, 20)
            assert np.array_equal(c.wolff(3), want.wolff(3))
            assert np.array_equal(c.state, want.state)
            if replays:
                replay()
        del graph
        torch.cuda.synchronize()
        c.set_stream(0)


def test_first_clusters_in_a_captured_call():
    """3D L = 32 is labelled, with scratch that a captured call cannot allocate: it
    stays on the bit planes there."""
    import marqov_b200 as M
    import torch
    from marqov_b200 import _lib
    lib = _lib.load()

    def make(resident):
        c = M.makeCore(M.RegularHypercubic(32, 3), M.Config(seed=4, resident=resident), M.Ising(-1.0), 0.2216546)
        c.init()
        c.emcs(2, 0, 1)
        return c

    with make(None) as c, make(True) as want:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        c.set_stream(stream.cuda_stream)
        with torch.cuda.graph(graph, stream=stream):
            _lib.check(lib.mqv_wolff(c.handle, 1, None))
        graph.replay()
        torch.cuda.synchronize()
        want.wolff(1)
        assert np.array_equal(c.state, want.state)
        assert np.array_equal(c.wolff(3), want.wolff(3))
        assert np.array_equal(c.state, want.state)
        assert "clusters=label " in c.describe()
        del graph
        torch.cuda.synchronize()
        c.set_stream(0)
