"""Clusters on a device whose free memory holds the breadth-first queues but not
the scratch of labelling in bit tiles: the calls run, on the same clusters."""
import contextlib
import ctypes as C
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def kernels_loaded():
    """A kernel's first launch loads its code, which takes memory of its own."""
    import marqov_b200 as M
    mem = [(M.RegularHypercubic(64, 2), M.Config(seed=5, resident=False), M.Ising(-1.0), 0.2)]
    with M.makeCore(*mem[0]) as c, M.Batch(mem) as b:
        for h in (c, b):
            h.set_wolff("bfs")
            h.init()
            h.emcs(9, 2, 1)


@contextlib.contextmanager
def free_memory(nbytes):
    """All device memory but `nbytes` taken, down to the allocator's 2 MB."""
    import torch
    gc.collect()  # handles of other tests that still wait for it
    torch.cuda.empty_cache()
    rt = C.CDLL("libcudart.so.12")  # torch's, already loaded
    taken = []

    def take(size):
        p = C.c_void_p()
        if rt.cudaMalloc(C.byref(p), C.c_size_t(size)):
            rt.cudaGetLastError()
            return False
        taken.append(p)
        return True

    assert take(nbytes)
    size = torch.cuda.mem_get_info()[0]
    while size >= 2 << 20:
        if not take(size):
            size //= 2
    rt.cudaFree(taken.pop(0))
    try:
        yield
    finally:
        for p in taken:
            rt.cudaFree(p)


def members(n, L):
    import marqov_b200 as M
    return [(M.RegularHypercubic(L, 2), M.Config(seed=5, repid=i), M.Ising(-1.0), 0.2) for i in range(n)]


@pytest.mark.parametrize("algo", ["auto", "label"])
def test_handle(algo):
    import marqov_b200 as M
    (lat, cfg, ham, beta), = members(1, 4096)
    got = []
    for limit in (True, False):
        with M.makeCore(lat, cfg, ham, beta) as c:
            c.set_wolff(algo)
            c.init()
            c.emcs(1, 0, 1)
            # queue and bitmap 66 MiB, tiles 102 MiB
            with free_memory(80 << 20) if limit else contextlib.nullcontext():
                got.append([c.wolff(4), *c.emcs(2, 2, 1), c.state])
                assert ("clusters=bfs" in c.describe()) == limit
            if limit:
                c.set_wolff("label")  # asked again, there is room
                c.wolff(1)
                assert "clusters=label" in c.describe()
    for x, y in zip(*got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("algo", ["auto", "label"])
def test_batch(algo):
    import marqov_b200 as M
    got = []
    for limit in (True, False):
        with M.Batch(members(4, 2048)) as b:
            b.set_wolff(algo)
            b.init()
            b.emcs(2, 0, 1)
            # queues and bitmaps 66 MiB, tiles 102 MiB
            with free_memory(84 << 20) if limit else contextlib.nullcontext():
                got.append([*b.emcs(6, 2, 1)] + [b.member(i).state for i in range(4)])
                if limit:
                    assert b.wolff == "bfs"
    for x, y in zip(*got):
        assert np.array_equal(x, y)


def test_queue_without_bitmap():
    """Room for the breadth-first queue and none for its bitmap: refused as often
    as it is asked for, then run when there is room."""
    import marqov_b200 as M
    (lat, cfg, ham, beta), = members(1, 4096)
    got = []
    for limit in (True, False):
        with M.makeCore(lat, cfg, ham, beta) as c:
            c.set_wolff("bfs")
            c.init()
            c.emcs(1, 0, 1)
            if limit:
                with free_memory(64 << 20):
                    for _ in range(2):
                        with pytest.raises(M.MarqovError, match="memory"):
                            c.wolff(1)
            got.append([c.wolff(3), c.state])
    for x, y in zip(*got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("algo", ["auto", "label", "bfs"])
def test_few_large_members_stay_on_bit_planes(algo):
    import marqov_b200 as M
    got = []
    for limit in (True, False):
        with M.Batch(members(20, 174)) as b:
            b.set_wolff(algo)
            b.init()
            b.emcs(250, 1, 1)
            # queues and bitmaps 2.4 MiB, tiles 4 MiB
            before = b.launches
            with free_memory(1 << 20) if limit else contextlib.nullcontext():
                out = [*b.emcs(10, 1, 1), *b.emcs(5, 2, 1)]
            assert (b.launches - before < 15) == (limit or algo == "bfs")
            b.set_wolff(algo)  # asked again, there is room
            before = b.launches
            got.append(out + [*b.emcs(4, 1, 0)] + [b.member(i).state for i in range(20)])
            assert (b.launches - before < 4) == (algo == "bfs")
    for x, y in zip(*got):
        assert np.array_equal(x, y)


def test_small_handle_stays_on_bit_planes():
    import marqov_b200 as M
    rt = C.CDLL("libcudart.so.12")
    got = []
    for limit in (True, False):
        with M.makeCore(M.RegularHypercubic(32, 3), M.Config(seed=5), M.Ising(-1.0), 0.2216546) as c:
            c.init()
            c.emcs(2, 0, 1)
            with free_memory(64 << 10) if limit else contextlib.nullcontext():
                small, size = [], 1 << 20
                while limit and size >= 64 << 10:  # what is left of the allocator's blocks; queue 131 KB, tiles 213
                    p = C.c_void_p()
                    if rt.cudaMalloc(C.byref(p), C.c_size_t(size)):
                        rt.cudaGetLastError()
                        size //= 2
                    else:
                        small.append(p)
                got.append([c.wolff(3), *c.emcs(2, 1, 1), c.state])
                for p in small:
                    rt.cudaFree(p)
            assert ("clusters=label-smem" in c.describe()) == limit
    for x, y in zip(*got):
        assert np.array_equal(x, y)
