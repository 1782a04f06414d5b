"""The steps of the one-launch graph sweeps (csr_sweep.cu) on the CPU: every CTA
has a word of every colour, and a model of their synchronisation (words that
count at two barriers in turn, a CTA barrier before every wait) in which warps
and words are late at random: no word counts at another step's phase, no wait
passes early and none is left waiting."""
import ctypes as C
import random

import numpy as np
import pytest


def layout(colours, ctas):
    from marqov_b200 import _lib
    colours = np.ascontiguousarray(colours, np.int32)
    ncol = C.c_int32()
    words = np.zeros((int(colours.max()) + 1, ctas), np.int32)
    _lib.check(_lib.load().mqv_selftest_graph_words(colours.size, colours.ctypes.data, ctas, words.ctypes.data,
                                                    words.size, C.byref(ncol)))
    return words[:ncol.value]


def colourings():
    rng = np.random.default_rng(2)
    greedy = np.minimum(rng.geometric(0.45, 3000) - 1, 9)  # few sites have a late colour
    return {"greedy": greedy, "empty_classes": np.array([0, 3, 4000])[rng.integers(0, 3, 2000)],
            "sorted": np.sort(rng.integers(0, 6, 1500)), "one": np.zeros(64, int), "word": np.arange(96) // 32,
            "split": np.r_[np.zeros(1000, int), np.full(1000, 2)]}


@pytest.mark.parametrize("name", list(colourings()))
@pytest.mark.parametrize("ctas", [1, 2, 16])
def test_every_cta_has_a_word_of_every_colour(name, ctas):
    col = colourings()[name]
    w = layout(col, ctas)
    ids = np.unique(col)
    assert len(w) == len(ids) and w.min() >= 1
    rng64 = -(-(-(-len(col) // ctas)) // 64) * 64
    for c, k in enumerate(ids):
        for r in range(ctas):
            have = int((col[r * rng64:(r + 1) * rng64] == k).sum())
            assert w[c, r] == max(1, -(-have // 32))


class Bar:
    def __init__(self):
        self.phase, self.pending, self.bytes = 0, 1, 0

    def settle(self):
        if self.pending == 0 and self.bytes == 0:
            self.phase, self.pending = self.phase + 1, 1


def simulate(words, seed, warps=3):
    """Random interleavings; raises AssertionError where the protocol breaks."""
    rng = random.Random(seed)
    steps, ctas = len(words), len(words[0])
    bars = [[Bar(), Bar()] for _ in range(ctas)]
    flying = []  # ("word", destination, step)

    def warp(r, w):
        for t in range(steps):
            if t:
                yield "sync", None
                yield "wait", t - 1
            if w == 0:
                b = bars[r][t & 1]
                b.pending -= 1
                b.bytes += sum(words[t])
                b.settle()
                yield "go", None
            for _ in range(w, words[t][r], warps):
                flying.extend(("word", q, t) for q in range(ctas))
                yield "go", None
        yield "sync", None
        yield "wait", steps - 1

    run = {(r, w): warp(r, w) for r in range(ctas) for w in range(warps)}
    at = {k: next(g) for k, g in run.items()}
    slow = {k: rng.choice([1.0, 1.0, 0.02]) for k in run}
    lag = [rng.choice([1.0, 0.02]) for _ in range(ctas)]

    def ready(k):
        kind, t = at[k]
        if kind == "sync":
            return all(at[k[0], w][0] == "sync" for w in range(warps))
        return kind == "go" or bars[k[0]][t & 1].phase % 2 != (t >> 1) % 2

    while run or flying:
        acts = [(slow[k], k) for k in run if ready(k)] + [(lag[m[1]], m) for m in sorted(set(flying))]
        assert acts, "left waiting"
        _, a = rng.choices(acts, [x for x, _ in acts])[0]
        if a in run:
            if at[a][0] == "wait":
                assert bars[a[0]][at[a][1] & 1].phase == at[a][1] // 2 + 1, "a wait passed early"
            for k in ([(a[0], w) for w in range(warps)] if at[a][0] == "sync" else [a]):
                try:
                    at[k] = next(run[k])
                except StopIteration:
                    del run[k], at[k]
        else:
            flying.remove(a)
            b = bars[a[1]][a[2] & 1]
            assert b.phase == a[2] // 2, "a word counts at another step's phase"
            b.bytes -= 1
            b.settle()


@pytest.mark.parametrize("name,ctas", [("greedy", 3), ("empty_classes", 2), ("sorted", 4), ("split", 2)])
def test_words_count_at_their_own_step(name, ctas):
    w = layout(colourings()[name][::8], ctas).tolist()
    for seed in range(60):
        simulate([[2] * ctas] + w * 3, seed)


def test_the_model_finds_a_cta_without_a_word():
    broken = 0
    for seed in range(60):
        try:
            simulate([[2, 2, 2]] + [[2, 1, 1], [1, 0, 0], [1, 0, 1], [0, 1, 0]] * 3, seed)
        except AssertionError:
            broken += 1
    assert broken > 10
