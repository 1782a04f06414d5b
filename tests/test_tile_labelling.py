"""The bit-tile labelling of Wolff clusters (wolff_tile.cuh) restated in Python
and checked on the CPU: the tiles' units cover every x-line word once, the
bonds drawn inside tiles and the bonds hooked between them are the lattice's
bonds, each once, with every index in its buffer; and runs, one union per pair
of adjacent runs, hooking and the carry closure give the seed's component of
the active bonds, as breadth-first search does."""
import numpy as np
import pytest

M32 = 0xFFFFFFFF


class Geo:
    def __init__(self, dim, L, U):
        self.dim, self.L, self.U = dim, L, U
        self.Lz = L if dim == 3 else 1
        self.TY = U if dim == 2 else (16 if U >= 256 else 8)
        self.TZ = U // self.TY
        self.nw = (L + 31) // 32
        self.ny = -(-L // self.TY)
        self.nz = -(-self.Lz // self.TZ)
        self.n = self.nw * self.ny * self.nz

    def at(self, t):
        q = t // self.nw
        return t % self.nw, q % self.ny, q // self.ny

    def row(self, t, u):
        _, ty, tz = self.at(t)
        y, z = ty * self.TY + u % self.TY, tz * self.TZ + u // self.TY
        return y + self.L * z if y < self.L and z < self.Lz else -1

    def site(self, t, u, b):
        return self.row(t, u) * self.L + self.at(t)[0] * 32 + b

    def live(self, t, u, b):
        return self.row(t, u) >= 0 and self.at(t)[0] * 32 + b < self.L

    def place(self, i):
        rw, x = divmod(i, self.L)
        z, y = divmod(rw, self.L) if self.Lz > 1 else (0, rw)
        return ((x >> 5) + self.nw * (y // self.TY + self.ny * (z // self.TZ)),
                y % self.TY + self.TY * (z % self.TZ), x & 31)

    def inner(self, t):
        """(unit, bit, unit, bit, dimension) of the bonds drawn inside tile t."""
        for u in range(self.U):
            for b in range(32):
                if not self.live(t, u, b):
                    continue
                if b < 31 and self.live(t, u, b + 1):
                    yield u, b, u, b + 1, 0
                if u % self.TY < self.TY - 1 and self.live(t, u + 1, b):
                    yield u, b, u + 1, b, 1
                if self.dim == 3 and u // self.TY < self.TZ - 1 and self.live(t, u + self.TY, b):
                    yield u, b, u + self.TY, b, 2

    def hooks(self, t):
        """(unit, bit, tile, unit, bit) of the bonds that leave tile t, item by item."""
        tx, ty, tz = self.at(t)
        L, TY, TZ, U = self.L, self.TY, self.TZ, self.U
        yl, zl = min(TY - 1, L - 1 - ty * TY), min(TZ - 1, self.Lz - 1 - tz * TZ)
        for k in range(U + 32 * TZ + (32 * TY if self.dim == 3 else 0)):
            if k < U:
                u, b, b2, u2 = k, min(31, L - 1 - tx * 32), 0, k
                t2 = t + 1 if tx + 1 < self.nw else t - tx
            elif k < U + 32 * TZ:
                q = k - U
                z, b = q >> 5, q & 31
                b2, u = b, yl + TY * z
                t2 = t + self.nw if ty * TY + yl + 1 < L else t - ty * self.nw
                u2 = TY * z
                if z > zl:
                    continue
            else:
                q = k - U - 32 * TZ
                y, b = q >> 5, q & 31
                b2, u = b, y + TY * zl
                plane = self.nw * self.ny
                t2 = t + plane if tz * TZ + zl + 1 < L else t - tz * plane
                u2 = y
            if self.live(t, u, b):
                yield u, b, t2, u2, b2


GEOS = [(2, 4, 64), (2, 30, 64), (2, 32, 64), (2, 48, 64), (2, 66, 64), (2, 130, 128), (2, 260, 128), (3, 4, 64),
        (3, 10, 64), (3, 16, 64), (3, 18, 128), (3, 34, 64), (3, 20, 128)]


@pytest.mark.parametrize("dim,L,U", GEOS)
def test_every_bond_once(dim, L, U):
    g = Geo(dim, L, U)
    n = L ** dim
    seen = np.zeros(n, int)
    bonds = set()

    def add(i, j):
        assert 0 <= i < n and 0 <= j < n
        e = (min(i, j), max(i, j))
        assert e not in bonds
        bonds.add(e)

    for t in range(g.n):
        for u in range(U):
            for b in range(32):
                if g.live(t, u, b):
                    i = g.site(t, u, b)
                    seen[i] += 1
                    assert g.place(i) == (t, u, b)
        for u, b, u2, b2, _ in g.inner(t):
            assert 0 <= u2 < U
            add(g.site(t, u, b), g.site(t, u2, b2))
        for u, b, t2, u2, b2 in g.hooks(t):
            assert 0 <= t2 < g.n and 0 <= u2 < U and g.live(t2, u2, b2)
            add(g.site(t, u, b), g.site(t2, u2, b2))
    assert (seen == 1).all()
    want = set()
    for i in range(n):
        for d in range(dim):
            p = L ** d
            x = (i // p) % L
            j = i + p if x + 1 < L else i - (L - 1) * p
            want.add((min(i, j), max(i, j)))
    assert bonds == want


def _find(p, x):
    while p[x] != x:
        x = p[x]
    return x


def _start(S, b):
    return (S & (M32 >> (31 - b))).bit_length() - 1


@pytest.mark.parametrize("prob", [0.3, 0.59, 0.9])
@pytest.mark.parametrize("dim,L,U", [(2, 30, 64), (2, 66, 64), (2, 130, 128), (3, 10, 64), (3, 18, 128), (3, 34, 64)])
def test_component_of_the_seed(dim, L, U, prob):
    g = Geo(dim, L, U)
    n = L ** dim
    rng = np.random.default_rng(L + int(100 * prob))
    cand = rng.random(n) < 0.75
    seed = int(rng.integers(n))
    cand[seed] = True
    draw = {}

    def active(i, j):
        e = (min(i, j), max(i, j))
        if e not in draw:
            draw[e] = rng.random() < prob
        return cand[i] and cand[j] and draw[e]

    C = [[sum(1 << b for b in range(32) if g.live(t, u, b) and cand[g.site(t, u, b)]) for u in range(U)]
         for t in range(g.n)]
    X, lab, forest = [], [], {}
    adj = {}
    for t in range(g.n):
        B = [[0] * U for _ in range(3)]
        for u, b, u2, b2, d in g.inner(t):
            i, j = g.site(t, u, b), g.site(t, u2, b2)
            if active(i, j):
                B[d][u] |= 1 << b
                adj.setdefault(i, []).append(j)
                adj.setdefault(j, []).append(i)
        S = [C[t][u] & ~(B[0][u] << 1) & M32 for u in range(U)]
        P = list(range(U * 32))
        unions = []
        for u in range(U):
            if u % g.TY:
                Y, A = B[1][u - 1], (B[0][u] << 1) & M32
                E = (Y << 1) & A
                above = E | ((((A + E) & M32) ^ A) & A)
                for b in range(32):
                    if ((Y & ~above) >> b) & 1:  # the run's parent by a plain store, once
                        x = u * 32 + _start(S[u], b)
                        assert P[x] == x
                        P[x] = (u - 1) * 32 + _start(S[u - 1], b)
                unions.append((u, u - 1, Y & above & ~((Y & B[0][u] & B[0][u - 1]) << 1)))
            if dim == 3 and u // g.TY < g.TZ - 1:
                Z = B[2][u]
                unions.append((u, u + g.TY, Z & ~((Z & B[0][u] & B[0][u + g.TY]) << 1)))
        for ua, ub, m in unions:
            for b in range(32):
                if (m >> b) & 1:
                    ra, rb = _find(P, ua * 32 + _start(S[ua], b)), _find(P, ub * 32 + _start(S[ub], b))
                    P[max(ra, rb)] = min(ra, rb)
        for u in range(U):
            for b in range(32):
                if (S[u] >> b) & 1:
                    x = u * 32 + b
                    r = _find(P, x)
                    if r == x:
                        forest[t * U * 32 + x] = t * U * 32 + x
        lab.append([_find(P, k) for k in range(U * 32)])
        X.append(B[0])

    def root_of(t, u, b):
        return t * U * 32 + lab[t][u * 32 + _start(C[t][u] & ~(X[t][u] << 1) & M32, b)]

    for t in range(g.n):
        for u, b, t2, u2, b2 in g.hooks(t):
            i, j = g.site(t, u, b), g.site(t2, u2, b2)
            if active(i, j):
                adj.setdefault(i, []).append(j)
                adj.setdefault(j, []).append(i)
                forest[_find(forest, root_of(t, u, b))] = _find(forest, root_of(t2, u2, b2))
    root = _find(forest, root_of(*g.place(seed)))
    got = np.zeros(n, bool)
    for t in range(g.n):
        S = [C[t][u] & ~(X[t][u] << 1) & M32 for u in range(U)]
        hit = [sum(1 << b for b in range(32) if (S[u] >> b) & 1 and lab[t][u * 32 + b] == u * 32 + b
                   and _find(forest, t * U * 32 + u * 32 + b) == root) for u in range(U)]
        for u in range(U):
            f = hit[u]
            for b in range(32):
                if (S[u] >> b) & 1:
                    q = lab[t][u * 32 + b]
                    if (hit[q >> 5] >> (q & 31)) & 1:
                        f |= 1 << b
            A = (X[t][u] << 1) & M32
            E = (f << 1) & A
            f = (f | E | ((((A + E) & M32) ^ A) & A)) & C[t][u]
            for b in range(32):
                if (f >> b) & 1:
                    got[g.site(t, u, b)] = True
    want = np.zeros(n, bool)
    want[seed] = True
    todo = [seed]
    while todo:
        for j in adj.get(todo.pop(), ()):
            if not want[j]:
                want[j] = True
                todo.append(j)
    assert (got == want).all()
