"""Performance cases of the engine: what its users run, through the public API.

Each case is one pass of a simulation that is already set up and thermalising:
a Core or a Batch is created, initialised and advanced a few EMCS in
``prepare``; ``run`` advances it by the EMCS of one call and returns the
observables of every EMCS with the updated state (large states as the device
buffers they live in).  ``exact`` restates the chain of the hypercubic models
in plain FP64 torch on the same keyed random words.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import marqov_b200 as M
import marqov_b200.autograd as A

BETA_C = 0.44068679  # critical coupling of the 2D Ising model
FARM_SIZES = (32, 48, 64, 96, 128, 192, 256, 384, 512)


def listed():
    return [
        # the reference's unit of work, one EMCS per call on the parity lattice: launch and call latency
        dict(name="ising2d_L64_step", kind="ising", dim=2, L=64, n=1, ncluster=1, nmetro=1),
        # the parity run itself: chunks of 1 cluster + 1 sweep + measurement on a small lattice
        dict(name="ising2d_L64_run", kind="ising", dim=2, L=64, n=100, ncluster=1, nmetro=1),
        # an ordinary finite-size-scaling lattice, cluster and sweep
        dict(name="ising2d_L1024_run", kind="ising", dim=2, L=1024, n=8, ncluster=1, nmetro=1),
        # a large critical lattice where clusters are mixed with sweeps
        dict(name="ising2d_L4096_run", kind="ising", dim=2, L=4096, n=2, ncluster=1, nmetro=4),
        # the largest lattice, Metropolis only: the headline sweep rate
        dict(name="ising2d_L16384_sweeps", kind="ising", dim=2, L=16384, n=4, ncluster=0, nmetro=5),
        # a farm of Potts replicas of uneven sizes around the transition, the scheduler's job
        dict(name="potts_farm_48", kind="farm", q=3, members=48, n=8, ncluster=1, nmetro=1),
        # replica exchange over a temperature ladder
        dict(name="tempering_32xL128", kind="tempering", L=128, members=32, n=20, ncluster=1, nmetro=1),
        # disorder realisations of a spin glass, Metropolis only
        dict(name="ea_32xL32", kind="ea", L=32, members=32, n=16, nmetro=1),
        # Heisenberg critical point: small-cap sweeps with one plane-reflection cluster per five
        dict(name="heisenberg_L128_run", kind="vector", model="heisenberg", proposal="smallcap", L=128, n=2,
             ncluster=1, nmetro=5),
        # phi^4 chains over a range of beta, cluster + sweep, as the gradient workload runs them
        dict(name="phi4_32xL64_run", kind="phi4", L=64, members=32, n=4, ncluster=1, nmetro=1),
        # differentiable observables: chains, device samples, forward and backward
        dict(name="phi4_autograd_16xL16", kind="autograd", L=16, members=16, n=200, ntherm=50),
        # a general graph: Ising on a random geometric graph, Metropolis only
        dict(name="rgg_131072_sweeps", kind="graph", N=131072, n=4, nmetro=5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _even(x, step=2):
    return max(step, int(round(x / step)) * step)


def draw(rng):
    kind = rng.choice(["ising", "ising", "ising3d", "farm", "tempering", "ea", "vector", "phi4", "autograd", "graph"])
    if kind == "ising":
        L = _even(_log(rng, 32, 8192), rng.choice([2, 64]))
        nc = rng.choice([0, 1, 1, 2])
        return dict(kind="ising", dim=2, L=L, n=max(1, min(100, int(_log(rng, 0.25, 4) * 2e6 / L ** 2))), ncluster=nc,
                    nmetro=rng.randint(1, 5))
    if kind == "ising3d":
        L = _even(_log(rng, 8, 160))
        return dict(kind="ising", dim=3, L=L, n=max(1, min(50, int(4e6 / L ** 3))), ncluster=rng.choice([0, 1]),
                    nmetro=rng.randint(1, 5))
    if kind == "farm":
        return dict(kind="farm", q=rng.choice([2, 3, 4, 5]), members=rng.randint(8, 56), n=rng.randint(2, 12),
                    ncluster=rng.choice([0, 1, 1]), nmetro=rng.randint(1, 2))
    if kind == "tempering":
        return dict(kind="tempering", L=_even(_log(rng, 32, 192)), members=rng.randint(8, 40), n=rng.randint(4, 24),
                    ncluster=rng.choice([0, 1]), nmetro=1)
    if kind == "ea":
        return dict(kind="ea", L=_even(_log(rng, 8, 40)), members=rng.randint(4, 48), n=rng.randint(4, 24),
                    nmetro=rng.randint(1, 2))
    if kind == "vector":
        model = rng.choice(["heisenberg", "xxz"])
        return dict(kind="vector", model=model, proposal=rng.choice(["fresh", "smallcap"]), L=_even(_log(rng, 12, 128)),
                    n=rng.randint(1, 3), ncluster=1 if model == "heisenberg" else 0, nmetro=rng.randint(1, 5))
    if kind == "phi4":
        L = _even(_log(rng, 12, 64))
        return dict(kind="phi4", L=L, members=max(2, min(48, int(_log(rng, 1, 8) * 1e6 / L ** 3))), n=rng.randint(1, 4),
                    ncluster=rng.choice([0, 1, 1]), nmetro=1)
    if kind == "autograd":
        return dict(kind="autograd", L=_even(rng.uniform(8, 20)), members=rng.randint(4, 24), n=rng.randint(60, 200),
                    ntherm=rng.randint(10, 50))
    return dict(kind="graph", N=int(_log(rng, 4096, 160000)), n=rng.randint(1, 4), nmetro=rng.randint(1, 5))


class _DeviceArray:
    """An engine buffer as torch sees it; holds its core, which owns the memory."""

    def __init__(self, core, ptr, shape, typestr):
        self.core = core
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _state(core):
    """The state on the GPU, as the engine's device buffer."""
    ptr, nbytes = core.state_device_ptr()
    item = np.dtype(core.dtype).itemsize
    return torch.as_tensor(_DeviceArray(core, ptr, (nbytes // item,), "<f4" if item == 4 else "|i1"), device="cuda")


def _betas(case):
    """The couplings of a batch, in the range the case's model is run at."""
    r = case["members"]
    lo, hi = {"tempering": (0.40, 0.48), "phi4": (0.36, 0.38), "autograd": (0.36, 0.38)}[case["kind"]]
    return [float(lo + (hi - lo) * (i + 0.5) / r) for i in range(r)]


def _farm_sizes(case):
    # the farm's lattices, evenly over the sizes
    return [FARM_SIZES[(5 * i + 2) % len(FARM_SIZES)] for i in range(case["members"])]


def _model(case):
    if case["model"] == "xxz":
        return M.XXZAntiferro(0.8, 0.2, case["proposal"], -0.5)
    return M.Heisenberg(-1.0, case["proposal"], -0.9697)


def _core(case, seed, lattice, ham, beta, warm):
    cfg = M.Config(seed=seed, ncluster=case.get("ncluster", 0), nmetro=case["nmetro"])
    core = M.makeCore(lattice, cfg, ham, beta)
    core.init()
    core.emcs(warm, cfg.ncluster, cfg.nmetro, measure=False)
    return core


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ising":
        beta = BETA_C if case["dim"] == 2 else 0.2216546
        core = _core(case, seed, M.RegularHypercubic(case["L"], case["dim"]), M.Ising(-1.0), beta, _warm(case))
        return {"case": case, "core": core}
    if kind == "vector":
        core = _core(case, seed, M.RegularHypercubic(case["L"], 3), _model(case), 0.693, _warm(case))
        return {"case": case, "core": core}
    if kind == "graph":
        lattice = M.RandomGeometricGraph2D(case["N"], 8.0, seed=seed)
        core = _core(case, seed, lattice, M.Ising(-1.0, "int8"), 0.5, _warm(case))
        return {"case": case, "core": core}
    if kind == "autograd":
        g = np.random.default_rng(seed)
        beta = torch.tensor(_betas(case), dtype=torch.float64, requires_grad=True)
        lam = torch.full((case["members"],), 1.1, dtype=torch.float64, requires_grad=True)
        ens = A.Phi4Ensemble(L=case["L"], dim=3, n_therm=case["ntherm"], n_meas=case["n"], seed=seed)
        return {"case": case, "beta": beta, "lam": lam, "ens": ens,
                "gout": torch.tensor(g.standard_normal((case["members"], 3)))}
    if kind == "farm":
        tc = 1.0 / math.log(1.0 + math.sqrt(case["q"]))
        members = [(M.RegularHypercubic(L, 2), M.Config(seed=seed + i, repid=i), M.Potts(case["q"], -1.0),
                    1.0 / (tc * (0.9 + 0.2 * (i + 0.5) / case["members"]))) for i, L in enumerate(_farm_sizes(case))]
    elif kind == "tempering":
        members = [(M.RegularHypercubic(case["L"], 2), M.Config(seed=seed, repid=i), M.Ising(-1.0), b)
                   for i, b in enumerate(_betas(case))]
    elif kind == "ea":
        members = [(M.RegularRandomBond(case["L"], 3, 0.5, seed=seed + i), M.Config(seed=seed, repid=i),
                    M.EdwardsAndersonIsing(-1.0), 0.9) for i in range(case["members"])]
    else:
        members = [(M.RegularHypercubic(case["L"], 3), M.Config(seed=seed, repid=i), M.Phi4(b, 1.1), b)
                   for i, b in enumerate(_betas(case))]
    batch = M.Batch(members)
    batch.init()
    batch.emcs(_warm(case), case.get("ncluster", 0), case["nmetro"])
    return {"case": case, "batch": batch}


def _warm(case):
    """EMCS before the first pass."""
    if case["kind"] == "ising" and case["dim"] == 2 and case["L"] <= 256:
        return 50
    return 4


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "autograd":
        out = A.phi4_observables(state["beta"], state["lam"], state["ens"])
        gb, gl = torch.autograd.grad(out, (state["beta"], state["lam"]), state["gout"])
        return {"obs": out.detach(), "grad_beta": gb, "grad_lambda": gl}
    if "core" in state:
        core = state["core"]
        if kind == "ising" and case["n"] == 1 and core.n <= 65536:
            mc = core.elementaryMCstep()
            return {"mean_cluster": mc, "state": core.state}
        obs, mc = core.emcs(case["n"], case.get("ncluster", 0), case["nmetro"])
        return {"obs": obs, "mean_cluster": mc, "state": core.state if core.n <= 65536 else _state(core)}
    batch = state["batch"]
    if kind == "tempering":
        obs, other = batch.tempering(case["n"], 1, case["ncluster"], case["nmetro"], seed=11)
    else:
        obs, other = batch.emcs(case["n"], case.get("ncluster", 0), case["nmetro"])
    return {"obs": obs, "mean_cluster" if kind != "tempering" else "accepted": other,
            "states": [_state(batch.member(i)) for i in range(len(batch))]}


def work(case):
    """The state is read and written once per pass, bonds and graph read once;
    operations: about 60 per site update (a keyed draw, the neighbours, the
    acceptance) and 30 per site of a cluster step's bonds."""
    kind = case["kind"]
    extra = 0
    if kind == "farm":
        sites = sum(L * L for L in _farm_sizes(case))
    elif kind == "graph":
        sites = case["N"]
        extra = 4 * (sites + 1) + 4 * 8 * sites
    elif kind == "ising":
        sites = case["L"] ** case["dim"]
    else:
        sites = case.get("members", 1) * case["L"] ** (2 if kind == "tempering" else 3)
    if kind == "ea":
        extra = 3 * sites
    item = {"vector": 12, "phi4": 4, "autograd": 4}.get(kind, 1)
    nobs = case.get("members", 1) * case["n"] * 32
    n = case["n"] + case.get("ntherm", 0)
    per = 60 * case.get("nmetro", 1) + 30 * case.get("ncluster", 1 if kind == "autograd" else 0)
    return {"bytes": float(2 * item * sites + extra + nobs), "flops": float(per * n * sites)}


# ---------------------------------------------------------------------------
# The chain of a hypercubic model in FP64, site by site on the keyed words of
# the engine's random streams (Philox4x32-10 on (site, sweep, block, stream)).

_MASK = 0xFFFFFFFF


def _mul(a, b):
    x, y = a * (b >> 16), a * (b & 0xFFFF)
    t = x + (y >> 16)
    return t >> 16, ((t & 0xFFFF) << 16) | (y & 0xFFFF)


def _philox(c0, c1, c2, c3, seed):
    k0, k1 = seed & _MASK, (seed >> 32) & _MASK
    for r in range(10):
        h0, l0 = _mul(0xD2511F53, c0)
        h1, l1 = _mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & _MASK, (k1 + 0xBB67AE85) & _MASK
    return c0, c1, c2, c3


def _real(lo, hi):
    """(word >> 11) 2^-53 of the word hi 2^32 + lo."""
    return ((hi << 21) | (lo >> 11)).to(torch.float64) * 2.0 ** -53


class _Chain:
    """One lattice: Ising (with bonds), phi^4 or 3-vector spins in [comp, n]."""

    def __init__(self, model, dim, L, beta, seed, rep, bonds=None, ham=None):
        self.model, self.dim, self.L, self.beta, self.seed, self.rep, self.ham = model, dim, L, beta, seed, rep, ham
        self.n = L ** dim
        self.shape = (L,) * dim
        self.i = torch.arange(self.n, dtype=torch.int64, device="cuda")
        par = sum((self.i // L ** j) % L for j in range(dim)) & 1
        self.colour = [par == c for c in (0, 1)]
        # +d bonds of every site
        self.bonds = None if bonds is None else [torch.from_numpy(np.ascontiguousarray(bonds[:, 2 * d])).cuda().double()
                                                 for d in range(dim)]
        self.fwd = [self.roll(self.i, d, -1) for d in range(dim)]
        self.sweep = self.cluster = 0
        x = self.words(2, 0, 0)
        if model == "ising":
            self.s = torch.where(x[0] > 0.5, 1.0, -1.0).double()[None]
        elif model == "phi4":
            self.s = self.f32((torch.sqrt(-2.0 * torch.log(1.0 - x[0])) * torch.cos(2 * math.pi * x[1]))[None])
        else:
            self.s = self.f32(self.direction(x[0], x[1]))

    @staticmethod
    def f32(v):
        return v.float().double()  # the stored precision

    @staticmethod
    def direction(u0, u1):
        a0, a1 = 2.0 * u0, 2.0 * u1
        r = torch.sqrt(a0 * (2.0 - a0))
        return torch.stack([1.0 - a0, r * torch.sin(math.pi * a1), r * torch.cos(math.pi * a1)])

    def tag(self, stream):
        return (stream << 24) | self.rep

    def words(self, stream, c1, block):
        """The two uniforms of every site's block."""
        z = torch.zeros_like(self.i)
        b = _philox(self.i, z + c1, z + block, z + self.tag(stream), self.seed)
        return _real(b[0], b[1]), _real(b[2], b[3])

    def roll(self, v, d, by):
        """v at the neighbour: by = -1 the +d neighbour's value, +1 the -d neighbour's."""
        return torch.roll(v.reshape(self.shape), by, self.dim - 1 - d).reshape(-1)

    def field(self):
        """Sum over the neighbours (bond weights on Ising lattices)."""
        out = torch.zeros_like(self.s)
        for c in range(self.s.shape[0]):
            for d in range(self.dim):
                v = self.s[c]
                if self.bonds is None:
                    out[c] += self.roll(v, d, -1) + self.roll(v, d, 1)
                else:
                    out[c] += self.bonds[d] * self.roll(v, d, -1) + self.roll(self.bonds[d] * v, d, 1)
        return out

    def accept_real(self):
        """Each site's acceptance uniform: bit-sliced top byte, 45 fine bits."""
        z = torch.zeros_like(self.i)
        g, q = ((self.i >> 6) << 1) | (self.i & 1), (self.i >> 1) & 31
        planes = _philox(g, z + self.sweep, z, z + self.tag(5), self.seed)
        planes += _philox(g, z + self.sweep, z + 1, z + self.tag(5), self.seed)
        top = sum(((p >> q) & 1) << b for b, p in enumerate(planes))
        f = _philox(self.i >> 1, z + self.sweep, z, z + self.tag(6), self.seed)
        odd = (self.i & 1) == 1
        fine = (torch.where(odd, f[3], f[1]) & 0xFFFFFF) << 21 | torch.where(odd, f[2], f[0]) >> 11
        return (top << 45 | fine).double() * 2.0 ** -53

    def propose(self):
        s, (u0, u1) = self.s, self.words(1, self.sweep, 0)
        if self.model == "ising":
            return -s
        if self.model == "phi4":
            return self.f32(s + self.ham.amp * (1.0 - 2.0 * u0))
        if self.ham.proposal != "smallcap":
            return self.f32(self.direction(u0, u1))
        ca = 1.0 - u0 * (1.0 - self.ham.cap)
        sa = torch.sqrt(torch.clamp(1.0 - ca * ca, min=0.0))
        dx, dy = sa * torch.cos(2 * math.pi * u1), sa * torch.sin(2 * math.pi * u1)
        x, y, z = s
        sg = torch.where(z < 0, -1.0, 1.0).double()
        a = 1.0 / (1.0 + sg * z)
        b = -x * y * a
        v = torch.stack([dx * (1.0 - x * x * a) + dy * b + ca * x, dx * b + dy * (1.0 - y * y * a) + ca * y,
                         -dx * x * sg - dy * y * sg + ca * z])
        return self.f32(v / torch.sqrt((v * v).sum(0)))

    def metropolis(self):
        u, new = self.accept_real(), self.propose()
        for mask in self.colour:
            d, f, s = new - self.s, self.field(), self.s
            if self.model == "phi4":
                n2, o2, h = new[0] ** 2, s[0] ** 2, self.ham
                dE = (-d[0] * f[0] + h.mass / h.beta * (n2 - o2)
                      + h.lambda_ / h.beta * ((n2 - 1) ** 2 - (o2 - 1) ** 2))
            elif self.model == "xxz":
                dE = self.ham.Delta * (d[0] * f[0] + d[1] * f[1]) + d[2] * f[2] + self.ham.H * d[2]
            else:
                dE = -(d * f).sum(0)
            ok = mask & ((dE <= 0) | (u < torch.exp(-self.beta * dE)))
            self.s = torch.where(ok[None], new, self.s)
        self.sweep += 1

    def wolff(self):
        t = [torch.tensor([v], dtype=torch.int64) for v in (0, self.cluster, 0, self.tag(3))]
        b0 = _philox(*t, self.seed)
        b1 = _philox(t[0], t[1], t[2] + 1, t[3], self.seed)
        seed = (int(b0[1]) << 32 | int(b0[0])) % self.n
        u1, u2 = _real(b0[2], b0[3]), _real(b1[0], b1[1])
        if self.model == "ising":
            a = self.s[0]
        elif self.model == "phi4":
            a = self.s[0] * (-1.0 if float(u1) < 0.5 else 1.0)
        else:
            r = self.f32(self.direction(u1, u2)).cuda()
            a = (self.s * r).sum(0)
        z = torch.zeros_like(self.i)
        act = []
        for d in range(self.dim):
            j = self.fwd[d]
            w = _philox(torch.minimum(self.i, j), z + self.cluster, torch.maximum(self.i, j), z + self.tag(4), self.seed)
            u, cpl = _real(w[0], w[1]), a * a[j]
            p = -torch.expm1(-2.0 * self.beta * cpl)
            act.append((cpl > 0) & ((u < p) if self.model == "ising" else (u >= 1.0 - p)))
        flood = torch.zeros(self.n, dtype=torch.bool, device="cuda")
        flood[seed] = True
        size = 1
        while True:
            for _ in range(16):
                for d in range(self.dim):
                    flood = flood | (act[d] & self.roll(flood, d, -1)) | self.roll(act[d] & flood, d, 1)
            now = int(flood.sum())
            if now == size:
                break
            size = now
        if self.model in ("ising", "phi4"):
            self.s = torch.where(flood[None], -self.s, self.s)
        else:
            v = self.s - 2.0 * a[None] * r
            self.s = torch.where(flood[None], self.f32(v / torch.sqrt((v * v).sum(0))), self.s)
        self.cluster += 1
        return size

    def observables(self):
        s, n = self.s, self.n
        f = self.field()
        if self.model == "phi4":
            h, p = self.ham, s[0] ** 2
            e = -float((s * f).sum()) / (2 * n) + (h.mass / h.beta * float(p.sum())
                                                   + h.lambda_ / h.beta * float(((p - 1) ** 2).sum())) / n
        elif self.model == "xxz":
            w = torch.tensor([self.ham.Delta ** 2, self.ham.Delta ** 2, 1.0], dtype=torch.float64, device="cuda")[:, None]
            e = float((w * s * f).sum()) / (2 * n) + self.ham.H * float(s[2].sum()) / n
        else:
            e = -float((s * f).sum()) / (2 * n)
        m = math.sqrt(sum(float(c.sum()) ** 2 for c in s)) / n
        return [e, m, m ** 2, m ** 4]

    def emcs(self, n, ncluster, nmetro, measure=True):
        obs, mean = [], []
        for _ in range(n):
            sizes = [self.wolff() for _ in range(ncluster)]
            for _ in range(nmetro):
                self.metropolis()
            if measure:
                obs.append(self.observables())
                mean.append(sum(sizes) / ncluster if ncluster else 0.0)
        return obs, mean


def exact(case, seed):
    """Observables and float states of the first pass, in FP64.  None for
    farms, exchanges, graphs and gradient runs, and for lattices where it takes
    long."""
    kind = case["kind"]
    nc, nm = case.get("ncluster", 0), case.get("nmetro", 1)
    if kind in ("ising", "vector"):
        model, beta, ham = "ising", BETA_C, None
        if kind == "vector":
            model, beta, ham = case["model"], 0.693, _model(case)
        elif case["dim"] == 3:
            beta = 0.2216546
        if case["L"] ** case.get("dim", 3) > 2200000:
            return None
        c = _Chain(model, case.get("dim", 3), case["L"], beta, seed, 0, ham=ham)
        c.emcs(_warm(case), nc, nm, measure=False)
        obs, mc = c.emcs(case["n"], nc, nm)
        if kind == "ising" and case["n"] == 1 and c.n <= 65536:
            return {"mean_cluster": mc[0], "state": None}
        full = kind == "vector"
        state = None
        if full:
            state = c.s.reshape(-1)
            if c.n <= 65536:
                state = c.s.T.reshape(-1)  # site-major, as Core.state returns it
        return {"obs": np.array(obs), "mean_cluster": np.array(mc), "state": state}
    if kind in ("ea", "phi4"):
        chains = []
        for i in range(case["members"]):
            if kind == "ea":
                chains.append(_Chain("ising", 3, case["L"], 0.9, seed, i,
                                     bonds=M.RegularRandomBond(case["L"], 3, 0.5, seed=seed + i).bonds))
            else:
                b = _betas(case)[i]
                chains.append(_Chain("phi4", 3, case["L"], b, seed, i, ham=M.Phi4(b, 1.1)))
        obs, mc = [], []
        for c in chains:
            c.emcs(_warm(case), nc, nm, measure=False)
            o, m = c.emcs(case["n"], nc, nm)
            obs.append(o)
            mc.append(m)
        return {"obs": np.array(obs).transpose(1, 0, 2), "mean_cluster": np.array(mc).T,
                "states": [c.s.reshape(-1) if kind == "phi4" else None for c in chains]}
    return None
