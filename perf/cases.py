"""The work that users of this package have it do, as cases that can be timed and compared.

Each case is one pass through the public entry points: ``PIMCKernel.run`` / ``runHost`` and
the getters a run loop calls after it, ``BatchSampler.run``, ``LearnedProposal.train`` and
``predict``.  ``listed()`` gives the cases, ``draw()`` more of the same ranges, ``prepare()``
what a program holds before the call, ``run()`` the pass, ``work()`` the bytes and operations
it cannot do without, and ``exact()`` the results in 64 bits from plain torch and numpy.
"""
import math

import numpy as np
import torch

SWEEP = {"kind": "sweep", "system": "ho", "n": 1, "walkers": 1024, "N": 128, "S": 3, "opruns": 10, "msteps": 1,
         "beta": 10.0, "luxury": -1, "double": False, "accumulation": "fp64", "partials": "fp32", "correlator": False,
         "histogram": False, "global_path": False, "per_group": 1, "fast": True, "per_block": 0, "blocks_per_sm": 0,
         "paths": False}


def listed():
    return [
        # one run of the N-doubling loop on the oscillator at its smallest sizes: launch and
        # read-back latency; every run reads the operators, the accepts and the paths
        dict(SWEEP, name="ho_run_loop", walkers=64, N=16, S=2, opruns=16, msteps=2, per_group=4, paths=True),
        # the oscillator benchmark: x^2 and <x(0)x(t)> after every sweep, 1024 walkers
        dict(SWEEP, name="ho_correlator", opruns=100, correlator=True),
        # the same measurement on long paths and a walker count that is no power of two
        dict(SWEEP, name="ho_correlator_long", walkers=6000, N=512, S=4, opruns=40, msteps=2, correlator=True),
        # one thread per walker: path shift, single-node move and bisection
        dict(SWEEP, name="ho_walker_moves", kind="moves", walkers=2048, N=16, S=2, opruns=50, msteps=4, beta=4.0),
        # the headline workload: He-4 trimer, RANLUX, virial energy and pair-distance histogram
        dict(SWEEP, name="he3_trimer", system="he", n=3, walkers=16384, N=256, S=4, opruns=5, msteps=10, beta=1.0,
             luxury=2, histogram=True, per_block=4, blocks_per_sm=7),
        # a step from and to page-locked host arrays, shorter paths, lower luxury, ragged walkers
        dict(SWEEP, name="he3_host", kind="host", system="he", n=3, walkers=5000, N=128, S=3, opruns=4, msteps=5,
             beta=1.0, luxury=1, histogram=True),
        # the three-particle example: bound trimer, paths in device memory, IEEE arithmetic,
        # four walkers per work-group
        dict(SWEEP, name="he3_bound_ieee", system="he3part", n=3, walkers=444, N=128, S=4, opruns=20, msteps=5,
             beta=1000.0, global_path=True, per_group=4, fast=False, paths=True),
        # the precision study: ten atoms, 1024 slices, every sum kept three ways
        dict(SWEEP, name="he10_study", system="he", n=10, walkers=4096, N=1024, S=2, opruns=2, msteps=2, beta=1.0,
             accumulation="study", correlator=True, global_path=True, blocks_per_sm=2),
        # FP64 everywhere on a five-atom cluster
        dict(SWEEP, name="he5_fp64", system="he", n=5, walkers=1024, N=128, S=3, opruns=2, msteps=2, beta=1.0,
             luxury=2, double=True, histogram=False),
        # many clusters of different sizes in one launch
        {"name": "ragged_batch", "kind": "batch", "systems": 24, "walkers": 256, "atoms": 10, "slices": 1024,
         "layout": 1, "block": 512, "target": 64},
        # the learned proposal inside the sweep
        dict(SWEEP, name="he3_learned", kind="learned", system="he", n=3, walkers=8192, N=256, S=4, opruns=5, msteps=2,
             beta=1.0, luxury=2),
        # training the proposal's network and its held-out predictions
        {"name": "train_proposal", "kind": "train", "rows": 200000, "held_out": 20011, "batch": 4096, "steps": 100,
         "dof": 6},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.choice(["loop", "correlator", "correlator", "moves", "trimer", "trimer", "host", "bound", "cluster",
                       "double", "batch", "learned", "train"])
    pow2 = lambda lo, hi: 2 ** rng.randint(lo, hi)  # noqa: E731
    if pick == "loop":
        N = pow2(3, 6)
        return dict(SWEEP, walkers=4 * _between(rng, 4, 500), N=N, S=rng.randint(1, int(math.log2(N))),
                    opruns=rng.randint(1, 20), msteps=rng.randint(1, 5), per_group=rng.choice([1, 2, 4]), paths=True,
                    luxury=rng.choice([-1, -1, 2]))
    if pick == "correlator":
        N = pow2(5, 9)
        S = rng.randint(2, 5)
        S = max(S, int(math.log2(N)) - 6)
        return dict(SWEEP, walkers=_between(rng, 100, 6000), N=N, S=S, opruns=rng.randint(5, 40),
                    msteps=rng.randint(1, 3), correlator=True, luxury=rng.choice([-1, -1, 1]),
                    accumulation=rng.choice(["fp64", "fp64", "kahan"]), partials=rng.choice(["fp32", "fp32", "exact"]))
    if pick == "moves":
        N = pow2(3, 6)
        return dict(SWEEP, kind="moves", walkers=_between(rng, 50, 4096), N=N, S=rng.randint(1, 3),
                    opruns=rng.randint(5, 50), msteps=rng.randint(1, 4), beta=4.0)
    if pick == "trimer":
        N = pow2(6, 8)
        S = rng.randint(2, 5)
        return dict(SWEEP, system="he", n=3, walkers=_between(rng, 500, 16384), N=N, S=S, opruns=rng.randint(1, 5),
                    msteps=rng.randint(1, 10), beta=rng.choice([0.5, 1.0, 2.0]), luxury=rng.choice([-1, 0, 1, 2, 2, 3]),
                    histogram=rng.choice([True, False]), fast=rng.choice([True, True, False]))
    if pick == "host":
        N = pow2(5, 8)
        return dict(SWEEP, kind="host", system="he", n=3, walkers=_between(rng, 300, 8000), N=N, S=rng.randint(2, 4),
                    opruns=rng.randint(1, 5), msteps=rng.randint(1, 5), beta=1.0, luxury=rng.choice([-1, 1, 2]),
                    histogram=True)
    if pick == "bound":
        return dict(SWEEP, system="he3part", n=3, walkers=4 * _between(rng, 10, 500), N=pow2(4, 8), S=rng.randint(2, 4),
                    opruns=rng.randint(5, 20), msteps=rng.randint(1, 5), beta=1000.0,
                    global_path=rng.choice([True, False]), per_group=4, fast=rng.choice([True, False]), paths=True)
    if pick == "cluster":
        return dict(SWEEP, system="he", n=rng.randint(4, 10), walkers=_between(rng, 200, 4096), N=pow2(7, 10),
                    S=rng.randint(2, 3), opruns=rng.randint(1, 2), msteps=rng.randint(1, 2), beta=1.0,
                    accumulation=rng.choice(["study", "fp64", "fp32"]), correlator=True, global_path=True)
    if pick == "double":
        return dict(SWEEP, system="he", n=rng.randint(3, 6), walkers=_between(rng, 100, 1024), N=pow2(5, 8),
                    S=rng.randint(2, 3), opruns=rng.randint(1, 2), msteps=rng.randint(1, 2), beta=1.0,
                    luxury=rng.choice([-1, 2]), double=True)
    if pick == "batch":
        return {"kind": "batch", "systems": rng.randint(4, 24), "walkers": _between(rng, 40, 256),
                "atoms": rng.randint(4, 10), "slices": pow2(7, 10), "layout": rng.randint(2, 10 ** 6),
                "block": rng.choice([256, 512]), "target": rng.choice([16, 32, 64])}
    if pick == "learned":
        S = rng.randint(4, 6)
        return dict(SWEEP, kind="learned", system="he", n=3, walkers=32 * _between(rng, 10, 256), N=pow2(7, 8), S=S,
                    opruns=rng.randint(1, 5), msteps=rng.randint(1, 2), beta=1.0, luxury=2)
    return {"kind": "train", "rows": _between(rng, 5000, 200000), "held_out": _between(rng, 100, 30000),
            "batch": _between(rng, 500, 8192), "steps": _between(rng, 10, 100), "dof": rng.choice([1, 3, 6, 8])}


# ------------------------------------------------------------------ inputs
HE_MASS_KELVIN = 6.64647617e-27 * (1e-10) ** 2 / 1.05457148e-34 ** 2 * 1.3806503e-23  # He-4 mass, Angstrom and Kelvin


def _jacobi(n, m):
    """Mass-scaled Jacobi vectors of n equal masses from positions, and the inverse."""
    J = np.zeros((n, n))
    for k in range(n - 1):
        J[k, :k + 1] = 1.0 / (k + 1)
        J[k, k + 1] = -1.0
        J[k] *= math.sqrt((k + 1) * m / (k + 2))
    J[n - 1] = math.sqrt(m / n)
    return J, np.linalg.inv(J)[:, :n - 1]


def _cluster_paths(n, m, unit, k, N, rng):
    """k walkers of n atoms on a sphere, the closest pair 3 to 5 Angstrom apart, 0.1 Angstrom of
    noise per slice; Jacobi coordinates in units of `unit` Angstrom, DOF-major."""
    i = np.arange(n) + 0.5
    z = 1.0 - 2.0 * i / n
    r, phi = np.sqrt(1.0 - z * z), np.pi * (1.0 + math.sqrt(5.0)) * i
    p = np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)
    p /= min(np.linalg.norm(p[a] - p[b]) for a in range(n) for b in range(a))
    q = np.linalg.qr(rng.standard_normal((k, 3, 3)))[0]
    pos = np.einsum("kxy,ay->kax", q, p) * rng.uniform(3.0, 5.0, (k, 1, 1)) / unit
    x = np.einsum("ia,kax->kix", _jacobi(n, m)[0], pos)[:, :n - 1].reshape(k, 3 * (n - 1), 1)
    return x + rng.normal(0.0, 0.1 * math.sqrt(m) / unit, (k, 3 * (n - 1), N))


def _mass_and_unit(c):
    return (1.0, 0.8988882118208078) if c["system"] == "he3part" else (HE_MASS_KELVIN, 1.0)


def _templates(c, seed):
    """Starting walkers, [k][DOF][N] float64; walker w starts as template w mod k."""
    rng = np.random.RandomState(seed)
    if c["system"] == "ho":
        return rng.normal(0.0, 0.7, (c["walkers"], 1, 1)) + rng.normal(0.0, 0.1, (c["walkers"], 1, c["N"]))
    k = min(c["walkers"], 64 if c["n"] > 5 else 512)
    return _cluster_paths(c["n"], *_mass_and_unit(c), k, c["N"], rng)


def _dof(c):
    return 1 if c["system"] == "ho" else 3 * (c["n"] - 1)


def _threads(c):
    return 1 if c["kind"] == "moves" else c["N"] >> c["S"]


def _xorshift_rows(rows, seed):
    return np.random.RandomState(seed).randint(0, 2 ** 31 - 1, size=(rows, 4)).astype(np.uint32)


def _system(c):
    from feynsimul_gb300.physical_systems.harm_osc import HarmOsc
    from feynsimul_gb300.physical_systems.lm2m2 import Lm2m2Cluster
    from feynsimul_gb300.physical_systems.lm2m2_3part import Lm2m2_3part
    if c["system"] == "ho":
        s = HarmOsc()
        return s, (s.energyOp,), ("x1",)
    s = Lm2m2_3part() if c["system"] == "he3part" else Lm2m2Cluster(c["n"], 1.0 / c["beta"])
    ops = (s.energyOp, s.meanSquaredRadiusOp) if c["system"] == "he3part" else (s.energyOp,)
    return s, ops, (" + ".join("x%d * x%d" % (d + 1, d + 1) for d in range(s.DOF)),)


def _network(dof, seed):
    rng = np.random.RandomState(seed)
    parts = []
    for out, inp, scale in ((128, 16, 1.0), (128, 128, 1.0), (128, 128, 1.0), (16, 128, 0.05)):
        parts += [scale * math.sqrt(2.0 / inp) * rng.randn(out * inp), 0.05 * scale * rng.randn(out)]
    return np.concatenate(parts).astype(np.float32)


def _train_data(c, seed):
    rng = np.random.RandomState(seed)
    n, d = c["rows"] + c["held_out"], c["dof"]
    x = np.zeros((n, 16), np.float32)
    x[:, :d] = rng.randn(n, d)
    x[:, d:2 * d] = 0.2 * rng.randn(n, d)
    z = np.zeros((n, 8), np.float32)
    z[:, :d] = 0.5 * np.tanh(x[:, :d]) + (0.6 + 0.2 * np.cos(x[:, :d])) * rng.randn(n, d)
    return x, z


def _workload(c):
    """The batch's systems: atoms, slices, temperature and walkers of each."""
    rng = np.random.RandomState(c["layout"])
    out = []
    for _ in range(c["systems"]):
        out.append({"n": int(rng.randint(3, c["atoms"] + 1)), "N": int(2 ** rng.randint(7, int(math.log2(c["slices"])) + 1)),
                    "T": float(rng.uniform(0.5, 2.0)), "walkers": int(rng.randint(max(8, c["walkers"] // 8), c["walkers"] + 1))})
    return out


def _batch_inputs(c, w, S, seed):
    rng = np.random.RandomState(seed)
    k = min(w["walkers"], 32)
    t = _cluster_paths(w["n"], HE_MASS_KELVIN, 1.0, k, w["N"], rng).astype(np.float32)
    paths = t[np.arange(w["walkers"]) % k]
    return paths, _xorshift_rows(w["walkers"] * (w["N"] >> S), seed + 1), _xorshift_rows(w["walkers"], seed + 2)


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "train":
        from feynsimul_gb300.learned import LearnedProposal
        x, z = _train_data(c, seed)
        m = LearnedProposal(c["dof"], 0.25, 5.0, params=_network(c["dof"], seed))
        return {"case": c, "model": m, "x": x[:c["rows"]], "z": z[:c["rows"]], "held_out": x[c["rows"]:]}
    if c["kind"] == "batch":
        from feynsimul_gb300.batch import BatchSampler
        load = _workload(c)
        b = BatchSampler(load, op_runs=1, msteps=4, block_threads=c["block"], tpw_target=c["target"], seed=seed)
        for i, w in enumerate(load):
            p, t, g = _batch_inputs(c, w, b.systems[i].bisection_level, seed * 1000 % 2 ** 30 + 10 * i)
            b.set_state(i, p.reshape(w["walkers"], -1), t, g)
        return {"case": c, "batch": b}
    from feynsimul_gb300.kernel import PIMCKernel
    from feynsimul_gb300.kernel_args import KernelArgs
    s, ops, cors = _system(c)
    moves = c["kind"] == "moves"
    more = {}
    if c["histogram"]:
        more.update(histograms=s.pairDistanceOps, histRange=(0.0, 20.0), histBins=200)
    if moves:
        more.update(alpha=0.5, PSAlpha=0.5)
    ka = KernelArgs(
        system=s, nbrOfWalkers=c["walkers"], N=c["N"], beta=float(c["beta"]), S=c["S"], enableOperator=True,
        enableCorrelator=c["correlator"], enableBisection=True, enablePathShift=moves, enableSingleNodeMove=moves,
        enableBins=False, nbrOfWalkersPerWorkGroup=c["per_group"], enableParallelizePath=not moves,
        enableGlobalPath=c["global_path"], enableGlobalOldPath=False, enableDouble=c["double"],
        enableRanlux=c["luxury"] >= 0, luxuaryFactor=max(c["luxury"], 0), ranluxIntMax=2 ** 32 - 1, operators=ops,
        correlators=cors if c["correlator"] else None, operatorRuns=c["opruns"], metroStepsPerOperatorRun=c["msteps"],
        accumulation=c["accumulation"], partials=c["partials"], fastMath=c["fast"], walkersPerBlock=c["per_block"],
        minBlocksPerSM=c["blocks_per_sm"], learnedProposal=c["kind"] == "learned", seed=seed % 2 ** 31, **more)
    k = PIMCKernel(ka)
    if c["luxury"] >= 0:
        k.initRanlux()
        k.groupInitRanlux()
    t = _templates(c, seed).astype(np.float64 if c["double"] else np.float32)
    t = t.reshape(t.shape[0], -1)
    state = {"case": c, "kernel": k}
    if c["kind"] == "learned":
        from feynsimul_gb300.learned import LearnedProposal, sigma_level
        k.setLearnedProposal(LearnedProposal(_dof(c), sigma_level(float(c["beta"]), c["N"], c["S"], 1), 5.0,
                                             params=_network(_dof(c), seed)))
    if c["kind"] == "host":
        state["paths"] = torch.from_numpy(t[np.arange(c["walkers"]) % t.shape[0]]).pin_memory().numpy()
        state["out"] = torch.empty(c["walkers"], t.shape[1], dtype=torch.float32).pin_memory().numpy()
    else:
        k.setPathsTiled(t)
    return state


def run(state):
    c = state["case"]
    if c["kind"] == "train":
        m = state["model"]
        losses = m.train(state["x"], state["z"], steps=c["steps"], batch=c["batch"], lr=1e-3, seed=7)
        return {"losses": losses, "params": m.params, "predictions": m.predict(state["held_out"])}
    if c["kind"] == "batch":
        b = state["batch"]
        b.run(1)
        ids = range(len(b.workload))
        return {"energies": np.concatenate([b.energy_sums(i) for i in ids]),
                "accepts": np.concatenate([b.accepts(i) for i in ids])}
    k = state["kernel"]
    out = {}
    if c["kind"] == "host":
        out["paths"] = k.runHost(state["paths"], state["out"])
    else:
        k.run()
    out["operators"] = k.getOperatorsStudy() if c["accumulation"] == "study" else k.getOperators()
    out["accepts"] = k.getAccepts()
    if c["correlator"]:
        out["correlator"] = k.getCorrelatorMoments()
    if c["histogram"]:
        out["histogram"] = k.getHistogram(density=False)[1].astype(np.int64)
    if c["paths"]:
        out["paths"] = k.getPaths()
    return out


# ------------------------------------------------------------------ the work
def _pair_flops(n):
    return {1: 3}.get(n, 9 * n * n + 35 * n * (n - 1) // 2)


def _sweep_work(n, dof, walkers, N, S, steps, measured, luxury, elem, correlator, moves=False):
    T = 1 if moves else N >> S
    nodes = walkers * T * (2 ** S - 1) * steps
    p = {-1: 8, 0: 3 + 8, 1: 6 + 8, 2: 28 + 8, 3: 50 + 8}[luxury]
    flops = nodes * (2 * dof * p + 9 * dof + _pair_flops(n)) + walkers * N * measured * 2 * _pair_flops(n)
    if moves:
        flops += walkers * steps * (N // 2) * 2 * _pair_flops(n)
    if correlator:
        flops += walkers * measured * (N // 2) * N * 2
    rows = walkers * (T + 1) * (112 if luxury >= 0 else 16)
    return {"bytes": 2 * walkers * dof * N * elem + 2 * rows + walkers * T * 12 + (walkers * N * 8 if correlator else 0),
            "flops": flops}


def work(case):
    c = case
    if c["kind"] == "train":
        per = 16 * 128 + 2 * 128 * 128 + 128 * 16
        params = per + 3 * 128 + 16
        rows = min(c["batch"], c["rows"])
        return {"bytes": c["steps"] * (rows * 96 + params * 4 * 7) + c["held_out"] * 128,
                "flops": c["steps"] * rows * 6 * per + c["held_out"] * 2 * per}
    if c["kind"] == "batch":
        total = {"bytes": 0, "flops": 0}
        for w in _workload(c):
            one = _sweep_work(w["n"], 3 * (w["n"] - 1), w["walkers"], w["N"], 4, 4, 1, -1, 4, False)
            total = {k: total[k] + one[k] for k in total}
        return total
    w = _sweep_work(c["n"], _dof(c), c["walkers"], c["N"], c["S"], c["opruns"] * c["msteps"], c["opruns"], c["luxury"],
                    8 if c["double"] else 4, c["correlator"], c["kind"] == "moves")
    if c["kind"] == "learned":
        w["flops"] += c["walkers"] * _threads(c) * c["opruns"] * c["msteps"] * 2 * (16 * 128 + 2 * 128 * 128 + 128 * 16)
    return w


# ------------------------------------------------------------------ 64-bit results
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Xorshift:
    """xorshift128 rows [n][4]; next() gives 32-bit integers, uniform() values in [0, 1)."""

    def __init__(self, rows):
        self.s = [torch.from_numpy(rows[:, i].astype(np.int64)).to(_device()) for i in range(4)]

    def next(self):
        x, y, z, w = self.s
        t = x ^ ((x << 11) & 0xFFFFFFFF)
        w2 = w ^ (w >> 19) ^ t ^ (t >> 8)
        self.s = [y, z, w, w2]
        return w2

    def uniform(self):
        return self.next().double() * 2.0 ** -32

    def below(self, n):
        return self.next() & (n - 1)


class _Ranlux:
    """24-bit subtract-with-borrow (lags 10 and 24) that drops `skip` steps after every 24
    values, seeded from 64-bit integers; `wide` joins two values to one of 48 bits."""

    def __init__(self, xs, skip, wide):
        x = xs.astype(np.uint64)
        lags = []
        for _ in range(3):
            words = []
            for _ in range(3):
                x = x ^ (x << np.uint64(13))
                x = x ^ (x >> np.uint64(7))
                x = x ^ (x << np.uint64(17))
                words.append(x)
            for b in range(8):  # 24 bits each of the 192, most significant first
                at, off = divmod(24 * b, 64)
                v = (words[at] << np.uint64(off)) >> np.uint64(40)
                if off > 40:
                    v = v | (words[at + 1] >> np.uint64(104 - off))
                lags.append(v & np.uint64(0xFFFFFF))
        self.s = [torch.from_numpy(v.astype(np.int64)).to(_device()) for v in lags]
        self.c = (self.s[23] == 0).long()
        self.at, self.out, self.skip, self.wide = 0, 0, skip, wide
        for _ in range(32 * 24):
            self._step()

    def _step(self):
        a = 23 - self.at
        d = self.s[(a + 10) % 24] - self.s[a] - self.c
        self.c = (d < 0).long()
        self.s[a] = d & 0xFFFFFF
        self.at = (self.at + 1) % 24
        return a

    def _one(self):
        a = self._step()
        v = self.s[a]
        f = v.double() * 2.0 ** -24 + torch.where(v < 4096, self.s[(a + 9) % 24].double() * 2.0 ** -48, 0.0)
        self.out += 1
        if self.out == 24:
            self.out = 0
            for _ in range(self.skip):
                self._step()
        return torch.where(f == 0, 2.0 ** -48, f)

    def uniform(self):
        if not self.wide:
            return self._one()
        a, b = self._one(), self._one()
        return torch.where(a == 2.0 ** -48, 0.0, a) + b / 16777216.0

    def below(self, n):
        return (self.uniform() * n).long() & (n - 1)


def _lm2m2(r2):
    """The LM2M2 pair potential in Kelvin and r^2 dV/d(r^2), r in Angstrom."""
    x = torch.sqrt(r2) / 2.9695
    c6, c8, c10 = 1.34687065, 0.41308398, 0.17060159
    rat = c6 / x ** 6 + c8 / x ** 8 + c10 / x ** 10
    drat = -6 * c6 / x ** 7 - 8 * c8 / x ** 9 - 10 * c10 / x ** 11
    q = torch.clamp(1.4088 / x - 1.0, min=0.0)
    F = torch.exp(-q * q)
    dF = F * 2.0 * q * 1.4088 / x ** 2
    near = r2 <= 0.0005 ** 2
    rat, drat = torch.where(near, 0.0, rat), torch.where(near, 0.0, drat)
    base = 1.89635353e5 * torch.exp(-10.70203539 * x - 1.90740649 * x * x)
    B = 2 * math.pi / (1.454790369 - 1.003535949)
    win = (x >= 1.003535949) & (x <= 1.454790369)
    w = B * (x - 1.003535949)
    v = base - F * rat + torch.where(win, 0.0026 * (1 - torch.cos(w)), 0.0)
    dv = base * (-10.70203539 - 2 * 1.90740649 * x) - F * drat - dF * rat + torch.where(win, 0.0026 * B * torch.sin(w), 0.0)
    return 10.97 * v, 10.97 * dv * x / 2


def _physics(c):
    """V of coordinates [..., DOF] and the operators' values, in the system's units."""
    if c["system"] == "ho":
        return (lambda x: 0.5 * x[..., 0] ** 2), (lambda x: [x[..., 0] ** 2])
    n = c["n"]
    m, unit = _mass_and_unit(c)
    scale = 8.6173324e-5 * 773.633685978724 if c["system"] == "he3part" else 1.0
    to_pos = torch.from_numpy(_jacobi(n, m)[1] * unit).to(_device())
    pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]

    def both(x):
        p = torch.einsum("ai,...ix->...ax", to_pos, x.reshape(*x.shape[:-1], n - 1, 3))
        v, vir = 0.0, 0.0
        for a, b in pairs:
            u, d = _lm2m2(((p[..., a, :] - p[..., b, :]) ** 2).sum(-1))
            v, vir = v + u, vir + d
        return scale * v, scale * vir

    def operators(x):
        v, vir = both(x)
        return [v + vir] + ([(x * x).sum(-1) / n] if c["system"] == "he3part" else [])

    return (lambda x: both(x)[0]), operators


def _sample(c, paths, threads, offsets):
    """The Metropolis-bisection sweeps of one run in 64 bits: paths [walkers][DOF][N] and the
    streams of the segment threads [walkers * T] and of the walkers.  Gives the paths, the
    operators' sums per walker and the correlator sums per walker and lag."""
    dev = _device()
    N, S, W = c["N"], c["S"], paths.shape[0]
    seg, T, eps = 2 ** S, N >> S, c["beta"] / N
    V, operators = _physics(c)
    x = torch.from_numpy(np.ascontiguousarray(paths.astype(np.float64).transpose(0, 2, 1))).to(dev)  # [W][N][DOF]
    dof = x.shape[2]
    rows = torch.arange(W, device=dev)[:, None]
    base = torch.arange(T, device=dev)[None, :] * seg
    sums, cor = None, torch.zeros(W, N // 2, dtype=torch.float64, device=dev)
    for _ in range(c["opruns"]):
        for _ in range(c["msteps"]):
            start = base + offsets.below(seg)[:, None]
            at = [(start + i) & (N - 1) for i in range(seg + 1)]
            node = [x[rows, a] for a in at]  # [W][T][DOF] each
            new = list(node)
            for n in range(1, S + 1):
                half = seg >> n
                sig = math.sqrt(seg * eps / (2.0 * 2 ** n))
                for m in range(half, seg, 2 * half):
                    z = []
                    for _ in range(dof):
                        u, v = threads.uniform(), threads.uniform()
                        z.append(torch.where(v > 0, torch.sqrt(-2.0 * torch.log(v)) * torch.sin(2 * math.pi * u), 0.0))
                    new[m] = 0.5 * (new[m - half] + new[m + half]) + sig * torch.stack(z, -1).reshape(W, T, dof)
            d = 0.0
            for m in range(1, seg):
                d = d + eps * (V(node[m]) - V(new[m]))
            take = ~(torch.exp(d) < threads.uniform().reshape(W, T))
            for m in range(1, seg):
                x[rows, at[m]] = torch.where(take[..., None], new[m], node[m])
        values = torch.stack([o.sum(1) for o in operators(x)])
        sums = values if sums is None else sums + values
        if c["correlator"]:
            f = x[..., 0] if c["system"] == "ho" else (x * x).sum(-1)
            for t in range(N // 2):
                cor[:, t] += (f * torch.roll(f, -t, 1)).sum(1)
    return x.permute(0, 2, 1).reshape(W, -1), sums, cor


def _streams(c, seed):
    """The generator rows that a kernel with this master seed draws for itself."""
    rs = np.random.RandomState(seed % 2 ** 31)
    W, n = c["walkers"], c["walkers"] * _threads(c)
    if c["luxury"] < 0:
        rows = rs.randint(0, high=2 ** 31 - 1, size=(n + 1, 4)).astype(np.uint32)
        w, t = np.divmod(np.arange(n), _threads(c))
        groups = W // c["per_group"]
        ids = (w // c["per_group"]) * _threads(c) + t + (w % c["per_group"]) * groups * _threads(c)
        return _Xorshift(rows[ids]), _Xorshift(rs.randint(0, high=2 ** 31 - 1, size=(W, 4)).astype(np.uint32))
    s = int(rs.randint(0, high=2 ** 31 - 1, size=n + 1)[0])
    skip = {0: 24, 1: 76, 2: 200, 3: 380}[c["luxury"]]
    w, t = np.divmod(np.arange(n), _threads(c))
    ids = (w // c["per_group"]) * _threads(c) + t + (w % c["per_group"]) * (W // c["per_group"]) * _threads(c)
    return (_Ranlux((np.uint64(s) << np.uint64(32)) + ids.astype(np.uint64), skip, c["double"]),
            _Ranlux((np.uint64(s ^ 0x80000000) << np.uint64(32)) + np.arange(W, dtype=np.uint64), skip, c["double"]))


def _exact_train(c, seed):
    if not torch.cuda.is_available():
        return None  # the batches are drawn by the device's generator
    dev = _device()
    x, z = (torch.from_numpy(v).to(dev).double() for v in _train_data(c, seed))
    held = x[c["rows"]:]
    flat = torch.from_numpy(_network(c["dof"], seed)).to(dev).double().requires_grad_()
    shapes = [(128, 16), (128,), (128, 128), (128,), (128, 128), (128,), (16, 128), (16,)]

    def net(v):
        p = torch.split(flat, [math.prod(s) for s in shapes])
        for i in range(0, 8, 2):
            v = v @ p[i].reshape(shapes[i]).T + p[i + 1]
            v = torch.relu(v) if i < 6 else v
        return v

    gen = torch.Generator(device=dev)
    gen.manual_seed(7)
    d, batch = c["dof"], min(c["batch"], c["rows"])
    m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    for it in range(1, c["steps"] + 1):
        idx = torch.randint(0, c["rows"], (batch,), device=dev, generator=gen)
        y = net(x[idx])
        s = 4.0 * torch.tanh(0.25 * y[:, d:2 * d])
        loss = (0.5 * (z[idx, :d] - y[:, :d]) ** 2 * torch.exp(-s) + 0.5 * s).sum() / batch
        (g,) = torch.autograd.grad(loss, flat)
        losses.append(loss.detach())
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            flat -= 1e-3 * (m / (1 - 0.9 ** it)) / (torch.sqrt(v / (1 - 0.999 ** it)) + 1e-8)
    with torch.no_grad():
        return {"losses": torch.stack(losses), "params": flat.detach(), "predictions": net(held)}


def _exact_batch(c, seed):
    sums = []
    for i, w in enumerate(_workload(c)):
        S = _batch_level(c, w)
        p, t, g = _batch_inputs(c, w, S, seed * 1000 % 2 ** 30 + 10 * i)
        one = dict(SWEEP, system="he", n=w["n"], walkers=w["walkers"], N=w["N"], S=S, opruns=1, msteps=4, beta=1.0 / w["T"])
        sums.append(_sample(one, p, _Xorshift(t), _Xorshift(g))[1][0])
    return {"energies": torch.cat(sums), "accepts": None}


def _batch_level(c, w):
    """The bisection level that a sampler of this CTA size and thread target gives a system."""
    S = max(1, min(int(math.log2(w["N"])) - int(math.log2(c["target"])), 10))
    most = max(1, 200 * 1024 // (3 * (w["n"] - 1) * (w["N"] + w["N"] // 8) * 4 + 512))
    if most * (w["N"] >> S) < c["block"]:
        T = min(2 ** int(math.log2(max(1, c["block"] // most))), w["N"] // 4)
        S = min(S, max(1, int(math.log2(w["N"] // T))))
    while (w["N"] >> S) > c["block"]:
        S += 1
    return S


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "train":
        return _exact_train(c, seed)
    if c["kind"] == "batch":
        return _exact_batch(c, seed)
    if c["kind"] in ("moves", "learned"):
        return None  # sequential moves, and a 16-bit network in every proposal
    t = _templates(c, seed)
    if not c["double"]:
        t = t.astype(np.float32)
    x, sums, cor = _sample(c, t[np.arange(c["walkers"]) % t.shape[0]], *_streams(c, seed))
    ops = sums / (c["opruns"] * c["N"])
    study = c["accumulation"] == "study"
    out = {"operators": torch.stack([ops] * 3) if study else ops, "accepts": None}
    if c["correlator"]:
        f = 1.0 / (c["opruns"] * c["N"])
        mean, sd = (cor * f).mean(0)[None], (cor * f).std(0, correction=0)[None] / math.sqrt(c["walkers"])
        out["correlator"] = (torch.stack([mean] * 3), torch.stack([sd] * 3)) if study else (mean, sd)
    if c["histogram"]:
        out["histogram"] = None
    if c["paths"] or c["kind"] == "host":
        out["paths"] = x
    return out
