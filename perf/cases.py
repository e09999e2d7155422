"""What a user of this framework has it compute, as cases that can be timed and checked.

Each case is one call (or the few calls that belong together) through the public entry points:
the drop-in calculator and driver, a single chain, batches of chains at several sizes and species
counts, the tempering ladder, the uneven ternary batch, and the full correlation-function
recompute.  Systems, sizes and launch shapes are those of the benchmark workloads and the tests;
``draw`` spreads them over the range between.
"""
import math
from functools import lru_cache

import numpy as np
import torch

from cemc_gb300 import engine as E
from cemc_gb300.batch import BatchRunner, MultiBatchRunner, fold_chemical_potential
from cemc_gb300.calculator import CE, SimpleAtoms
from cemc_gb300.lattice import fcc_settings, hcp_settings, seeded_ecis
from cemc_gb300.mcmc import Montecarlo, SGCMonteCarlo
from cemc_gb300.parallel_tempering import ParallelTempering
from cemc_gb300.tables import CEModel

KB = 8.6173303e-5
SPECIES = ["Al", "Mg", "Si"]
# Cluster recipes (pair, triplet, quadruplet shells): the headline batch's, the tempering ladder's,
# the ternary batch's and a small one for HCP cells.
RECIPES = {"binary": (4, 2, 1), "binary6": (6, 2, 1), "ternary": (5, 3, 1), "hcp3": (2, 1, 1)}


def listed():
    return [
        # The drop-in calculator inside a user's own Monte Carlo loop: propose a swap, read the energy
        # and correlation functions, take it back.  Latency of the smallest calls.
        {"name": "calculator_swap_256", "kind": "calculator", "system": "binary", "L": 4},
        {"name": "calculator_swap_ternary_4000", "kind": "calculator", "system": "ternary", "L": 10},
        # The drop-in driver on a cell of the size its users run interactively (runMC with its energy-bias
        # probing and thermodynamic averages), reference precision.
        {"name": "driver_sgc_256", "kind": "driver", "system": "binary", "L": 4, "move": "flip", "steps": 10000},
        # One canonical chain in FP64, the reference's plain single-chain run.
        {"name": "chain_swap_2048_fp64", "kind": "chain", "system": "binary", "L": 8, "chains": 1, "move": "swap",
         "precision": "fp64", "sweeps": 10},
        # Several translation-symmetry groups, three species, reference precision: a small HCP batch.
        {"name": "chain_flip_hcp_4x1000_fp64", "kind": "chain", "system": "hcp3", "L": 10, "chains": 4, "move": "flip",
         "precision": "fp64", "sweeps": 10},
        # The headline batch: a T x mu grid of semi-grand-canonical chains, 10 sweeps and the drift reset a
        # step, in the launch shape the autotuner picks for it.
        {"name": "batch_sgc_64x16384", "kind": "batch", "system": "binary", "L": 16, "chains": 64, "move": "flip",
         "warps": 8, "kernel": 6, "sweeps": 10},
        # Many small cells (more chains than SMs), default form and width: scans over temperature.
        {"name": "batch_sgc_200x864", "kind": "batch", "system": "binary", "L": 6, "chains": 200, "move": "flip",
         "warps": 4, "kernel": 0, "sweeps": 20},
        # Ternary semi-grand-canonical chains of an ordinary size.
        {"name": "batch_sgc_ternary_32x4000", "kind": "batch", "system": "ternary", "L": 10, "chains": 32,
         "move": "flip", "warps": 16, "kernel": 0, "sweeps": 4},
        # The tempering ladder: 48 replicas of the largest cell, one sweep and one exchange.
        {"name": "ladder_swap_48x131072", "kind": "ladder", "system": "binary6", "L": 32, "chains": 48, "sweeps": 1},
        # Ternary canonical chains of uneven cells stepped by one graph launch.
        {"name": "uneven_swap_ternary_64", "kind": "uneven", "system": "ternary", "Lmin": 4, "Lmax": 24, "sizes": 8,
         "chains": 64, "sweeps": 1},
        # The full FP64 recompute alone: drift reset and validation of large batches.
        {"name": "recompute_48x131072", "kind": "recompute", "system": "binary6", "L": 32, "chains": 48},
        {"name": "recompute_ternary_32x13500", "kind": "recompute", "system": "ternary", "L": 15, "chains": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calculator", "driver", "chain", "batch", "batch", "ladder", "uneven", "recompute"])
    if kind == "calculator":
        return {"kind": kind, "system": rng.choice(["binary", "ternary"]), "L": rng.randint(4, 15)}
    if kind == "driver":
        return {"kind": kind, "system": "binary", "L": rng.randint(4, 8), "move": rng.choice(["flip", "swap"]),
                "steps": _log_int(rng, 1000, 20000)}
    if kind == "chain":
        system = rng.choice(["binary", "binary", "ternary", "hcp3"])
        return {"kind": kind, "system": system, "L": rng.randint(4, 12), "chains": rng.randint(1, 6),
                "move": rng.choice(["flip", "swap"]), "precision": rng.choice(["fp64", "fp32"]),
                "sweeps": rng.randint(1, 6)}
    if kind == "batch":
        system, move = rng.choice([("binary", "flip"), ("binary", "flip"), ("binary", "swap"), ("ternary", "flip")])
        return {"kind": kind, "system": system, "L": rng.randint(5, 18 if system == "binary" else 12),
                "chains": _log_int(rng, 4, 160), "move": move, "warps": rng.choice([4, 8, 12, 16]),
                "kernel": rng.choice([0, 6]) if (system, move) == ("binary", "flip") else 0,
                "sweeps": rng.randint(1, 4)}
    if kind == "ladder":
        return {"kind": kind, "system": rng.choice(["binary", "binary6"]), "L": rng.randint(8, 26),
                "chains": rng.randint(8, 48), "sweeps": 1}
    if kind == "uneven":
        return {"kind": kind, "system": "ternary", "Lmin": rng.randint(4, 6), "Lmax": rng.randint(8, 20),
                "sizes": rng.randint(2, 5), "chains": rng.randint(12, 60), "sweeps": 1}
    system = rng.choice(["binary", "binary6", "ternary", "hcp3"])
    return {"kind": kind, "system": system, "L": rng.randint(5, 24 if system.startswith("binary") else 13),
            "chains": _log_int(rng, 1, 40)}


# ---- systems: the settings, model and device tables a program builds once ------------------------

@lru_cache(maxsize=None)
def _settings(system, L):
    if system == "hcp3":
        return hcp_settings(L, max(4, L - 6) | 1, *RECIPES[system], SPECIES)
    return fcc_settings(L, *RECIPES[system], SPECIES[:3 if system == "ternary" else 2])


@lru_cache(maxsize=None)
def _geometry(system, L):
    s = _settings(system, L)
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    return s, eci, m, E.Geometry(m, "cuda")


@lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


def _uneven_sizes(case):
    lo, hi, k = case["Lmin"], case["Lmax"], case["sizes"]
    sizes = sorted({int(round(lo + (hi - lo) * i / max(1, k - 1))) for i in range(k)})
    each = [case["chains"] // len(sizes) + (i < case["chains"] % len(sizes)) for i in range(len(sizes))]
    return [(L, n) for L, n in zip(sizes, each) if n]


def _occupations(m, n, seed, move):
    """Flips: random species on every site.  Swaps: a shuffled, slightly uneven composition per chain."""
    rng = np.random.default_rng(seed)
    if move == "flip":
        return rng.integers(0, m.n_sym, (n, m.n_sites)).astype(np.int8)
    occ = np.empty((n, m.n_sites), dtype=np.int8)
    for c in range(n):
        share = rng.dirichlet([8.0] * m.n_sym)
        counts = np.maximum(2, np.floor(share * m.n_sites).astype(int))
        counts[np.argmax(counts)] += m.n_sites - counts.sum()
        occ[c] = rng.permutation(np.repeat(np.arange(m.n_sym), counts))
    return occ


def _move(case):
    return E.MOVE_FLIP if case.get("move", "swap") == "flip" else E.MOVE_SWAP


def _temperatures(n):
    return np.linspace(300.0, 1200.0, n) if n > 1 else np.array([800.0])


def _mu(c):
    return -0.2 + 0.4 * ((3 * c) % 8) / 7.0


def _ecis(m, eci, n, move):
    """One row per chain; flips carry a chemical potential between -0.2 and 0.2 eV in the singlet ECI."""
    if move == "flip":
        return fold_chemical_potential(m, m.eci_vector(eci), [_mu(c) for c in range(n)])
    return np.repeat(m.eci_vector(eci)[None], n, 0)


def _ternary_shape(m):
    """(warps, CTAs per chain) of a ternary swap batch, as the uneven benchmark workload chooses them."""
    if m.n_sites >= 16384:
        return 16, 2
    return max(2, min(16, max(4, m.n_sites // (4 * m.n_cols)))), 1


# ---- the cases ----------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "uneven":
        runners = []
        for L, n in _uneven_sizes(case):
            _, eci, m, geo = _geometry(case["system"], L)
            warps, cluster = _ternary_shape(m)
            runners.append(BatchRunner(geo, _occupations(m, n, [seed, L], "swap"), m.eci_vector(eci), 800.0,
                                       E.MOVE_SWAP, seed=seed + L, warps=warps, cluster=cluster,
                                       sweeps_per_step=case["sweeps"]))
        multi = MultiBatchRunner(runners)
        multi.capture()
        return {"case": case, "multi": multi}
    s, eci, m, geo = _geometry(case["system"], case["L"])
    if kind in ("calculator", "driver"):
        occ = _occupations(m, 1, seed, "swap")[0]
        atoms = SimpleAtoms(m.symbols_of(occ))
        calc = CE(atoms, s, eci=dict(eci))
        atoms.set_calculator(calc)
        if kind == "driver":
            driver = SGCMonteCarlo if case["move"] == "flip" else Montecarlo
            return {"case": case, "mc": driver(atoms, 800.0, seed=seed), "calc": calc}
        a, b = _calculator_sites(occ, seed)
        return {"case": case, "calc": calc, "atoms": atoms,
                "changes": [(a, atoms[a].symbol, atoms[b].symbol), (b, atoms[b].symbol, atoms[a].symbol)]}
    n = case["chains"]
    if kind == "ladder":
        occ = _occupations(m, 1, seed, "swap")[0]
        return {"case": case, "pt": ParallelTempering(geo, occ, m.eci_vector(eci),
                                                      temperatures=np.geomspace(200.0, 1500.0, n), seed=seed,
                                                      warps=16)}
    if kind == "recompute":
        occ = _occupations(m, n, seed, "flip")
        return {"case": case, "cb": E.ChainBatch(geo, occ, _ecis(m, eci, n, "swap"), KB * 800.0, E.MOVE_FLIP, seed=1)}
    occ = _occupations(m, n, seed, case["move"])
    ev = _ecis(m, eci, n, case["move"])
    if kind == "chain":
        return {"case": case, "cb": E.ChainBatch(geo, occ, ev, KB * _temperatures(n), _move(case), seed=seed)}
    runner = BatchRunner(geo, occ, ev, _temperatures(n), _move(case), seed=seed, warps=case["warps"], cluster=1,
                         kernel=case["kernel"], sweeps_per_step=case["sweeps"], stream=_stream())
    runner.capture()
    return {"case": case, "runner": runner}


def _calculator_sites(occ, seed):
    """Two sites of different species."""
    rng = np.random.default_rng([seed, 1])
    a = int(rng.integers(len(occ)))
    other = np.nonzero(occ != occ[a])[0]
    return a, int(other[rng.integers(len(other))])


def _chain_outputs(cb):
    out = {"occ": cb.occ, "cf": cb.cf, "energy": cb.energy, "trial": cb.trial,
           "sums": cb.accum[:, :E.A_NSAMP], "counts": cb.accum[:, E.A_NSAMP:].view(torch.int64)}
    if cb.trk is not None:
        out["site_lists"] = cb.trk
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "calculator":
        calc = state["calc"]
        energy = calc.calculate(state["atoms"], ["energy"], state["changes"])
        cf = calc.get_cf()
        calc.undo_changes()
        return {"energy": energy, "cf": np.array(list(cf.values())), "energy_back": calc.get_energy()}
    if kind == "driver":
        mc, calc = state["mc"], state["calc"]
        if case["move"] == "flip":
            mc.runMC(steps=case["steps"], chem_potential={"c1_0": -0.05}, equil=False)
        else:
            mc.runMC(steps=case["steps"], equil=False)
        thermo = {k: v for k, v in mc.get_thermodynamic().items() if not isinstance(v, str)}
        return {"thermo": thermo, "occ": calc.updater.occupation(), "cf": np.array(list(calc.get_cf().values())),
                "energy": calc.get_energy()}
    if kind == "chain":
        cb = state["cb"]
        cb.run(int(case["sweeps"]) * cb.geo.n_sites,
               precision=E.PREC_F64 if case["precision"] == "fp64" else E.PREC_F32)
        return _chain_outputs(cb)
    if kind == "batch":
        state["runner"].step()
        return _chain_outputs(state["runner"].cb)
    if kind == "ladder":
        pt = state["pt"]
        pt.run(sweeps_per_cycle=float(case["sweeps"]), num_exchange_cycles=1)
        return dict(_chain_outputs(pt.cb), kT=pt.cb.kT, replica_of=pt.replica_of)
    if kind == "uneven":
        state["multi"].step()
        return [_chain_outputs(r.cb) for r in state["multi"].runners]
    cb = state["cb"]
    cb.recompute()
    return {"cf": cb.cf, "energy": cb.energy}


def work(case):
    """Chain state read and written once; one multiply-add per cluster term of each changed site."""
    kind = case["kind"]
    if kind == "uneven":
        parts = [(L, n) for L, n in _uneven_sizes(case)]
    else:
        parts = [(case["L"], case.get("chains", 1))]
    total = {"bytes": 0.0, "flops": 0.0}
    for L, n in parts:
        s = _settings(case["system"], L)
        t = _terms(case["system"], L)
        per_site = sum(len(g["eci"]) for g in t["groups"]) / len(t["groups"])
        N, K = s.n_sites, len(t["names"])
        if kind == "recompute":
            total["bytes"] += n * (N + 24.0 * K)
            total["flops"] += 2.0 * n * N * per_site
            continue
        if kind == "calculator":
            total["bytes"] += 2 * (per_site / 2.0 + 8.0 * K)
            total["flops"] += 2 * 2.0 * per_site
            continue
        trials = n * (case["steps"] + 1001.0 if kind == "driver" else case["sweeps"] * float(N))
        swap = case.get("move", "swap") == "swap"
        total["bytes"] += n * (2.0 * N + 48.0 * K + 300.0 + (16.0 * N if swap else 0.0))
        total["flops"] += trials * 2.0 * per_site * (2 if swap else 1)
    return total


# ---- 64-bit values in plain numpy / torch ---------------------------------------------------------

@lru_cache(maxsize=None)
def _terms(system, L):
    """The cluster products of a site, from the settings object: per translation group and (ECI,
    equivalent decoration, sub-cluster) the decoration of the site and the (column, decoration) of
    the other members (column -1: absent), and per ECI the increment and full-sum weights."""
    s = _settings(system, L)
    names = sorted(n.name for n in s.cset.eci_names)
    symbols = sorted(s.unique_elements)
    bf = np.array([[float(b[x]) for x in symbols] for b in s.basis_functions])
    col = {int(c): i for i, c in enumerate(s.column_sites.tolist())}
    sizes = [len(g) for g in s.index_by_trans_symm]
    group = np.zeros(s.n_sites, dtype=np.int64)
    for g, sites in enumerate(s.index_by_trans_symm):
        group[np.asarray(sites)] = g
    kinds, inc, full = [], np.zeros(len(names)), np.zeros(len(names))
    groups = [{"eci": [], "ref": [], "cols": [], "decs": []} for _ in sizes]
    for k, name in enumerate(names):
        if name.startswith("c0"):
            kinds.append(("empty", 0))
            continue
        prefix, deco = name.rsplit("_", 1)
        if name.startswith("c1"):
            kinds.append(("singlet", int(deco)))
            continue
        kinds.append(("cluster", 0))
        deco = [int(c) for c in deco]
        found = [g.get(prefix) for g in s.cluster_info]
        equiv = next(c for c in found if c)["equiv_sites"]
        decos = _equivalent(deco, equiv)
        m = [len(c["indices"]) if c else 0 for c in found]
        inc[k] = len(deco) / len(decos) / (sum(m) * sizes[0])
        full[k] = 1.0 / (len(decos) * sum(a * b for a, b in zip(m, sizes)))
        for c, g in zip(found, groups):
            for d in decos if c else []:
                for members, order in zip(c["indices"], c["order"]):
                    where = [0] * len(deco)
                    for i, o in enumerate(order):
                        where[o] = i
                    own = [d[where[p]] for p in range(len(deco))]
                    g["eci"].append(k)
                    g["ref"].append(own[0])
                    pad = 3 - len(members)
                    g["cols"].append([col[int(x)] for x in members] + [-1] * pad)
                    g["decs"].append(own[1:] + [0] * pad)
    groups = [{k: np.array(v, dtype=np.int64) for k, v in g.items()} for g in groups]
    return {"names": names, "symbols": symbols, "bf": bf, "kinds": kinds, "inc": inc, "full": full, "groups": groups,
            "site_group": group, "table": np.asarray(s.table, dtype=np.int64)}


def _equivalent(deco, equiv):
    """Decorations that permuting the equivalent sites makes of `deco`."""
    from itertools import permutations
    seen, todo = {tuple(deco)}, [tuple(deco)]
    while todo:
        d = todo.pop()
        for sites in equiv:
            for p in permutations(sites):
                e = list(d)
                for a, b in zip(sites, p):
                    e[a] = d[b]
                if tuple(e) not in seen:
                    seen.add(tuple(e))
                    todo.append(tuple(e))
    return sorted(seen)


def _full_cf(system, L, occ):
    """Correlation functions of every chain by direct summation over all sites, [chains, ECIs]."""
    t = _terms(system, L)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    occ = torch.as_tensor(np.asarray(occ, dtype=np.int64), device=dev)
    bf = torch.as_tensor(t["bf"], device=dev)
    C, N = occ.shape
    out = torch.zeros((C, len(t["names"])), dtype=torch.float64, device=dev)
    for k, (kind, d) in enumerate(t["kinds"]):
        if kind == "empty":
            out[:, k] = 1.0
        elif kind == "singlet":
            out[:, k] = bf[d][occ].mean(1)
    for g, terms in enumerate(t["groups"]):
        sites = torch.as_tensor(np.nonzero(t["site_group"] == g)[0], device=dev)
        table = torch.as_tensor(t["table"], device=dev)[sites]
        around = {}
        for i in range(len(terms["eci"])):
            p = bf[int(terms["ref"][i])][occ[:, sites]]
            for c, d in zip(terms["cols"][i].tolist(), terms["decs"][i].tolist()):
                if c < 0:
                    continue
                if (c, d) not in around:
                    if len(around) * C * len(sites) > 2e8:
                        around.clear()
                    around[c, d] = bf[d][occ[:, table[:, c]]]
                p = p * around[c, d]
            out[:, int(terms["eci"][i])] += p.sum(1)
    for k, (kind, _) in enumerate(t["kinds"]):
        if kind == "cluster":
            out[:, k] *= float(t["full"][k])
    return out.cpu().numpy()


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 over arrays of counters."""
    mask = np.uint64(0xFFFFFFFF)
    c = [np.asarray(np.broadcast_to(np.asarray(x, dtype=np.uint64), np.shape(c0))) for x in (c0, c1, c2, c3)]
    k0, k1 = int(k0), int(k1)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


class _Chain:
    """The Metropolis chain of the counter-based stream, one trial at a time in 64 bits."""

    def __init__(self, system, L, occ, eci, kT, move, seed, key=0):
        self.t = t = _terms(system, L)
        self.occ, self.kT, self.move, self.seed, self.key = occ.astype(np.int64).copy(), kT, move, seed, key
        self.N, self.S = len(occ), len(t["symbols"])
        self.next = 0
        self.set_eci(eci)
        self.energy = self.N * float(np.dot(self.eci, _full_cf(system, L, occ[None])[0]))
        self.system, self.L = system, L
        self.phi = [t["bf"][d] for d in range(len(t["bf"]))]
        self.singlet = np.array([p[self.occ].mean() for p in self.phi])
        self.lists = [np.nonzero(self.occ == s)[0].tolist() for s in range(self.S)]

    def set_eci(self, eci):
        t, self.eci = self.t, np.asarray(eci, dtype=np.float64)
        self.groups = []
        for g in t["groups"]:
            cols, decs = g["cols"], g["decs"]
            vals = np.concatenate([t["bf"], np.ones((1, t["bf"].shape[1]))])  # row n_bf: absent member
            decs = np.where(cols < 0, len(t["bf"]), decs)
            self.groups.append((self.eci[g["eci"]] * self.N * t["inc"][g["eci"]], g["ref"], np.maximum(cols, 0), decs,
                                vals))
        self.alone = np.zeros(len(t["bf"]))
        for k, (kind, d) in enumerate(t["kinds"]):
            if kind == "singlet":
                self.alone[d] = self.eci[k]

    def change(self, site, new):
        """Energy change of putting `new` on `site`."""
        t, old = self.t, self.occ[site]
        w, ref, cols, decs, vals = self.groups[t["site_group"][site]]
        around = self.occ[t["table"][site]]
        delta = t["bf"][:, new] - t["bf"][:, old]
        return float(np.dot(w * delta[ref], vals[decs, around[cols]].prod(1)) + np.dot(self.alone, delta))

    def put(self, site, new):
        self.singlet += (self.t["bf"][:, new] - self.t["bf"][:, self.occ[site]]) / self.N
        self.occ[site] = new

    def trials(self, n):
        """The next n trials: energy and singlets after each, and the number accepted."""
        at = np.arange(self.next, self.next + n, dtype=np.uint64)
        self.next += n
        key = (self.seed & 0xFFFFFFFF, ((self.seed >> 32) & 0xFFFFFFFF) ^ self.key)
        w = np.stack(_philox(at & np.uint64(0xFFFFFFFF), at >> np.uint64(32), 0, 0, *key), 1).tolist()
        x = np.stack(_philox(at & np.uint64(0xFFFFFFFF), at >> np.uint64(32), 1, 0, *key), 1).tolist()
        below = lambda word, m: (word * m) >> 32  # noqa: E731
        energies, singlets, accepted = np.empty(n), np.empty((n, len(self.phi))), 0
        present = [s for s in range(self.S) if self.lists[s]]
        for i in range(n):
            if self.move == "flip":
                site = below(w[i][0], self.N)
                new = below(w[i][1], self.S - 1)
                new += new >= self.occ[site]
                old = int(self.occ[site])
                de, (ua, ub) = self.change(site, new), w[i][2:4]
            else:
                ia, ib = below(w[i][0], len(present)), below(w[i][1], len(present) - 1)
                A, B = present[ia], present[ib + (ib >= ia)]
                pa, pb = below(w[i][2], len(self.lists[A])), below(w[i][3], len(self.lists[B]))
                sa, sb = self.lists[A][pa], self.lists[B][pb]
                de = self.change(sa, B)
                self.occ[sa] = B
                de += self.change(sb, A)
                self.occ[sa] = A
                ua, ub = x[i][0:2]
            u = ((ua >> 5) * 67108864.0 + (ub >> 6)) / 9007199254740992.0
            if de < 0 or u <= math.exp(-de / self.kT):
                accepted += 1
                self.energy += de
                if self.move == "flip":
                    self.put(site, new)
                    assert old != new
                else:
                    self.occ[sa], self.occ[sb] = B, A
                    self.lists[A][pa], self.lists[B][pb] = sb, sa
            energies[i], singlets[i] = self.energy, self.singlet
        return energies, singlets, accepted

    def cf(self):
        return _full_cf(self.system, self.L, self.occ[None])[0]


def _sums(e_ref, energies, singlets):
    """Running sums in the order a chain keeps them (unused decorations zero)."""
    e, nb = energies - e_ref, singlets.shape[1]
    out = np.zeros(15)
    out[:3] = e_ref, e.sum(), (e * e).sum()
    out[3:3 + nb], out[7:7 + nb] = singlets.sum(0), (singlets ** 2).sum(0)
    out[11:11 + nb] = (singlets * e[:, None]).sum(0)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("calculator", "driver", "chain", "recompute"):
        return None  # the chain is sequential: these would take far too long one trial at a time
    system, L = case["system"], case["L"]
    s, t = _settings(system, L), _terms(system, L)
    seeds = seeded_ecis(s.cset, 0)
    eci = np.array([float(seeds[n]) for n in t["names"]])

    class Shape:  # what _occupations reads of a model
        n_sites, n_sym = s.n_sites, len(t["symbols"])

    if kind == "recompute":
        n = case["chains"]
        cf = _full_cf(system, L, _occupations(Shape, n, seed, "flip"))
        return {"cf": cf, "energy": s.n_sites * cf @ eci}
    if kind == "calculator":
        occ = _occupations(Shape, 1, seed, "swap")[0]
        a, b = _calculator_sites(occ, seed)
        before = _full_cf(system, L, occ[None])[0]
        occ[a], occ[b] = occ[b], occ[a]
        cf = _full_cf(system, L, occ[None])[0]
        return {"energy": float(s.n_sites * cf @ eci), "cf": cf, "energy_back": float(s.n_sites * before @ eci)}
    if kind == "driver":
        occ = _occupations(Shape, 1, seed, "swap")[0]
        k1 = t["names"].index("c1_0")
        mu = -0.05 if case["move"] == "flip" else 0.0
        eci[k1] -= mu
        mc = _Chain(system, L, occ, eci, KB * 800.0, case["move"], seed)
        mc.trials(1)
        mc.trials(1000)
        energies, singlets, _ = mc.trials(case["steps"])
        mean, var = float(energies.mean()), float(energies.var())
        thermo = {"temperature": 800.0}
        if case["move"] == "flip":
            m1 = float(singlets[:, 0].mean())
            thermo.update(sgc_energy=mean, sgc_heat_capacity=var / (KB * 800.0 ** 2), energy=mean + mu * m1 * s.n_sites,
                          singlet_c1_0=m1, var_singlet_c1_0=float(singlets[:, 0].var()), mu_c1_0=mu)
        else:
            thermo.update(energy=mean, heat_capacity=var / (KB * 800.0 ** 2))
        cf = mc.cf()
        eci[k1] += mu
        return {"thermo": thermo, "occ": None, "cf": cf, "energy": float(s.n_sites * cf @ eci)}
    n, trials = case["chains"], int(case["sweeps"]) * s.n_sites
    if n * trials * (1 if case["move"] == "flip" else 2) * len(t["groups"][0]["eci"]) > 1.2e8:
        return None
    occ, kT = _occupations(Shape, n, seed, case["move"]), KB * _temperatures(n)
    cfs, energy, sums = [], [], []
    for c in range(n):
        ev = eci.copy()
        if case["move"] == "flip":
            ev[t["names"].index("c1_0")] -= _mu(c)
        mc = _Chain(system, L, occ[c], ev, float(kT[c]), case["move"], seed, key=c)
        e_ref = mc.energy
        energies, singlets, _ = mc.trials(trials)
        cf = mc.cf()
        cfs.append(cf)
        energy.append(s.n_sites * float(np.dot(ev, cf)))
        sums.append(_sums(e_ref, energies, singlets))
    return {"cf": np.array(cfs), "energy": np.array(energy), "sums": np.array(sums)}
