"""Launches whose kernel the device chooses by the chains' acceptance so far and their composition (cemc_route.cu):
whatever the running sums say, every chain is run once, by either kernel, to the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


def _batch(E, L, recipe, species, move, chains, occ=None):
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(L, *recipe, ["Al", "Mg", "Si"][:species])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    if occ is None:
        occ = np.random.default_rng(L).integers(0, species, (chains, m.n_sites)).astype(np.int8)
    geo = E.Geometry(m)
    return [E.ChainBatch(geo, occ, m.eci_vector(eci), KB * np.linspace(300.0, 1500.0, chains), move, seed=2)
            for _ in range(3)]


def _counters(E, cb, samples, accepted):
    cb.accum[:, E.A_NSAMP] = torch.tensor(samples, dtype=torch.int64).view(torch.float64)
    cb.accum[:, E.A_NACC] = torch.tensor(accepted, dtype=torch.int64).view(torch.float64)


def _left(E, cb, samples, accepted):
    torch.cuda.synchronize()
    cb.check_status()
    n = cb.accum[:, E.A_NSAMP:].view(torch.int64).clone()
    n[:, 0] -= samples
    n[:, 1] -= accepted
    out = [cb.occ, cb.cf, cb.energy, cb.trial, cb.accum[:, :E.A_NSAMP], n]
    return [t.clone() for t in (out + ([cb.trk, cb.loc] if cb.trk is not None else []))]


# cells of 8 and 12 evaluating warps, and rounds of more than 32 trials; cold, hot and unknown acceptance
@pytest.mark.parametrize("L,warps,kernel", [(8, 4, 6), (8, 8, 0), (9, 8, 6), (12, 8, 6), (12, 16, 6)])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("budgets", [False, True])
def test_flips_by_acceptance(L, warps, kernel, prec, budgets):
    from cemc_gb300 import engine as E
    chains, n = 4, 3001
    states = [(5000, 0), (5000, 4999), (100, 100)]
    per = torch.tensor([n, 0, 65, 2999], dtype=torch.int64, device="cuda") if budgets else None
    got = []
    for cb, (samples, accepted) in zip(_batch(E, L, (4, 2, 1), 2, E.MOVE_FLIP, chains), states):
        _counters(E, cb, samples, accepted)
        for _ in range(2):  # the second call finds the counters of the first
            cb.run(n, precision=prec, warps=warps, kernel=kernel, cluster=1, chain_trials=per)
            assert cb.last_scheduled == 2
        got.append(_left(E, cb, samples, accepted))
    assert torch.equal(got[0][3], 2 * (per if budgets else torch.full((chains,), n, device="cuda")))
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert torch.equal(x, y)


def test_short_calls_and_calls_without_status_are_not_routed():
    from cemc_gb300 import engine as E
    a, b, c = _batch(E, 8, (4, 2, 1), 2, E.MOVE_FLIP, 2)
    a.run(2047, precision=E.PREC_F32, warps=8, cluster=1)
    assert a.last_scheduled == 0
    c.run(2048, precision=E.PREC_F32, warps=8, cluster=1)
    assert c.last_scheduled == 2
    b.status = None
    b.run(3000, precision=E.PREC_F32, warps=8, cluster=1)
    assert b.last_scheduled == 0
    torch.cuda.synchronize()
    assert b.trial.tolist() == [3000, 3000] and c.trial.tolist() == [2048, 2048]


def test_routed_launch_in_a_graph():
    """A captured launch decides anew at each replay; after replays the chain is the one of separate calls."""
    from cemc_gb300 import engine as E
    from cemc_gb300.batch import BatchRunner
    a, _, _ = _batch(E, 8, (4, 2, 1), 2, E.MOVE_FLIP, 3)
    r = BatchRunner(a.geo, a.occ.cpu().numpy(), a.eci.cpu().numpy(), np.linspace(300.0, 1500.0, 3), E.MOVE_FLIP,
                    seed=2, warps=8, cluster=1, sweeps_per_step=1.0, recompute_every=1)
    r.step(4)
    r.synchronize()
    assert r.cb.last_scheduled == 2
    for _ in range(4):
        a.run(r.trials_per_step, precision=E.PREC_F32, warps=8, cluster=1, kernel=E.KERNEL_SPIN_HALFWARP)
        a.recompute()
    torch.cuda.synchronize()
    for k in ("occ", "cf", "energy", "trial"):
        assert torch.equal(getattr(a, k), getattr(r.cb, k)), k


def _composition(kind, n_sites, species, chains):
    """Site occupations of `chains` chains; the solutes of `kind` atoms each, or equal parts."""
    counts = [n_sites // species] * species if kind == "equal" else [0] + [kind] * (species - 1)
    counts[0] = n_sites - sum(counts[1:])
    rng = np.random.default_rng(n_sites)
    return np.stack([rng.permutation(np.repeat(np.arange(species), counts)) for _ in range(chains)]).astype(np.int8)


# lists in shared memory (8 trials a tick; 18 columns) and in device memory (16 and 24 a tick); solutes of 1 to 3
# atoms, of as many as share slots most often in the scheduled kernel (40 and 32), and equal parts
@pytest.mark.parametrize("L,recipe,species", [(10, (5, 3, 1), 3), (10, (2, 1, 0), 3), (14, (5, 3, 1), 3), (24, (6, 2, 1), 2)])
@pytest.mark.parametrize("kind", [1, 3, 40, 200, "equal"])
@pytest.mark.parametrize("prec", [0, 1])
def test_swaps_by_acceptance_and_composition(L, recipe, species, kind, prec):
    from cemc_gb300 import engine as E
    chains, n = 3, 3001
    n_sites = 4 * L ** 3
    occ = _composition(kind, n_sites, species, chains)
    per = torch.tensor([n, 0, 2999], dtype=torch.int64, device="cuda")
    got = []
    states = [(5000, 0), (5000, 4999), (100, 100)]
    for cb, (samples, accepted) in zip(_batch(E, L, recipe, species, E.MOVE_SWAP, chains, occ), states):
        _counters(E, cb, samples, accepted)
        for _ in range(2):
            cb.run(n, precision=prec, warps=8, cluster=1, chain_trials=per)
            assert cb.last_scheduled == 2
        got.append(_left(E, cb, samples, accepted))
    assert torch.equal(got[0][3], 2 * per)
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert torch.equal(x, y)


def _other(E, kind, move):
    from cemc_gb300.lattice import fcc_settings, hcp_settings, seeded_ecis, with_background
    from cemc_gb300.tables import CEModel
    names = ["Al", "Mg", "Si"]
    s = hcp_settings(16, 8, 2, 1, 1, names) if kind == "hcp" else fcc_settings(10, 5, 3, 1, names)
    eci = seeded_ecis(s.cset, 0)
    if kind == "background":
        s = with_background(s)
    m = CEModel(s, list(eci))
    occ = np.random.default_rng(7).integers(0, 3, (2, m.n_sites)).astype(np.int8)
    if len(m.background):
        occ[:, m.background] = 0
    geo = E.Geometry(m)
    return [E.ChainBatch(geo, occ, m.eci_vector(eci), KB * np.array([400.0, 2000.0]), move, seed=11) for _ in range(2)]


@pytest.mark.parametrize("kind,move,prec", [("hcp", 1, 0), ("hcp", 1, 1), ("background", 1, 1), ("background", 0, 1),
                                            ("fcc", 0, 1)])
@pytest.mark.parametrize("cluster", [1, 2])
def test_other_cells_and_flips(kind, move, prec, cluster):
    """Two translation groups, background sites, flips; rounds of one CTA and of a pair."""
    from cemc_gb300 import engine as E
    got = []
    for cb, accepted in zip(_other(E, kind, move), (0, 5000)):
        _counters(E, cb, 5000, accepted)
        for _ in range(2):
            cb.run(2500, precision=prec, warps=16, cluster=cluster, kernel=E.KERNEL_TABLE)
            assert cb.last_scheduled == 2
        got.append(_left(E, cb, 5000, accepted))
    for x, y in zip(*got):
        assert torch.equal(x, y)


def test_decision_ahead_of_the_launch():
    """cemc_decide and cemc_run_decided are cemc_run; several batches stepped together decide ahead of their launches."""
    from cemc_gb300 import engine as E
    from cemc_gb300.batch import BatchRunner, MultiBatchRunner
    a, b, c = _batch(E, 9, (4, 2, 1), 2, E.MOVE_FLIP, 3)
    for cb, accepted in ((a, 4000), (b, 4000), (c, 0)):
        _counters(E, cb, 5000, accepted)
    kw = dict(precision=E.PREC_F32, warps=16, cluster=1)
    a.run(3000, **kw)
    for cb in (b, c):
        cb.run(3000, part="cemc_decide", **kw)
        torch.cuda.synchronize()
        assert cb.trial.tolist() == [0, 0, 0]  # nothing has run
        cb.run(3000, part="cemc_run_decided", **kw)
    left = [_left(E, cb, 5000, accepted) for cb, accepted in ((a, 4000), (b, 4000), (c, 0))]
    for other in left[1:]:
        for x, y in zip(left[0], other):
            assert torch.equal(x, y)
    runners = [BatchRunner(cb.geo, cb.occ.cpu().numpy(), cb.eci.cpu().numpy(), 700.0, move, seed=5, warps=8, cluster=1,
                           chain_keys=np.arange(3))
               for cb, move in ((a, E.MOVE_FLIP), (_batch(E, 14, (2, 1, 0), 3, E.MOVE_SWAP, 3)[0], E.MOVE_SWAP),
                                (_batch(E, 5, (2, 1, 0), 2, E.MOVE_FLIP, 3)[0], E.MOVE_FLIP))]
    alone = [BatchRunner(r.geo, r.cb.occ.cpu().numpy(), r.cb.eci.cpu().numpy(), 700.0, r.cb.move, seed=5, warps=8, cluster=1,
                         chain_keys=np.arange(3)) for r in runners]
    multi = MultiBatchRunner(runners)
    multi.step(3)
    multi.synchronize()
    for r, s in zip(runners, alone):
        s.step(3)
        s.synchronize()
        r.cb.check_status()
        for k in ("occ", "cf", "energy", "trial", "accum"):
            assert torch.equal(getattr(r.cb, k).view(torch.uint8), getattr(s.cb, k).view(torch.uint8)), k
