"""The scheduled flip kernel (cemc_sched.cu) against the speculative spin forms and the CPU oracle.

The forms draw the same trials from the counter-based stream, evaluate the same energy changes and book the
same rounds, so a launch of the scheduled kernel must equal one of the half-warp form with the same round
width bit for bit: occupations, correlation functions, energies, running sums and traces, in both precisions.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


@pytest.fixture(scope="module")
def E():
    from cemc_gb300 import engine
    return engine


def _model(L, recipe=(4, 2, 1), background=False, swap_basis=False):
    from cemc_gb300.lattice import fcc_settings, seeded_ecis, with_background
    from cemc_gb300.tables import CEModel
    s = fcc_settings(L, *recipe, ["Al", "Mg"])
    eci = seeded_ecis(s.cset, 0)
    if swap_basis:  # the other species holds the -1
        s.basis_functions = [{k: -v for k, v in b.items()} for b in s.basis_functions]
    if background:
        s = with_background(s)
    m = CEModel(s, list(eci))
    return m, m.eci_vector(eci)


def _state(E, cb):
    torch.cuda.synchronize()
    cb.check_status()
    return [t.clone() for t in (cb.occ, cb.cf, cb.energy, cb.trial, cb.accum[:, :E.A_NSAMP],
                                cb.accum[:, E.A_NSAMP:].view(torch.int64))]


def _batch(E, geo, m, ev, n, seed=5):
    rng = np.random.default_rng(seed)
    occ = rng.integers(0, 2, (n, m.n_sites)).astype(np.int8)
    if len(m.background):
        occ[:, m.background] = 0
    return E.ChainBatch(geo, occ, ev, KB * np.linspace(250.0, 1500.0, n), E.MOVE_FLIP, seed=seed), occ


# cells: the smallest that is scheduled (8 evaluating warps), 12 and 16 warps, a hash smaller than the cell;
# more than four multi-site cluster ECIs; the other spin sign; movable sites among background ones
CELLS = [(8, (4, 2, 1), False, False), (9, (4, 2, 1), False, True), (12, (4, 2, 1), False, False),
         (24, (4, 2, 1), False, False), (8, (3, 2, 2), False, False), (8, (4, 2, 1), True, False)]


@pytest.mark.parametrize("cell", CELLS)
@pytest.mark.parametrize("warps", [1, 3, 8])
@pytest.mark.parametrize("prec", [0, 1])
def test_scheduled_equals_half_warp_form(cell, warps, prec, E):
    m, ev = _model(*cell)
    geo = E.Geometry(m)
    a, _ = _batch(E, geo, m, ev, 3)
    b, _ = _batch(E, geo, m, ev, 3)
    for n in (1, 31, 65, 3000):  # remainders of rounds and batches, then several ring turns
        ta = a.run(n, precision=prec, warps=warps, kernel=E.KERNEL_SPIN_QUARTER, trace=True)
        tb = b.run(n, precision=prec, warps=2 * warps, kernel=E.KERNEL_SPIN_HALFWARP, trace=True, cluster=1)
        for x, y in zip(_state(E, a) + list(ta), _state(E, b) + list(tb)):
            assert torch.equal(x, y)


@pytest.mark.parametrize("warps", [9, 12, 16])
def test_scheduled_wide_rounds_and_default_form(warps, E):
    """Booking rounds of 33 to 64 trials (two bookers), and the automatic form's own width."""
    m, ev = _model(10)
    geo = E.Geometry(m)
    a, _ = _batch(E, geo, m, ev, 2)
    b, _ = _batch(E, geo, m, ev, 2)
    a.run(5000, precision=0, warps=warps, kernel=E.KERNEL_SPIN_QUARTER)
    assert a.last_kernel == E.KERNEL_SPIN_QUARTER
    b.run(5000, precision=0, warps=4, kernel=E.KERNEL_SPIN, cluster=1)
    sa, sb = _state(E, a), _state(E, b)
    for i in (0, 1, 2, 3, 5):
        assert torch.equal(sa[i], sb[i])
    # FP64 sums of 5000 trials in another order: 5000 roundings of 2^-53 each at most
    assert torch.allclose(sa[4], sb[4], rtol=5000 * 2.0 ** -53, atol=1e-9)
    c, _ = _batch(E, geo, m, ev, 2)
    d, _ = _batch(E, geo, m, ev, 2)
    c.run(2000, precision=1, warps=warps)  # automatic: the half-warp form's round width
    d.run(2000, precision=1, warps=warps, kernel=E.KERNEL_SPIN_HALFWARP, cluster=1)
    for x, y in zip(_state(E, c), _state(E, d)):
        assert torch.equal(x, y)


def test_scheduled_uneven_budgets_and_oracle(E, oracle_mod):
    """Chains with their own trial counts (one of them none), against the oracle's sequential chain."""
    m, ev = _model(8)
    geo = E.Geometry(m)
    cb, occ = _batch(E, geo, m, ev, 4)
    counts = [2500, 0, 1, 64]
    cb.run(2500, precision=0, chain_trials=torch.tensor(counts, dtype=torch.int64, device="cuda"))
    occ_d, cf_d, energy_d, trial_d, _, n_d = _state(E, cb)
    orc = oracle_mod.Oracle(m)
    for c, n in enumerate(counts):
        st = orc.new_chain_state(occ[c], ev, float(cb.kT[c].item()), 0)
        tr = orc.run(st, seed=5, chain_id=c, t_begin=0, n_trials=n, trace=True) if n else None
        assert np.array_equal(occ_d[c].cpu().numpy(), st.occ)
        assert np.allclose(cf_d[c].cpu().numpy(), st.cf, rtol=1e-9, atol=1e-14)
        assert int(trial_d[c]) == n and int(n_d[c, 0]) == n
        assert int(n_d[c, 1]) == (int(tr.acc.sum()) if n else 0)
