"""The scheduled table kernel (cemc_schedt.cu) against the speculative table form and the CPU oracle.

A launch with a constraint mask that allows everything runs the speculative form on the same stream, so with
the same round width everything it leaves must be equal bit for bit: occupations, site lists, correlation
functions, energies, running sums and traces, in both precisions.
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


def _model(kind, L):
    from cemc_gb300.lattice import fcc_settings, hcp_settings, seeded_ecis, with_background
    from cemc_gb300.tables import CEModel
    if kind == "hcp":
        s = hcp_settings(L, 8, 2, 1, 1, ["Al", "Mg", "Si"])
    elif kind == "binary":
        s = fcc_settings(L, 6, 2, 1, ["Al", "Mg"])
    else:
        s = fcc_settings(L, 5, 3, 1, ["Al", "Mg", "Si"])
    eci = seeded_ecis(s.cset, 0)
    if kind == "background":
        s = with_background(s)
    m = CEModel(s, list(eci))
    return m, m.eci_vector(eci)


def _state(E, cb):
    torch.cuda.synchronize()
    cb.check_status()
    out = [cb.occ, cb.cf, cb.energy, cb.trial, cb.accum[:, :E.A_NSAMP], cb.accum[:, E.A_NSAMP:].view(torch.int64)]
    if cb.trk is not None:
        out += [cb.trk, cb.loc]
    return [t.clone() for t in out]


def _batch(E, geo, m, ev, n, move):
    occ = np.random.default_rng(7).integers(0, m.n_sym, (n, m.n_sites)).astype(np.int8)
    if len(m.background):
        occ[:, m.background] = 0
    return E.ChainBatch(geo, occ, ev, KB * np.linspace(300.0, 2000.0, n), move, seed=11), occ


# smallest swap cell (8 trials a tick), 16 and 24 a tick, two translation groups, background sites; flips
CELLS = [("ternary", 10, 1), ("ternary", 15, 1), ("binary", 24, 1), ("hcp", 16, 1), ("background", 10, 1),
         ("ternary", 10, 0), ("binary", 10, 0)]


@pytest.mark.parametrize("kind,L,move", CELLS)
@pytest.mark.parametrize("warps", [1, 8, 16])
@pytest.mark.parametrize("prec", [0, 1])
def test_scheduled_table_equals_speculative_form(kind, L, move, warps, prec, E):
    if move == 0 and prec == 0:
        pytest.skip("FP64 flips run the speculative form")
    m, ev = _model(kind, L)
    geo = E.Geometry(m)
    a, _ = _batch(E, geo, m, ev, 2, move)
    b, _ = _batch(E, geo, m, ev, 2, move)
    allow = torch.full((2, m.n_sites), 255, dtype=torch.uint8, device="cuda")
    for n in (1, 31, 65, 2500):  # remainders of rounds and lists, then several ring turns
        ta = a.run(n, precision=prec, warps=warps, kernel=E.KERNEL_TABLE, cluster=1, trace=True)
        tb = b.run(n, precision=prec, warps=warps, kernel=E.KERNEL_TABLE, cluster=1, trace=True, site_allow=allow)
        assert a.last_kernel == E.KERNEL_TABLE
        for x, y in zip(_state(E, a) + list(ta), _state(E, b) + list(tb)):
            assert torch.equal(x, y)


@pytest.mark.parametrize("move", [0, 1])
def test_scheduled_table_uneven_budgets_and_oracle(move, E, oracle_mod):
    """Chains with their own trial counts (one of them none), a pair shape asked for where it fits, against the
    oracle's sequential chain."""
    m, ev = _model("ternary", 10)
    geo = E.Geometry(m)
    cb, occ = _batch(E, geo, m, ev, 4, move)
    counts = [1500, 0, 1, 64]
    cb.run(1500, precision=1, chain_trials=torch.tensor(counts, dtype=torch.int64, device="cuda"), warps=16)
    occ_d, cf_d, _, trial_d, _, n_d = _state(E, cb)[:6]
    orc = oracle_mod.Oracle(m)
    for c, n in enumerate(counts):
        st = orc.new_chain_state(occ[c], ev, float(cb.kT[c].item()), move)
        tr = orc.run(st, seed=11, chain_id=c, t_begin=0, n_trials=n, trace=True) if n else None
        if n:
            # FP32 energy changes: decisions are the oracle's outside |dE / kT + ln u| < 1e-5 eV / kT
            margin = np.abs(tr.de / float(cb.kT[c].item()) + np.log(np.maximum(tr.u, 1e-300)))
            if np.any(margin < 1e-5 / float(cb.kT[c].item())):
                continue
        assert np.array_equal(occ_d[c].cpu().numpy(), st.occ)
        assert np.allclose(cf_d[c].cpu().numpy(), st.cf, rtol=1e-9, atol=1e-12)
        assert int(trial_d[c]) == n and int(n_d[c, 0]) == n
        assert int(n_d[c, 1]) == (int(tr.acc.sum()) if n else 0)


def test_scheduled_table_needs_two_species(E):
    m, ev = _model("ternary", 10)
    geo = E.Geometry(m)
    cb, _ = _batch(E, geo, m, ev, 1, 1)
    cb.occ.fill_(1)
    cb.trk_count.copy_(torch.tensor([[0, m.n_sites, 0]], dtype=torch.int32))
    before = cb.occ.clone()
    cb.run(100, precision=1, warps=8)
    torch.cuda.synchronize()
    assert int(cb.status[0]) == 4 and torch.equal(cb.occ, before)  # CEMC_ERR_STATE
