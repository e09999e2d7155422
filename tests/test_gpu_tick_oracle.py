"""FP64 swaps of the scheduled table kernel against the CPU oracle's sequential chain: equal parts, and solutes of as few
atoms as the kernel is given, whose trials share list slots at almost every tick.  In FP64 both evaluate the same
energy changes to rounding (1e-12 eV), and no uniform of the streams lies that close to a decision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


@pytest.mark.parametrize("solute", [0, 100, 140])
def test_fp64_swaps(solute, oracle_mod):
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(13, 5, 3, 1, ["Al", "Mg", "Si"])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    ev, geo = m.eci_vector(eci), E.Geometry(m)
    n, chains = 2500, 2
    counts = [m.n_sites // 3] * 3 if not solute else [0, solute, solute]
    counts[0] = m.n_sites - sum(counts[1:])
    rng = np.random.default_rng(9)
    occ = np.stack([rng.permutation(np.repeat(np.arange(3), counts)) for _ in range(chains)]).astype(np.int8)
    kT = KB * np.array([500.0, 1500.0])
    cb = E.ChainBatch(geo, occ, ev, kT, E.MOVE_SWAP, seed=21)
    cb.accum[:, E.A_NSAMP:].view(torch.int64)[:] = 10000  # chains that have accepted every trial so far
    cb.run(n, precision=E.PREC_F64, warps=8, cluster=1)
    torch.cuda.synchronize()
    cb.check_status()
    assert cb.last_scheduled == 2 and cb.last_kernel == E.KERNEL_TABLE
    orc = oracle_mod.Oracle(m)
    for c in range(chains):
        st = orc.new_chain_state(occ[c], ev, float(kT[c]), E.MOVE_SWAP)
        tr = orc.run(st, seed=21, chain_id=c, t_begin=0, n_trials=n, trace=True)
        margin = np.abs(tr.de / kT[c] + np.log(np.maximum(tr.u, 1e-300)))
        assert margin.min() > 1e-12 / kT[c]  # checked, not skipped
        assert np.array_equal(cb.occ[c].cpu().numpy(), st.occ)
        assert np.allclose(cb.cf[c].cpu().numpy(), st.cf, rtol=1e-9, atol=1e-12)
        got = cb.accum[c, E.A_NSAMP:].view(torch.int64).tolist()
        assert got == [10000 + n, 10000 + int(tr.acc.sum())]
