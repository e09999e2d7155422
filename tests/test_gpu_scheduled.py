"""Which launches a scheduled kernel takes, as reported by the run descriptor: cells on both sides of each size below
which trials touch one another too often (a cell's room is its number of neighbourhoods of a trial's sites)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


def _batch(E, L, recipe, species, move, chains=2, kT=KB * 800.0):
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(L, *recipe, ["Al", "Mg", "Si"][:species])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    occ = np.random.default_rng(L).integers(0, species, (chains, m.n_sites)).astype(np.int8)
    return E.ChainBatch(E.Geometry(m), occ, m.eci_vector(eci), kT, move, seed=2), m


# binary flips: room 24 and 37; three-species swaps of 54 columns: room 9 and 13; of 18 columns: room 38 and 52
# (room 39 and 31 are in no cubic cell); the largest cell; two-species swaps by the spin form: never
@pytest.mark.parametrize("L,recipe,species,move,scheduled", [
    (7, (4, 2, 1), 2, 0, False), (8, (4, 2, 1), 2, 0, True), (24, (4, 2, 1), 2, 0, True),
    (8, (4, 2, 1), 3, 1, False), (9, (4, 2, 1), 3, 1, True), (9, (2, 1, 0), 3, 1, False), (10, (2, 1, 0), 3, 1, True),
    (24, (5, 3, 1), 3, 1, True), (16, (4, 2, 1), 2, 1, False)])
def test_launches_a_scheduled_kernel_takes(L, recipe, species, move, scheduled):
    from cemc_gb300 import engine as E
    cb, m = _batch(E, L, recipe, species, move)
    cb.run(3000, precision=E.PREC_F32, warps=8, cluster=1)
    assert bool(cb.last_scheduled) == scheduled
    torch.cuda.synchronize()
    cb.check_status()
    # a constraint (here one that allows everything) is never scheduled
    allow = torch.full((2, m.n_sites), 255, dtype=torch.uint8, device="cuda")
    cb.run(100, precision=E.PREC_F32, warps=8, cluster=1, site_allow=allow)
    assert not cb.last_scheduled


def test_more_chains_than_sms_share_them():
    """Where two CTAs of the speculative form share an SM, more chains than SMs keep it, in one launch or several."""
    from cemc_gb300 import engine as E
    from cemc_gb300.batch import BatchRunner, MultiBatchRunner
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def scheduled(L, chains, beside=0):
        cb, _ = _batch(E, L, (4, 2, 1), 2, E.MOVE_FLIP, chains)
        cb.beside = beside
        cb.run(2100, precision=E.PREC_F32, warps=4, cluster=1)
        torch.cuda.synchronize()
        cb.check_status()
        return cb.last_scheduled

    assert scheduled(8, sms) == 2 and scheduled(8, sms + 1) == 0
    assert scheduled(8, sms - 9, 9) == 2 and scheduled(8, sms - 9, 10) == 0
    assert scheduled(14, sms + 1) == 1  # one CTA of either kernel takes an SM
    cb, m = _batch(E, 8, (4, 2, 1), 2, E.MOVE_FLIP, 3)
    runners = [BatchRunner(cb.geo, cb.occ.cpu().numpy()[:n], cb.eci.cpu().numpy()[:n], 500.0, E.MOVE_FLIP, warps=4,
                           cluster=1) for n in (1, 2, 3)]
    MultiBatchRunner(runners)
    assert [r.cb.beside for r in runners] == [5, 4, 3]
