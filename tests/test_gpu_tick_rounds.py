"""Booking rounds of the scheduled table kernel: a round ends before the first trial that an accepted trial of the round
touches, whatever the moment in which the cutter sees that trial finished.  Rounds cut at other trials give FP32
running sums of another rounding, so repeated launches from one state, and the speculative form (here with a
constraint mask that allows everything), give the same sums bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


@pytest.mark.parametrize("move,L,recipe", [(1, 14, (2, 1, 0)), (1, 15, (5, 3, 1)), (0, 10, (5, 3, 1))])
def test_repeated_launches_book_the_same_rounds(move, L, recipe):
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(L, *recipe, ["Al", "Mg", "Si"])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    geo = E.Geometry(m)
    n = 24
    occ = np.random.default_rng(3).integers(0, 3, (n, m.n_sites)).astype(np.int8)
    allow = torch.full((n, m.n_sites), 255, dtype=torch.uint8, device="cuda")
    cb = E.ChainBatch(geo, occ, m.eci_vector(eci), KB * np.linspace(300.0, 3000.0, n), move, seed=5)
    torch.cuda.synchronize()
    names = ["occ", "cf", "energy", "trial", "accum"] + (["trk", "loc"] if move else [])
    start = {k: getattr(cb, k).clone() for k in names}
    start["accum"][:, E.A_NSAMP:].view(torch.int64)[:] = 10000  # chains that have accepted every trial so far
    want = None
    for i in range(20):
        for k in names:
            getattr(cb, k).copy_(start[k])
        cb.run(3000, precision=E.PREC_F32, warps=16, kernel=E.KERNEL_TABLE, cluster=1,
               site_allow=allow if i == 0 else None)
        torch.cuda.synchronize()
        cb.check_status()
        got = {k: getattr(cb, k).clone() for k in names}
        if want is None:
            want = got
        for k in names:
            assert torch.equal(want[k].view(torch.uint8), got[k].view(torch.uint8)), (i, k)
