"""Calls of more trials than one kernel launch takes (2^25 per chain): the running sums and the state are those of
the same trials in two calls, bit for bit, by the scheduled table kernel (flips and swaps), the speculative table
form and the spin form.

Every launch starts its running sums from the chain's energy and correlation functions, so these have to be
up to date between the launches of one call, as they are between two calls.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5
CHUNK = 1 << 25


def test_sums_of_a_split_call():
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    pairs = []
    # (cell, recipe, species, move, kernel): scheduled flips and swaps, speculative table form, spin form
    for L, recipe, species, move, kernel in ((10, (5, 3, 1), 3, E.MOVE_FLIP, E.KERNEL_TABLE),
                                             (16, (2, 1, 0), 3, E.MOVE_SWAP, E.KERNEL_TABLE),
                                             (6, (2, 1, 0), 3, E.MOVE_FLIP, E.KERNEL_TABLE),
                                             (6, (2, 1, 0), 2, E.MOVE_FLIP, E.KERNEL_AUTO)):
        s = fcc_settings(L, *recipe, ["Al", "Mg", "Si"][:species])
        eci = seeded_ecis(s.cset, 0)
        m = CEModel(s, list(eci))
        geo = E.Geometry(m)
        occ = np.random.default_rng(7).integers(0, species, (1, m.n_sites)).astype(np.int8)
        batches = []
        for _ in range(2):
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                batches.append(E.ChainBatch(geo, occ, m.eci_vector(eci), KB * 600.0, move, seed=11, stream=stream))
        one, two = batches
        torch.cuda.synchronize()
        kw = dict(precision=E.PREC_F32, warps=16, cluster=1, kernel=kernel)
        one.run(CHUNK + 3001, **kw)  # the launches of all batches run side by side
        two.run(CHUNK, **kw)
        two.run(3001, **kw)
        pairs.append((one, two))
    torch.cuda.synchronize()
    for one, two in pairs:
        one.check_status()
        assert int(one.trial[0]) == CHUNK + 3001
        for name in ("occ", "cf", "energy", "trial", "accum"):
            assert torch.equal(getattr(one, name).view(torch.uint8), getattr(two, name).view(torch.uint8)), name
