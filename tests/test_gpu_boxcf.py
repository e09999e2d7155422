"""The bit-plane recompute (cemc_boxcf.cu) against the oracle's brute force: odd and even boxes, rows of more
than 32 sites, offsets that wrap onto themselves, several CTAs per chain, one and many chains, 2 and 3 species
and a binary basis that is not +1/-1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


@pytest.mark.parametrize("lattice,L,recipe,species,chains", [
    ("fcc", 4, (4, 2, 1), 2, 1), ("fcc", 5, (4, 2, 1), 2, 7), ("fcc", 9, (4, 2, 1), 2, 40), ("fcc", 16, (4, 2, 1), 2, 3),
    ("sc", 33, (3, 2, 1), 2, 2), ("sc", 64, (2, 1, 1), 2, 1), ("bcc", 32, (3, 2, 1), 2, 2),
    ("fcc", 4, (3, 2, 1), 3, 2), ("fcc", 7, (5, 3, 1), 3, 5), ("sc", 33, (2, 2, 1), 3, 1), ("bcc", 11, (3, 2, 1), 3, 30),
])
@pytest.mark.parametrize("basis", ["own", "scaled"])
def test_bit_plane_recompute_matches_brute_force(lattice, L, recipe, species, chains, basis, oracle_mod):
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import cubic_settings, fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    names = ["Al", "Mg", "Si"][:species]
    s = fcc_settings(L, *recipe, names) if lattice == "fcc" else cubic_settings(lattice, L, *recipe, names)
    eci = seeded_ecis(s.cset, 0)
    if basis == "scaled":  # no +1/-1 values: species tuples are counted
        s.basis_functions = [{k: 0.75 * v + 0.125 * i for i, (k, v) in enumerate(sorted(b.items()))}
                             for b in s.basis_functions]
    m = CEModel(s, list(eci))
    geo = E.Geometry(m)
    occ = np.random.default_rng(L).integers(0, species, (chains, m.n_sites)).astype(np.int8)
    cb = E.ChainBatch(geo, occ, m.eci_vector(eci), KB * 800.0, E.MOVE_FLIP, seed=1)
    cf, energy = cb.cf.cpu().numpy(), cb.energy.cpu().numpy()
    orc = oracle_mod.Oracle(m)
    for c in (0, chains - 1):
        want = orc.full_cf(occ[c])
        # a sum of N products of at most four values of magnitude <= 1.5, divided by N: rounding of a few
        # N 2^-53 / N at most
        assert np.max(np.abs(cf[c] - want)) < 1e-12
        assert abs(energy[c] - m.n_sites * float(np.dot(m.eci_vector(eci), cf[c]))) <= 1e-12 * abs(energy[c])
