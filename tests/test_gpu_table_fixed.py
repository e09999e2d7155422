"""FP64 table form with its entries in 64-bit fixed point (cemc_mc.cu, fixed_point_scale): decisions and energy
changes, with ECIs over many orders of magnitude, flips and swaps, one and two groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


@pytest.mark.parametrize("cell", ["fcc", "hcp"])
@pytest.mark.parametrize("move", [0, 1])
@pytest.mark.parametrize("factor", [2.0 ** -60, 1.0, 2.0 ** 40])
def test_fixed_point_table_matches_term_by_term_form(cell, move, factor):
    """Against the generic form, which sums the changed terms in FP64 (the oracle's energy change is the
    difference of two total energies, good to 1e-12 eV only)."""
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, hcp_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    names = ["Al", "Mg", "Si"]
    s = fcc_settings(5, 3, 2, 1, names) if cell == "fcc" else hcp_settings(5, 5, 2, 1, 1, names)
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    ev = m.eci_vector(eci)
    ev[m.eci_kind != 0] *= factor
    kT = KB * 800.0 * factor
    occ = np.random.default_rng(1).integers(0, 3, (1, m.n_sites)).astype(np.int8)
    geo = E.Geometry(m)
    got = []
    for kernel in (E.KERNEL_TABLE, E.KERNEL_GENERIC):
        cb = E.ChainBatch(geo, occ, ev, kT, move, seed=3)
        _, acc, de = cb.run(1500, precision=E.PREC_F64, warps=8, kernel=kernel, trace=True)
        torch.cuda.synchronize()
        cb.check_status()
        got.append((acc.cpu().numpy()[0], cb.occ.cpu().numpy()[0], de.cpu().numpy()[0]))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
    # the quantum is 2^-60 (n + 5) times the largest entry (below 1 eV times the factor) and a change adds n
    # entries rounded to it; the term-by-term sum is of FP64 roundings of the same size
    assert np.max(np.abs(got[0][2] - got[1][2])) < 1e-13 * factor


def test_fixed_point_table_needs_finite_entries():
    """An infinite ECI cannot be held in fixed point: such a launch keeps FP64 entries and rejects what it did."""
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(4, 2, 1, 0, ["Al", "Mg", "Si"])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    ev = m.eci_vector(eci)
    ev[[k for k in range(m.n_eci) if m.eci_kind[k] == 1][0]] = np.inf  # a singlet
    occ = np.random.default_rng(1).integers(0, 3, (1, m.n_sites)).astype(np.int8)
    got = []
    for kernel in (E.KERNEL_TABLE, E.KERNEL_GENERIC):
        cb = E.ChainBatch(E.Geometry(m), occ, ev, KB * 800.0, 0, seed=3)
        _, acc, _ = cb.run(400, precision=E.PREC_F64, warps=4, kernel=kernel, trace=True)
        torch.cuda.synchronize()
        got.append(acc.cpu().numpy()[0])
    assert np.array_equal(got[0], got[1])
