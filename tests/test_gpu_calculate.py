"""Short change lists through kernel arguments (cemc_calculate, cemc_revert) and longer ones
through device arrays, against the full recompute of the changed occupation.

Tolerances: a correlation function is a mean of products of basis values below 2 in magnitude; adding
n <= 30 changes one after the other in FP64 rounds at 1e-16 each, and the recompute sums up to
1e5 such products, so 1e-12 bounds both.  Taking changes back copies the values: equal bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _updater(system):
    from cemc_gb300 import engine as E
    from cemc_gb300.calculator import DeviceUpdater
    from cemc_gb300.lattice import fcc_settings, hcp_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    if system == "hcp":
        s = hcp_settings(6, 5, 2, 1, 1, ["Al", "Mg", "Si"])
    elif system == "pairs":  # 12 terms: lanes without any between the lanes of one ECI
        s = fcc_settings(4, 1, 0, 0, ["Al", "Mg"])
    elif system == "ternary":
        s = fcc_settings(5, 5, 3, 1, ["Al", "Mg", "Si"])
    else:
        s = fcc_settings(4, 4, 2, 1, ["Al", "Mg"])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    rng = np.random.default_rng(3)
    occ = rng.integers(0, len(m.symbols), m.n_sites)
    return DeviceUpdater(E.Geometry(m, "cuda"), occ, m.eci_vector(eci)), m, m.eci_vector(eci), occ, rng


@pytest.mark.parametrize("system", ["binary", "pairs", "ternary", "hcp"])
@pytest.mark.parametrize("n", [1, 2, 24, 25])
def test_changes_and_undo(system, n):
    from cemc_gb300.calculator import DeviceUpdater
    up, m, eci, occ, rng = _updater(system)
    cf0, e0, occ0 = up.cf(), up.energy(), up.occupation()
    now, changes = occ.copy(), []
    for i in range(n):
        # a site changed twice, and one left as it is, are part of the list
        s = changes[0][0] if i == n - 1 and n > 2 else int(rng.integers(m.n_sites))
        new = int(now[s]) if i == 1 and n > 2 else int((now[s] + 1) % len(m.symbols))
        changes.append((s, int(now[s]), new))
        now[s] = new
    up.apply(changes)
    ref = DeviceUpdater(up.geo, now, eci)
    assert np.array_equal(up.occupation(), now)
    assert np.allclose(up.cf(), ref.cf(), rtol=0, atol=1e-12)
    assert up.energy() == pytest.approx(ref.energy(), abs=1e-12 * m.n_sites * np.abs(eci).sum())
    assert up.undo() == changes[::-1]
    assert np.array_equal(up.occupation(), occ0)
    assert np.array_equal(up.cf(), cf0) and up.energy() == e0 and up.history == []


@pytest.mark.parametrize("n", [2, 25])
def test_refused_changes(n):
    """A change whose old species is not on the site stops the list; what came before it stands."""
    up, m, eci, occ, _ = _updater("binary")
    changes = [(i, int(occ[i]), int(1 - occ[i])) for i in range(n)]
    changes[-1] = (n - 1, int(1 - occ[n - 1]), int(occ[n - 1]))
    with pytest.raises(RuntimeError, match="position tracker"):
        up.apply(changes)
    now = occ.copy()
    now[:n - 1] = 1 - now[:n - 1]
    assert np.array_equal(up.occupation(), now) and up.history == []
    with pytest.raises(IndexError):
        up.apply([(m.n_sites, 0, 1)])
    with pytest.raises(IndexError):
        up.apply([(-1, 0, 1)])
    with pytest.raises(ValueError):  # an empty array has no truth value; an empty list changes nothing
        up.apply(np.zeros((0, 3), dtype=int))
    up.apply([])
    assert np.array_equal(up.occupation(), now)
