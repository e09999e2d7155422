"""The spin forms of several flips a warp are refused for their limits only: the argument error, for expansions of more
cluster ECIs than lanes; everything else runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KB = 8.6173303e-5


@pytest.mark.parametrize("recipe", [(1, 0, 0), (4, 2, 1), (2, 2, 2), (2, 3, 2), (2, 4, 1), (3, 1, 4)])
@pytest.mark.parametrize("kernel,lanes", [("SPIN_HALFWARP", 16), ("SPIN_QUARTER", 8)])
@pytest.mark.parametrize("warps", [1, 4, 16])
def test_refused_for_their_limits_only(recipe, kernel, lanes, warps):
    from cemc_gb300 import _lib, engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(6, *recipe, ["Al", "Mg"])
    eci = seeded_ecis(s.cset, 1)
    m = CEModel(s, list(eci))
    kind, n_terms = np.asarray(m.eci_kind), np.bincount(np.asarray(m.term_eci), minlength=m.n_eci)
    multi = np.bincount(np.asarray(m.term_eci)[np.asarray(m.term_size) > 2], minlength=m.n_eci)
    clusters = int(((kind == 2) & (n_terms > 0)).sum())
    occ = np.random.default_rng(2).integers(0, 2, (1, m.n_sites)).astype(np.int8)
    cb = E.ChainBatch(E.Geometry(m), occ, m.eci_vector(eci), KB * 700.0, E.MOVE_FLIP, seed=9)
    kw = dict(precision=E.PREC_F64, kernel=getattr(E, "KERNEL_" + kernel), warps=warps, cluster=1)
    fits = clusters <= lanes and (kernel == "SPIN_HALFWARP" or multi.max() <= 255)
    if fits:
        cb.run(100, **kw)
        cb.check_status()
        assert cb.last_kernel == kw["kernel"]
    else:
        with pytest.raises(_lib.CemcError) as exc:
            cb.run(100, **kw)
        assert exc.value.code == _lib.ERR_ARG
        cb.run(100, precision=E.PREC_F64, warps=min(warps, 4))  # the library's own choice takes it
        cb.check_status()
