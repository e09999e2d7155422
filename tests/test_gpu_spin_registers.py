"""Two and four flips per warp with the lane's terms in registers (at most four multi-site ECIs and a
few terms a lane) and without, against one flip per warp: the chain is the same chain.

The proposals, energy changes (integer counts times the same coefficients) and acceptances of the forms are
those of one sequential chain, so the occupation and the accept count agree exactly and the correlation functions,
integer sums scaled once, to rounding (1e-12); energies add the same FP64 terms in another grouping (1e-9).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KB = 8.6173303e-5


@pytest.mark.parametrize("recipe", [(1, 0, 0), (4, 2, 1), (2, 2, 2), (2, 3, 2), (2, 4, 1), (3, 1, 4)])
@pytest.mark.parametrize("kernel,warps", [("HALF", 1), ("HALF", 4), ("HALF", 16), ("QTR", 1), ("QTR", 4), ("QTR", 8)])
def test_same_chain(recipe, kernel, warps):
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(6, *recipe, ["Al", "Mg"])
    eci = seeded_ecis(s.cset, 1)
    m = CEModel(s, list(eci))
    geo = E.Geometry(m, "cuda")
    C = 3
    occ = np.random.default_rng(2).integers(0, 2, (C, m.n_sites)).astype(np.int8)
    ev, kT = np.tile(m.eci_vector(eci), (C, 1)), KB * np.array([300.0, 700.0, 3000.0])
    out = []
    forms = {"HALF": E.KERNEL_SPIN_HALFWARP, "QTR": E.KERNEL_SPIN_QUARTER}
    for k, w in ((E.KERNEL_SPIN, 4), (forms[kernel], warps)):
        cb = E.ChainBatch(geo, occ, ev, kT, E.MOVE_FLIP, seed=9)
        try:
            cb.run(1000 + 37, precision=E.PREC_F64, kernel=k, warps=w, cluster=1)
        except RuntimeError as exc:
            pytest.skip("form not available for this expansion: %s" % exc)
        cb.check_status()
        out.append((cb.occ.cpu().numpy(), cb.cf.cpu().numpy(), cb.energy.cpu().numpy(),
                    cb.accum.cpu().numpy()[:, :E.A_NSAMP], cb.accum[:, E.A_NSAMP:].cpu().numpy().view(np.int64)))
    (o0, c0, e0, s0, n0), (o1, c1, e1, s1, n1) = out
    assert np.array_equal(o0, o1) and np.array_equal(n0[:, :2], n1[:, :2])
    assert np.allclose(c0, c1, rtol=0, atol=1e-12)
    assert np.allclose(e0, e1, rtol=1e-9, atol=1e-9) and np.allclose(s0, s1, rtol=1e-9, atol=1e-6)


@pytest.mark.parametrize("recipe", [(1, 0, 0), (4, 2, 1), (2, 2, 2), (2, 3, 2), (2, 4, 1)])
@pytest.mark.parametrize("move", ["FLIP", "SWAP"])
@pytest.mark.parametrize("warps,cluster", [(1, 1), (5, 1), (16, 1), (4, 2)])
@pytest.mark.parametrize("prec", ["F64", "F32"])
def test_one_move_per_warp(recipe, move, warps, cluster, prec):
    """One flip or swap per warp (differences of two sites' counts, the uniform's parts and list slots by
    the fetcher) against the generic form.  In FP32 a uniform that falls between the two forms' rounded
    energy changes (1e-6 of kT) would part the chains: 1037 x 3 trials meet one with probability 0.3 %."""
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(6, *recipe, ["Al", "Mg"])
    eci = seeded_ecis(s.cset, 1)
    m = CEModel(s, list(eci))
    geo = E.Geometry(m, "cuda")
    C = 3
    occ = np.random.default_rng(2).integers(0, 2, (C, m.n_sites)).astype(np.int8)
    ev, kT = np.tile(m.eci_vector(eci), (C, 1)), KB * np.array([300.0, 700.0, 3000.0])
    out = []
    for k, w, c in ((E.KERNEL_GENERIC, 4, 1), (E.KERNEL_SPIN, warps, cluster)):
        cb = E.ChainBatch(geo, occ, ev, kT, getattr(E, "MOVE_" + move), seed=9)
        cb.run(1000 + 37, precision=getattr(E, "PREC_" + prec), kernel=k, warps=w, cluster=c)
        cb.check_status()
        out.append((cb.occ.cpu().numpy(), cb.cf.cpu().numpy(), cb.accum[:, E.A_NSAMP:].cpu().numpy().view(np.int64)))
    (o0, c0, n0), (o1, c1, n1) = out
    assert np.array_equal(o0, o1) and np.array_equal(n0[:, :2], n1[:, :2])
    # FP32 launches of the generic form add the changes of the correlation functions in double-float
    assert np.allclose(c0, c1, rtol=0, atol=1e-12 if prec == "F64" else 1e-6)
