"""FP64 launches with ECI coefficients in fixed point: energy changes of ECIs of very different magnitudes.

Reference: the coefficients as FP64 numbers, the integer counts, and exact rational sums, along the traced chain.
Bound where the coefficients span less than 2^18: the sum is exact and rounded once (2^-53 of it; 2^-52 asked).  Where
they span more, FP64 arithmetic stays: each of K products and K + 1 sums rounds to 2^-53 of a partial sum.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


def _exact(m, ev, occ, sites, new, acc, move):
    """(energy change, sum of the magnitudes of its parts) of every trial along the chain."""
    spin = np.asarray(m.bf).reshape(-1)
    coef = {k: ev[k] * float(m.n_sites) * m.eci_weight[k] for k in range(m.n_eci) if m.eci_kind[k] == 2}
    sing = sum(ev[k] for k in range(m.n_eci) if m.eci_kind[k] == 1)
    nb, size, eci = np.asarray(m.term_nb).reshape(-1, 3), np.asarray(m.term_size), np.asarray(m.term_eci)
    table, occ = np.asarray(m.gpu_table), occ.astype(np.int64).copy()

    def counts(site):
        s = spin[occ[table[site]]].astype(np.int64)
        prod = np.ones(len(eci), dtype=np.int64)
        for j in range(3):
            prod = np.where(size - 1 > j, prod * s[nb[:, j]], prod)
        return {k: int(prod[eci == k].sum()) for k in coef}

    out = []
    for (a, b), nw, ok in zip(sites, new, acc):
        delta = int(spin[nw] - spin[occ[a]]) if move == 0 else int(spin[occ[b]] - spin[occ[a]])
        p = counts(a)
        old = occ[a], occ[b]
        if move == 1:
            occ[a] = old[1]
            q = counts(b)
            p = {k: p[k] - q[k] for k in p}
            occ[a] = old[0]
        parts = [Fraction(coef[k]) * p[k] * delta for k in p] + ([Fraction(sing) * delta] if move == 0 else [])
        out.append((sum(parts, Fraction(0)), float(sum(abs(x) for x in parts))))
        if ok:
            if move == 0:
                occ[a] = nw
            else:
                occ[a], occ[b] = old[1], old[0]
    return out


# the small cell's forms, swaps, and the scheduled kernel (always taken at 16,384 sites)
@pytest.mark.parametrize("L,kernel,warps,move", [(6, "SPIN_HALFWARP", 2, 0), (6, "SPIN_QUARTER", 2, 0),
                                                 (6, "SPIN", 3, 0), (6, "SPIN", 3, 1), (16, "SPIN_QUARTER", 8, 0)])
@pytest.mark.parametrize("span", [1.0, 1e-5, 1e-12])
def test_spin_forms(L, kernel, warps, move, span):
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    s = fcc_settings(L, 4, 2, 1, ["Al", "Mg"])
    eci = seeded_ecis(s.cset, 1)
    m = CEModel(s, list(eci))
    ev = m.eci_vector(eci)
    pair = int(np.nonzero(np.asarray(m.eci_kind) == 2)[0][0])  # one large ECI, often of a zero count
    scale = np.abs(ev[np.asarray(m.eci_kind) != 0]).max()
    ev = np.where(np.arange(m.n_eci) == pair, 0.1, ev / scale * 0.1 * span)
    occ = np.random.default_rng(4).integers(0, 2, (1, m.n_sites)).astype(np.int8)
    cb = E.ChainBatch(E.Geometry(m), occ, ev, KB * 3000.0, move, seed=6)
    n = 300
    site, acc, de = cb.run(n, precision=E.PREC_F64, kernel=getattr(E, "KERNEL_" + kernel), warps=warps, cluster=1,
                           trace=True)
    torch.cuda.synchronize()
    cb.check_status()
    assert getattr(cb, "last_scheduled", None) == (1 if L == 16 else 0)
    site, acc, de = site.cpu().numpy()[0], acc.cpu().numpy()[0], de.cpu().numpy()[0]
    ref = _exact(m, ev, occ[0], [(a, b if move else 0) for a, b in site], site[:, 1], acc, move)
    K = int((np.asarray(m.eci_kind) == 2).sum())
    for got, (want, parts) in zip(de, ref):
        bound = 2.0 ** -52 * abs(float(want)) if span > 1e-6 else (2 * K + 3) * 2.0 ** -53 * parts
        assert abs(float(Fraction(float(got)) - want)) <= bound
    assert (np.abs([float(w) for w, _ in ref]) < 0.01).sum() > 10 or span == 1.0  # trials without the large ECI


def _table_exact(m, ev, occ, site, new, acc, move, groups):
    """(energy change, sum of the magnitudes of its terms) of every trial along the chain, with the products of basis
    values and coefficients as exact rationals."""
    bf = [[Fraction(float(x)) for x in row] for row in np.asarray(m.bf).reshape(m.n_bf, m.n_sym)]
    coef = [Fraction(float(ev[k] * float(m.n_sites) * m.eci_weight[k])) for k in range(m.n_eci)]
    nb, size = np.asarray(m.term_nb).reshape(-1, 3), np.asarray(m.term_size)
    eci, ref = np.asarray(m.term_eci), np.asarray(m.term_ref)
    table, occ = np.asarray(m.gpu_table), occ.astype(int).copy()

    def change(i, old, nw):
        g = int(groups[i])
        total = mags = Fraction(0)
        for t in range(int(m.group_terms[g]), int(m.group_terms[g + 1])):
            p = coef[eci[t]] * (bf[ref[t]][nw] - bf[ref[t]][old]) * Fraction(float(m.group_scale[g]))
            for j in range(size[t] - 1):
                col, d = divmod(int(nb[t, j]), m.n_bf)
                p *= bf[d][occ[table[i, col]]]
            total, mags = total + p, mags + abs(p)
        if move == 0:
            for k in range(m.n_eci):
                if m.eci_kind[k] == 1:
                    p = Fraction(float(ev[k])) * (bf[m.eci_dec[k]][nw] - bf[m.eci_dec[k]][old])
                    total, mags = total + p, mags + abs(p)
        return total, mags

    out = []
    for (a, b), ok in zip(site, acc):
        old = occ[a], occ[b] if move else 0
        nw = old[1] if move else int(b)
        de, mags = change(a, old[0], nw)
        if move:
            occ[a] = nw
            e2, m2 = change(b, old[1], old[0])
            de, mags = de + e2, mags + m2
            occ[a] = old[0]
        out.append((de, float(mags)))
        if ok:
            occ[a] = nw
            if move:
                occ[b] = old[0]
    return out


# the speculative table form (flips, swaps, two groups) and the scheduled one (swaps of 10,976 sites)
@pytest.mark.parametrize("cell,L,move", [("fcc", 4, 0), ("fcc", 4, 1), ("hcp", 5, 0), ("fcc", 14, 1)])
@pytest.mark.parametrize("span", [1.0, 1e-4, 1e-12, "singlets"])
def test_table_form(cell, L, move, span):
    """Entries are sums of products evaluated in FP64 (at most 10 roundings of 2^-53 of the terms' magnitudes), and their
    sum has no further rounding but the last one; FP64 sums (span 1e-12) add n roundings of partial sums.  Singlet ECIs
    of 10^6 eV are no part of a swap's energy change and must not coarsen it."""
    if span == "singlets" and move == 0:
        pytest.skip("swaps only")
    big, span = span == "singlets", 1.0 if span == "singlets" else span
    from cemc_gb300 import engine as E
    from cemc_gb300.lattice import fcc_settings, hcp_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    names = ["Al", "Mg", "Si"]
    s = fcc_settings(L, 2, 1, 0, names) if cell == "fcc" else hcp_settings(L, 5, 1, 1, 0, names)
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    ev = m.eci_vector(eci)
    kind = np.asarray(m.eci_kind)
    large = int(np.nonzero(kind == 2)[0][0])
    ev = np.where(np.arange(m.n_eci) == large, 0.1, ev / np.abs(ev[kind != 0]).max() * 0.1 * span)
    if span < 1e-9:  # a coefficient too far below the others
        ev[kind == 1] = 0.05
    if big:
        ev[kind == 1] = 1e6
    occ = np.random.default_rng(4).integers(0, 3, (1, m.n_sites)).astype(np.int8)
    cb = E.ChainBatch(E.Geometry(m), occ, ev, KB * 3000.0, move, seed=6)
    n = 40
    if L == 14:  # calls of fewer trials are not scheduled: the trace's first trials are compared
        site, acc, de = cb.run(2100, precision=E.PREC_F64, kernel=E.KERNEL_TABLE, warps=8, cluster=1, trace=True)
        assert getattr(cb, "last_scheduled", None) == 2
    else:
        site, acc, de = cb.run(n, precision=E.PREC_F64, kernel=E.KERNEL_TABLE, warps=4, cluster=1, trace=True)
    torch.cuda.synchronize()
    cb.check_status()
    site, acc, de = site.cpu().numpy()[0][:n], acc.cpu().numpy()[0][:n], de.cpu().numpy()[0][:n]
    groups = np.asarray(m.site_group) if m.n_groups > 1 else np.zeros(m.n_sites, dtype=int)
    ref = _table_exact(m, ev, occ[0], site, site[:, 1], acc, move, groups)
    terms = m.n_terms * (2 if move else 1)
    for got, (want, mags) in zip(de, ref):
        bound = (10 + (terms if span < 1e-9 else 0)) * 2.0 ** -53 * mags + 2.0 ** -53 * abs(float(want))
        assert abs(float(Fraction(float(got)) - want)) <= bound
