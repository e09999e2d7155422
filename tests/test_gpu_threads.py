"""Threads with cells of different sizes that launch the same kernels at the same time.

The dynamic shared memory a kernel may use is set per function, not per launch: a thread with a small cell must not
lower it between another thread's setting and launch.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KB = 8.6173303e-5


def _work(kind, L, calls, errors, start):
    from cemc_gb300 import _lib
    from cemc_gb300 import engine as E
    from cemc_gb300.calculator import DeviceUpdater
    from cemc_gb300.lattice import fcc_settings, seeded_ecis
    from cemc_gb300.tables import CEModel
    species = 3 if kind.startswith("table") else 2
    s = fcc_settings(L, 4, 2, 1, ["Al", "Mg", "Si"][:species])
    eci = seeded_ecis(s.cset, 0)
    m = CEModel(s, list(eci))
    ev = m.eci_vector(eci)
    geo = E.Geometry(m)
    stream = torch.cuda.Stream()
    occ = np.random.default_rng(L).integers(0, species, (1, m.n_sites)).astype(np.int8)
    with torch.cuda.stream(stream):
        cb = E.ChainBatch(geo, occ, ev, KB * 800.0, E.MOVE_SWAP if kind == "table_swap" else E.MOVE_FLIP, seed=1,
                          stream=stream)
        up = DeviceUpdater(geo, occ[0], ev) if kind == "delta" else None
        kernel = {"table_flip": E.KERNEL_TABLE, "table_swap": E.KERNEL_TABLE, "field": E.KERNEL_FIELD,
                  "generic": E.KERNEL_GENERIC}.get(kind, E.KERNEL_AUTO)
        run = {"recompute": cb.recompute, "delta": lambda: up.delta_flip(0, 1 - int(occ[0, 0])) if up else None}.get(
            kind, lambda: cb.run(1, precision=E.PREC_F32, kernel=kernel))
        start.wait()
        try:
            for _ in range(calls):
                run()
        except _lib.CemcError as exc:
            errors.append("%s, L = %d: %s" % (kind, L, exc))
        stream.synchronize()


# cells on both sides of the forms' sizes: speculative and scheduled flips, table flips and swaps, the local-field
# form, the generic form, the bit-plane recompute and single energy changes
@pytest.mark.parametrize("kind,sizes", [("flip", (4, 7)), ("flip", (9, 16)), ("table_flip", (6, 9)),
                                        ("table_flip", (10, 11)), ("table_swap", (12, 16)), ("field", (6, 9)),
                                        ("generic", (4, 8)), ("recompute", (6, 30)), ("delta", (4, 8))])
def test_threads_with_different_cells(kind, sizes):
    errors, start = [], threading.Barrier(4)
    calls = 3000
    threads = [threading.Thread(target=_work, args=(kind, L, calls, errors, start)) for L in sizes + sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[:3]
