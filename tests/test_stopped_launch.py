"""What a host does after a consistency check stopped a chain's launch (CEMC_ERR_INTERNAL), with a fake of the status."""
from types import SimpleNamespace

import numpy as np
import pytest

torch = pytest.importorskip("torch")


def test_site_lists_of_a_stopped_chain_are_rebuilt():
    from cemc_gb300 import _lib, engine as E
    occ = np.random.default_rng(0).integers(0, 3, (3, 40)).astype(np.int8)
    trk, loc, start, count = E.build_tracker(occ, 3)
    cb = E.ChainBatch.__new__(E.ChainBatch)
    cb.geo = SimpleNamespace(model=SimpleNamespace(n_sym=3, background=[]))
    cb.occ = torch.as_tensor(occ)
    moved = trk.copy()
    moved[:, [0, 39]] = moved[:, [39, 0]]  # a swap that the occupations do not have
    cb.trk, cb.loc = torch.as_tensor(moved), torch.as_tensor(loc.copy())
    cb.trk_start, cb.trk_count = torch.as_tensor(start), torch.as_tensor(count)
    cb.status = torch.tensor([0, _lib.ERR_INTERNAL, 0], dtype=torch.int32)
    place = cb.trk.data_ptr()
    with pytest.raises(_lib.CemcError, match="chain 1"):
        cb.check_status()
    assert cb.trk.data_ptr() == place  # in place: captured launches go on using it
    assert np.array_equal(cb.trk[1].numpy(), trk[1]) and np.array_equal(cb.loc[1].numpy(), loc[1])
    assert np.array_equal(cb.trk[0].numpy(), moved[0])  # the other chains' lists are theirs
