"""The order of a track's initial events (t, i, j) where one block sorts them in shared
memory (up to 4096), in the track's slots (more, in a short track), and where chunks of
2048 are sorted and merged: bit for bit against the oracle, whose events run in that
order; all outputs are whole numbers, so nothing may differ."""
import ctypes as C

import numpy as np
import pytest

import oracle
from test_irt_tiles import tracks
from wgdna import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,spread", [
    ((470,), 6.0),                               # short and dense
    ((1000,), 25.0),                             # about one block's limit
    ((1500,), 40.0),                             # 4 chunks
    ((3000,), 45.0),
    ((8192,), 85.0),                             # the longest track, dense
    ((1500, 20, 1600, 5, 1700, 1, 300), 38.0),   # large and small tracks
    ((1500,) * 40 + (3,) * 30, 38.0),
])
def test_sorted_events_bit_exact(ctx, sizes, spread):
    rad = tracks(sizes, (0, 1, 2, 5), spread, len(sizes) + sizes[0])
    ref = oracle.irt(rad, len(sizes), 1000.0, seed=29)
    r = _lib.IrtResult()
    _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], len(sizes), 1000.0, 29,
                                                         C.byref(r)))
    np.testing.assert_array_equal(np.array(r.counts), ref["tl"])
    np.testing.assert_array_equal(np.array(r.rxn_counts[:]), ref["rxn_counts"])
    assert (r.n_reacted, r.n_pairs, r.n_events) == (ref["n_reacted"], ref["n_pairs"], ref["n_events"])
