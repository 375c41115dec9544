"""SamplePDC in the IRT pairing kernel: pairs wait in a queue of 96 per warp, are taken by
lanes, go back with their place in the trials or end in whole-warp rounds.  Bit for bit
against the oracle with few and many pairs per warp and with pairs of many tracks
in one queue: all outputs are whole numbers, so nothing may differ."""
import ctypes as C

import numpy as np
import pytest

import oracle
from test_irt_tiles import tracks
from wgdna import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("n_tracks,lo,hi,codes,spread", [
    (1, 2, 3, (0, 1), 0.5),                      # one pair at most
    (7, 5, 12, (0, 1, 2, 5), 1.0),               # a few: whole-warp rounds alone
    (40, 30, 70, (0, 1, 2, 5), 3.0),
    (1, 900, 901, (0, 1, 2, 5), 25.0),           # dense: the queue runs over within one tile
    (3, 300, 420, (0,), 8.0),
    (6000, 2, 9, (0, 1, 2, 5), 1.0),             # many tracks in one queue
    (4000, 1, 120, (0, 1, 2, 3, 5, 6), 4.0),
])
def test_queued_pairs_bit_exact(ctx, n_tracks, lo, hi, codes, spread):
    g = np.random.default_rng(n_tracks + hi)
    rad = tracks(list(g.integers(lo, hi, n_tracks)), codes, spread, n_tracks + lo)
    ref = oracle.irt(rad, n_tracks, 1000.0, seed=31)
    r = _lib.IrtResult()
    _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], n_tracks, 1000.0, 31,
                                                         C.byref(r)))
    np.testing.assert_array_equal(np.array(r.counts), ref["tl"])
    np.testing.assert_array_equal(np.array(r.rxn_counts[:]), ref["rxn_counts"])
    assert (r.n_reacted, r.n_pairs, r.n_events) == (ref["n_reacted"], ref["n_pairs"], ref["n_events"])
