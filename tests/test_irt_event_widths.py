"""The IRT event kernel with 1, 2, 4, 8 and 16 warps per track (it takes more of them
the fewer tracks there are), and a track too large for the species states and the
heap nodes in shared memory among small ones, bit for bit against the oracle: all
outputs are whole numbers, so nothing may differ."""
import ctypes as C

import numpy as np
import pytest

import oracle
from test_irt_tiles import tracks
from wgdna import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("n_tracks,large,spread", [
    (3, 0, 20.0),
    (1, 8192, 1200.0),                   # the largest track that is taken
    (100, 0, 15.0),
    (90, 3000, 250.0),
    (250, 0, 15.0),
    (200, 4200, 250.0),
    (1000, 0, 15.0),
    (900, 4200, 250.0),
    (2500, 0, 15.0),
    (2400, 2300, 150.0),
    (2400, 4200, 250.0),
])
def test_event_widths_bit_exact(ctx, n_tracks, large, spread):
    g = np.random.default_rng(n_tracks)
    sizes = list(g.integers(1, 70, n_tracks))
    if large:
        sizes[n_tracks // 2] = large
    rad = tracks(sizes, (0, 1, 2, 3, 5, 6), spread, n_tracks + 5)
    ref = oracle.irt(rad, n_tracks, 1000.0, seed=23)
    r = _lib.IrtResult()
    _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], n_tracks, 1000.0, 23,
                                                         C.byref(r)))
    np.testing.assert_array_equal(np.array(r.counts), ref["tl"])
    np.testing.assert_array_equal(np.array(r.rxn_counts[:]), ref["rxn_counts"])
    assert (r.n_reacted, r.n_pairs, r.n_events) == (ref["n_reacted"], ref["n_pairs"], ref["n_events"])


@pytest.mark.gpu
def test_larger_track_is_refused(ctx):
    """More than 8192 entries in one track end in an error, and the context still works."""
    rad = tracks([16400], (0, 1, 2, 3, 5, 6), 2500.0, 6)
    r = _lib.IrtResult()
    with pytest.raises(_lib.WgdnaError):
        _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], 1, 1000.0, 23, C.byref(r)))
    test_event_widths_bit_exact(ctx, 3, 0, 20.0)
