"""Large copies to and from pageable host memory go through page-locked slots by several
threads; smaller ones and those of page-locked memory do not.  The bytes have to be the same
either way, at sizes around the threshold (4 MiB), the slots (512 KiB) and the
threads' parts."""
import ctypes as C

import numpy as np
import pytest
import torch

import wgdna
from wgdna import _lib

SIZES = (262143, 262144, 262145, 294913, 300001, 524288, 700003)      # of 16 bytes each


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_both_directions_keep_every_byte(n):
    L = _lib.lib()
    ctx = wgdna.Context(max_primaries=1024, max_rad=2_000_000, max_sec=300_000)
    p = wgdna.transport_params(700, 1e4, 15000.0, 7.5, seed=9, dna_enable=0)
    st = _lib.TransportStats()
    _lib.check("wgdna_transport", L.wgdna_transport(ctx.h, C.byref(p), C.byref(st)))
    assert st.rad_n_stored >= n
    got = C.c_uint64()

    def out(buf, elems):
        _lib.check("copy_out", L.wgdna_transport_copy_out(ctx.h, None, None, C.c_void_p(buf), elems, C.byref(got)))

    locked = torch.full((n, 4), -1.0, dtype=torch.float32).pin_memory()
    out(locked.data_ptr(), n)
    guarded = np.full((n + 2, 4), -7.0, np.float32)
    out(guarded[1:].ctypes.data, n)
    np.testing.assert_array_equal(guarded[1:-1].view(np.uint32), locked.numpy().view(np.uint32))
    assert (guarded[0] == -7).all() and (guarded[-1] == -7).all()

    # back up: the chemistry of the same entries from either memory
    res = []
    for buf in (locked.data_ptr(), guarded[1:].ctypes.data):
        r = _lib.IrtResult()
        _lib.check("wgdna_run_irt", L.wgdna_run_irt(ctx.h, C.c_void_p(buf), n, 700, 1e4, 3, C.byref(r)))
        res.append((list(r.rxn_counts), r.n_pairs, r.n_events, r.n_reacted, np.array(r.counts).tolist()))
    assert res[0] == res[1]
    ctx.close()
