"""The IRT pairing kernel passes by chunks of 32 partners that lie beyond R_CUT (551 nm)
of a tile of 32 particles: long tracks whose entries come in order of their place, with
groups of entries just inside and just beyond R_CUT of one another, bit for bit
against the oracle (pairs inside R_CUT are counted)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from wgdna import _lib


def line(n, step, jitter, group, codes, pid, g):
    """n entries, `group` of them at each place of a line, places `step` nm apart."""
    x = np.repeat(np.arange(n // group + 1), group)[:n] * step
    pos = g.normal(0, jitter, (n, 3))
    pos[:, 0] += x
    return np.concatenate([pos, (g.choice(codes, n) + 8 * pid)[:, None]], axis=1)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,step,jitter,group", [
    ((1300,), 3.0, 2.0, 1),                      # 3.9 um
    ((33, 64, 65, 500), 40.0, 1.0, 4),
    ((640,), 551.0, 1e-3, 32),                   # chunks at R_CUT itself
    ((640, 96), 550.5, 0.4, 16),
    ((640, 700), 275.6, 0.2, 32),                # every second one at R_CUT
    ((1000,), 5000.0, 1.0, 8),                   # everything else far away
])
def test_far_chunks_bit_exact(ctx, sizes, step, jitter, group):
    g = np.random.default_rng(len(sizes) + group)
    rad = np.ascontiguousarray(np.concatenate([line(n, step, jitter, group, (0, 1, 2, 3, 5, 6), k, g)
                                               for k, n in enumerate(sizes)]), np.float32)
    ref = oracle.irt(rad, len(sizes), 1000.0, seed=37)
    r = _lib.IrtResult()
    _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], len(sizes), 1000.0, 37,
                                                         C.byref(r)))
    np.testing.assert_array_equal(np.array(r.counts), ref["tl"])
    np.testing.assert_array_equal(np.array(r.rxn_counts[:]), ref["rxn_counts"])
    assert (r.n_reacted, r.n_pairs, r.n_events) == (ref["n_reacted"], ref["n_pairs"], ref["n_events"])
