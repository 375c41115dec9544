"""The IRT pairing kernel's tiles (32 particles of one species, partners in
Philox blocks of 4, staged 32 at a time) at the sizes where they can go wrong,
bit for bit against the oracle: counts, reactions, pairs inside R_CUT and events
are whole numbers, so nothing may differ."""
import ctypes as C

import numpy as np
import pytest

import oracle
from wgdna import _lib


def tracks(sizes, codes, spread, seed):
    """One track per size: entries of the given codes, clustered in spurs over +-spread nm."""
    g = np.random.default_rng(seed)
    out = []
    for pid, n in enumerate(sizes):
        centre = g.uniform(-spread, spread, (n // 6 + 1, 3))
        pos = centre[g.integers(0, len(centre), n)] + g.normal(0, 1.5, (n, 3))
        w = g.choice(codes, n) + 8 * pid
        out.append(np.concatenate([pos, w[:, None]], axis=1))
    return np.ascontiguousarray(np.concatenate(out), np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,codes,spread", [
    ((1, 2, 3, 4, 5), (0, 1), 2.0),
    ((31, 32, 33, 63, 64, 65), (0, 1, 2, 3, 5, 6), 20.0),
    ((127, 128, 129, 1, 500), (0,), 60.0),                 # one species: every pair can react
    ((40, 41, 42), (3,), 5.0),                             # one species that does not react with itself
    ((96, 200), (3, 6), 8.0),                              # Coulomb TDC only
    ((700, 1031), (0, 1, 2, 3, 4, 5, 6, 7), 900.0),        # most pairs beyond R_CUT (551 nm)
    ((300, 301), (0, 1, 5), 320.0),                        # many near R_CUT
])
def test_pairing_tiles_bit_exact(ctx, sizes, codes, spread):
    rad = tracks(sizes, codes, spread, len(sizes) + sizes[0])
    ref = oracle.irt(rad, len(sizes), 1000.0, seed=17)
    r = _lib.IrtResult()
    _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], len(sizes), 1000.0, 17,
                                                         C.byref(r)))
    np.testing.assert_array_equal(np.array(r.counts), ref["tl"])
    np.testing.assert_array_equal(np.array(r.rxn_counts[:]), ref["rxn_counts"])
    assert (r.n_reacted, r.n_pairs, r.n_events) == (ref["n_reacted"], ref["n_pairs"], ref["n_events"])
