"""One warp per track, four tracks to a block that go from one re-pairing to the next
together: blocks whose warps come to the meeting a very different number of times, or
never, bit for bit against the oracle; and no barrier of the event kernel that CUDA wants
reached by the whole block under one condition stands where warps diverge."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import oracle
from test_irt_tiles import tracks
from wgdna import _lib

IRT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgpu-dna_b200", "csrc", "irt.cu")


def test_event_kernel_has_no_block_wide_cuda_barrier():
    with open(IRT) as f:
        text = "\n".join(line.split("//")[0] for line in f)
    body = text[text.index("k_irt_loop("):text.index("k_group_keys(")]
    assert not re.search(r"__syncthreads\w*\s*\(", body)


@pytest.mark.gpu
@pytest.mark.parametrize("n_tracks,every,size", [(1185, 1185, 900), (2369, 400, 700), (9471, 37, 120), (2500, 3, 60)])
def test_tracks_of_very_different_lengths(ctx, n_tracks, every, size):
    """Most tracks have one or two species and no reaction."""
    sizes = np.random.default_rng(every).integers(1, 3, n_tracks)
    sizes[::every] = size
    rad = tracks(list(sizes), (0, 1, 2, 3, 5, 6), 30.0, every)
    ref = oracle.irt(rad, n_tracks, 1000.0, seed=31)
    r = _lib.IrtResult()
    _lib.check("wgdna_run_irt", _lib.lib().wgdna_run_irt(ctx.h, _lib.ptr(rad), rad.shape[0], n_tracks, 1000.0, 31,
                                                         C.byref(r)))
    np.testing.assert_array_equal(np.array(r.counts), ref["tl"])
    np.testing.assert_array_equal(np.array(r.rxn_counts[:]), ref["rxn_counts"])
    assert (r.n_reacted, r.n_pairs, r.n_events) == (ref["n_reacted"], ref["n_pairs"], ref["n_events"])
