"""The grid chemistry's cell-ordered neighbour search: sizes at the edges of a warp
and a block, and steps with an overfull cell (more than 128 radicals in 0.75 nm),
which walk the reference's lists; against the oracle, whose claims run in radical
order."""
import ctypes as C

import numpy as np
import pytest

import oracle
from wgdna import _lib


def clusters(n, k, sigma, seed):
    g = np.random.default_rng(seed)
    centre = np.arange(k)[:, None] * np.array([[400.0, -250.0, 130.0]])
    pos = centre[g.integers(0, k, n)] + g.normal(0, sigma, (n, 3))
    code = g.choice([0, 1, 2, 3, 5, 6, 7], n, p=[0.3, 0.2, 0.1, 0.2, 0.1, 0.05, 0.05])
    return np.ascontiguousarray(np.concatenate([pos, code[:, None]], axis=1), np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,sigma", [
    (1, 1, 1.0), (31, 3, 0.5), (33, 2, 0.5), (257, 20, 0.8),
    (30_000, 600, 1.5),        # about 50 radicals per cluster: no overfull cell
    (30_000, 15, 0.4),         # 2000 per cluster within a nanometre: overfull until they spread
])
def test_yields_against_oracle(ctx, n, k, sigma):
    """t = 0 exactly; later the mean of eight calls, whose claims race, within 2 % (the order
    of the claims, as in test_grid_chemistry_gpu_against_oracle) and 4 standard deviations of a
    count."""
    rad = clusters(n, k, sigma, n + k)
    ref, _, _ = oracle.chem_grid(rad, seed=9)
    runs = []
    for _ in range(8):
        r = _lib.ChemGridResult()
        _lib.check("grid", _lib.lib().wgdna_chem_grid(ctx.h, _lib.ptr(rad), n, 16, 1000.0, 9, C.byref(r), None, None, 0))
        runs.append(np.array(r.counts).astype(float))
        np.testing.assert_array_equal(runs[-1][0], ref[0])
    got, ref = np.mean(runs, axis=0), ref.astype(float)
    assert np.all(np.abs(got - ref) <= 0.02 * ref + 4 * np.sqrt(ref + 1)), (got, ref)


@pytest.mark.gpu
def test_captured_schedule_serves_other_sizes_and_keys(ctx):
    """Calls of 4097 to 4350 radicals share one grid size (4352), 255 does not: each
    gives its own n and key's yields, with buffers that still hold the call before."""
    for n, seed in ((4350, 3), (4097, 3), (4350, 4), (255, 5), (4200, 6)):
        rad = clusters(n, 40, 1.0, n)
        ref, _, _ = oracle.chem_grid(rad, seed=seed)
        r = _lib.ChemGridResult()
        _lib.check("grid", _lib.lib().wgdna_chem_grid(ctx.h, _lib.ptr(rad), n, 16, 1000.0, seed, C.byref(r), None, None, 0))
        got, want = np.array(r.counts).astype(float), ref.astype(float)
        assert r.chem_n == n
        np.testing.assert_array_equal(got[0], want[0])
        assert np.all(np.abs(got - want) <= 0.02 * want + 4 * np.sqrt(want + 1)), (n, seed, got, want)
