"""Scoring on grids so wide that an f32 distance from the grid's corner no longer tells
where the nearest fibre is: every entry within reach is found, as by the oracle."""
import numpy as np
import pytest

import oracle
import wgdna


def near_fibres(d, n, seed, most=9e4):
    """Entries at the backbones of the fibres within `most` nm of the centre."""
    g = np.random.default_rng(seed)
    off = -(d.grid_N - 1) * d.spacing_nm / 2
    k = np.flatnonzero(np.abs(off + np.arange(d.grid_N) * d.spacing_nm) < most)
    f = g.choice(k, n) * d.grid_N + g.choice(k, n)
    b, s = g.integers(d.n_bp_per, size=n), g.integers(2, size=n)
    at = np.where(s[:, None] == 0, d.rbb0.reshape(-1, 2)[b], d.rbb1.reshape(-1, 2)[b])
    xyz = np.stack([d.x0 + b * d.rise, d.fy[f] + at[:, 0], d.fz[f] + at[:, 1]], axis=1) + g.normal(0, 0.1, (n, 3))
    return np.concatenate([xyz, np.zeros((n, 1))], axis=1).astype(np.float32)


def f32_offset(y, off, sp):
    """The offset from the nearest axis as f32 arithmetic gives it."""
    f = np.float32
    u = (y - f(off)) * f(1 / sp)
    return np.abs(u - np.rint(u)) * f(sp)


WIDE = [(101, 40_000.3), (1001, 1999.9)]


@pytest.mark.parametrize("n,sp", WIDE)
def test_the_f32_offset_fails_there(n, sp):
    d = oracle.DnaTarget(L_nm=20.0, grid_N=n, spacing_nm=sp)
    rad = near_fibres(d, 20_000, 1)
    off = -(n - 1) * sp / 2
    assert np.any(np.maximum(f32_offset(rad[:, 1], off, sp), f32_offset(rad[:, 2], off, sp)) > 1.34)


@pytest.mark.gpu
@pytest.mark.parametrize("n,sp", WIDE + [(21, 150.0), (3, 90_000.0), (1, 1e7)])
def test_direct_scoring_on_wide_grids(n, sp):
    d = oracle.DnaTarget(L_nm=20.0, grid_N=n, spacing_nm=sp)
    dna = wgdna.build_dna_target(L_nm=20.0, grid_N=n, spacing_nm=sp)
    ctx = wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000)
    try:
        rad = near_fibres(d, 20_000, 1)
        rng = wgdna.make_ssb_rng()
        got = wgdna.score_direct_ssb_events(ctx, dna, rad, rad.shape[0], rng)
        ref = oracle.score_direct(d, rad, 0x12345678)
        assert ref["in_reach"] > 1000
        assert (got["ssb_count"], got["candidates"], got["in_reach"]) == (ref["ssb"], ref["candidates"], ref["in_reach"])
        assert rng.state == ref["lcg_state"]
        np.testing.assert_array_equal(got["hits"], ref["hits"])
    finally:
        ctx.close()
