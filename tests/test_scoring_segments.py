"""Direct SSB scoring over segments of 512 entries: list lengths at a segment's and a
block's edges, and runs of equal positions that start, end or lie across them
(the reference's walk visits every second entry of a run), bit for bit against the
oracle."""
import numpy as np
import pytest

import oracle
import wgdna


def sites(dna, runs, seed):
    """One backbone site (or one far point) per run, repeated."""
    g = np.random.default_rng(seed)
    out = []
    for k in runs:
        if g.random() < 0.7:
            f, b, s = g.integers(dna.n_fibers), g.integers(dna.n_bp_per), g.integers(2)
            off = (dna.rbb0 if s == 0 else dna.rbb1)[2 * b: 2 * b + 2]
            p = (dna.x0 + b * dna.rise + g.normal(0, 0.1), dna.fy[f] + off[0] + g.normal(0, 0.1),
                 dna.fz[f] + off[1] + g.normal(0, 0.1))
        else:
            p = g.uniform(-2000, 2000, 3)
        out += [(*p, 0.0)] * int(k)
    return np.array(out, np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("runs", [
    [1], [2], [511], [512], [513], [1, 511, 1], [1, 512, 1], [3, 1021, 7, 512, 5],
    [5000], [1, 20000, 2, 3],                                   # runs over many segments
    list(range(1, 90)), [1] * 4095 + [2] + [1] * 33,
    [40000] + [1, 2, 3] * 400,                                  # 148 blocks' worth of one run
])
def test_direct_scoring_at_segment_edges(ctx, runs):
    dna, od = wgdna.build_dna_target(), oracle.DnaTarget()
    rad = sites(dna, runs, len(runs) + runs[0])
    rng = wgdna.make_ssb_rng()
    got = wgdna.score_direct_ssb_events(ctx, dna, rad, rad.shape[0], rng)
    ref = oracle.score_direct(od, rad, 0x12345678)
    assert (got["ssb_count"], got["candidates"], got["in_reach"]) == (ref["ssb"], ref["candidates"], ref["in_reach"])
    assert rng.state == ref["lcg_state"]
    np.testing.assert_array_equal(got["hits"], ref["hits"])


@pytest.mark.gpu
@pytest.mark.parametrize("every", [1, 7, 8823])
def test_cluster_at_fibre_edges(ctx, every):
    """Hits on the first and last base pairs of fibres (8823 bp: fibres start at any byte of a
    word), bytes other than 1 that do not count, and a full strand."""
    dna, od = wgdna.build_dna_target(), oracle.DnaTarget()
    hits = np.zeros(2 * dna.n_bp, np.uint8)
    hits[::every] = 1
    hits[5::every] = 3
    edge = np.arange(1, dna.n_fibers) * dna.n_bp_per
    hits[edge] = 1
    hits[dna.n_bp + edge - 1] = 1
    got, ref = wgdna.cluster_dsb(ctx, dna, hits), oracle.cluster_dsb(od, hits)
    assert (got["dsb"], got["ssb0"], got["ssb1"]) == (ref["dsb"], ref["ssb0"], ref["ssb1"])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 512, 513, 1537])
def test_scoring_scratch_of_a_full_context(n):
    """As many entries as the context holds, every one near a site and drawn once: lists and summaries
    at their largest in the keys' buffer."""
    dna, od = wgdna.build_dna_target(), oracle.DnaTarget()
    ctx = wgdna.Context(max_primaries=4, max_rad=n, max_sec=1000)
    try:
        g = np.random.default_rng(n)
        b, f = g.integers(dna.n_bp_per, size=n), g.integers(dna.n_fibers, size=n)
        off = dna.rbb0.reshape(-1, 2)[b]
        rad = np.stack([dna.x0 + b * dna.rise, dna.fy[f] + off[:, 0], dna.fz[f] + off[:, 1], np.zeros(n)], 1).astype(np.float32)
        for _ in range(2):
            rng = wgdna.make_ssb_rng()
            got = wgdna.score_direct_ssb_events(ctx, dna, rad, n, rng)
            ref = oracle.score_direct(od, rad, 0x12345678)
            assert (got["ssb_count"], got["candidates"], got["in_reach"]) == (ref["ssb"], ref["candidates"], ref["in_reach"])
            assert rng.state == ref["lcg_state"]
            np.testing.assert_array_equal(got["hits"], ref["hits"])
    finally:
        ctx.close()
