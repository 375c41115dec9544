"""Dose scoring after a change of the DNA target: the per-site arrays have the new target's
size, larger or smaller, against the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle
import wgdna
from wgdna import _lib


@pytest.mark.gpu
def test_dose_scoring_on_targets_of_other_sizes():
    dose = np.ascontiguousarray(oracle.transport(48, 10000.0, seed=6, rng_mode=0)["dose"])
    L, ctx = _lib.lib(), wgdna.Context(max_primaries=64, max_rad=1_000_000, max_sec=100_000)
    try:
        for size in ((300.0, 3, 30.0), (3000.0, 21, 150.0), (300.0, 3, 30.0)):
            d = oracle.DnaTarget(*size)
            _lib.check("target", L.wgdna_set_dna_target(ctx.h, *size))
            hits = (np.random.default_rng(7).random(2 * d.n_bp) < 0.01).astype(np.uint8)
            want_e, want = oracle.voxel_ssb(d, dose, box_nm=15000.0)
            x = C.c_double()
            assert L.wgdna_expected_dsb_local(ctx.h, None, None, C.byref(x)) == _lib.WGDNA_ERR_STATE
            lam, e = np.zeros(2 * d.n_bp, np.float32), C.c_double()
            _lib.check("voxel", L.wgdna_score_voxel_ssb(ctx.h, _lib.ptr(dose), 15000.0, _lib.ptr(lam), C.byref(e)))
            np.testing.assert_array_equal(lam.view(np.uint32), want.view(np.uint32))
            for h in (None, hits):
                _lib.check("dsb", L.wgdna_expected_dsb_local(ctx.h, None, _lib.ptr(h) if h is not None else None, C.byref(x)))
                assert x.value == pytest.approx(oracle.expected_dsb_local(d, want, h), rel=1e-9)   # as test_dose_scoring
    finally:
        ctx.close()
