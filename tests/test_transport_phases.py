"""The transport kernel's phases where a run of steps is cut short and where a block
goes from many electrons to few: step caps inside a run of elastic steps, starts
off the origin, small boxes, one primary, and more primaries than a block's
share; bit for bit against the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle
import wgdna
from wgdna import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E,kw", [
    (1, 10000.0, {}),
    (3, 30.0, {}),
    (300, 2000.0, {"max_steps": 7, "sec_steps": 5}),
    (300, 2000.0, {"max_steps": 1, "sec_steps": 1}),
    (257, 500.0, {"start_half": 120.0, "box": 150.0}),          # some start next to the box
    (512, 3000.0, {"start_half": 5.0, "box": 40.0, "sec_steps": 33}),
    (1500, 400.0, {"ce": 7.4}),
])
def test_transport_run_ends(ctx, n, E, kw):
    box, ce = kw.get("box", 15000.0), kw.get("ce", 7.5)
    p = wgdna.transport_params(n, E, box, ce, seed=n + 7, dna_enable=0)
    p.max_steps, p.sec_steps = kw.get("max_steps", p.max_steps), kw.get("sec_steps", p.sec_steps)
    p.start_half = kw.get("start_half", 0.0)
    st, L = _lib.TransportStats(), _lib.lib()
    _lib.check("wgdna_transport", L.wgdna_transport(ctx.h, C.byref(p), C.byref(st)))
    res, k = np.zeros(8 * n, np.float32), C.c_uint64()
    dose, rad = np.zeros(ctx.vc ** 3, np.uint32), np.zeros((st.rad_n_stored, 4), np.float32)
    _lib.check("copy_out", L.wgdna_transport_copy_out(ctx.h, _lib.ptr(res), _lib.ptr(dose), _lib.ptr(rad),
                                                      st.rad_n_stored, C.byref(k)))
    o = oracle.transport(n, E, seed=n + 7, rng_mode=0, dna_enable=0, box_nm=box, ce_eV=ce, start_half=p.start_half,
                         max_steps=p.max_steps, sec_steps=p.sec_steps)
    np.testing.assert_array_equal(res.view(np.uint32), o["results"].view(np.uint32))
    np.testing.assert_array_equal(np.array(st.counters[:7]), o["counters"][:7])
    np.testing.assert_array_equal(np.array(st.sec_stats[:]), o["sec_stats"])
    np.testing.assert_array_equal(rad.view(np.uint32), o["rad"].view(np.uint32))
    np.testing.assert_array_equal(dose, o["dose"])
    assert st.steps == o["steps"]
