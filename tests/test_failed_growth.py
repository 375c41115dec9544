"""A call that asks for more memory than there is fails, and the next one of an ordinary
size gives what it gave before (the requests are of terabytes, so nothing is taken)."""
import ctypes as C

import numpy as np
import pytest

import oracle
import wgdna
from oracle import surrogate_ref as ref
from wgdna import _lib


@pytest.fixture()
def small():
    c = wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000)
    yield c
    c.close()


@pytest.mark.gpu
def test_grid_chemistry(small):
    rad = np.zeros((300, 4), np.float32)
    rad[:, 0] = 2500.0 * np.arange(300) - 375_000.0          # no two ever meet
    want, _, _ = oracle.chem_grid(rad, seed=3)
    L = _lib.lib()
    r = _lib.ChemGridResult()
    for n in (300, 1 << 36, 299, 300):
        got = L.wgdna_chem_grid(small.h, _lib.ptr(rad), n, 16, 1000.0, 3, C.byref(r), None, None, 0)
        assert got == (_lib.WGDNA_ERR_NOMEM if n > 300 else _lib.WGDNA_OK)
        if n == 300:
            np.testing.assert_array_equal(np.array(r.counts), want)


@pytest.mark.gpu
def test_surrogate(small):
    L = _lib.lib()
    g = np.random.default_rng(1)
    X = g.normal(size=(200, ref.IN)).astype(np.float32)
    T = g.normal(size=(200, ref.OUT)).astype(np.float32)
    _lib.check("init", L.wgdna_surrogate_init(small.h, 5))
    p = ref.init(5)
    _lib.check("params", L.wgdna_surrogate_params(small.h, None, _lib.ptr(p)))
    out = []
    for n in (200, 1 << 33, 199, 200):
        G = np.zeros((200, ref.OUT), np.float32)
        got = L.wgdna_surrogate_predict(small.h, _lib.ptr(X), n, _lib.ptr(G))
        assert got == (_lib.WGDNA_ERR_NOMEM if n > 200 else _lib.WGDNA_OK)
        if n == 200:
            out.append(G)
    np.testing.assert_array_equal(out[0], out[1])
    _lib.check("load", L.wgdna_surrogate_load(small.h, _lib.ptr(X), _lib.ptr(T), 200))
    assert L.wgdna_surrogate_load(small.h, _lib.ptr(X), _lib.ptr(T), 1 << 33) == _lib.WGDNA_ERR_NOMEM
    loss = C.c_double()
    assert L.wgdna_surrogate_grad(small.h, 200, None, C.byref(loss)) == _lib.WGDNA_ERR_ARG      # no data now
    _lib.check("load", L.wgdna_surrogate_load(small.h, _lib.ptr(X), _lib.ptr(T), 200))
    _lib.check("grad", L.wgdna_surrogate_grad(small.h, 200, None, C.byref(loss)))
    want, _ = ref.loss_and_grad(p, X, T)
    assert abs(loss.value - want) <= 1e-4 * want             # as test_gradient_at_tile_edges
