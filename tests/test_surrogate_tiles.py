"""The surrogate's kernel at the edges of its 128-row tiles and where a CTA takes
several of them (more than 148 tiles), against the numpy reference."""
import ctypes as C

import numpy as np
import pytest

from oracle import surrogate_ref as ref
from wgdna import _lib


IDENTITY = np.concatenate([np.zeros(64), np.ones(64), np.zeros(80), np.ones(80)]).astype(np.float32)


def _model(ctx, seed):
    L = _lib.lib()
    _lib.check("init", L.wgdna_surrogate_init(ctx.h, seed))
    p = ref.init(seed)
    g = np.random.default_rng(seed + 1)
    for (w0, b0), (n_out, _) in zip(ref.OFFS, ref.SHAPES):
        p[b0:b0 + n_out] = g.normal(0, 0.2, n_out)
    _lib.check("params", L.wgdna_surrogate_params(ctx.h, None, _lib.ptr(p)))
    _lib.check("norm", L.wgdna_surrogate_norm(ctx.h, None, _lib.ptr(IDENTITY)))
    return L, p, g


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 148 * 128 + 1])
def test_gradient_at_tile_edges(ctx, n):
    """Per layer within 2e-2 of the reference's norm: both round weights, layer inputs
    and output gradients to bf16 (2^-9 relative each) at the same points."""
    L, p, g = _model(ctx, n % 97 + 1)
    X = g.normal(size=(n, ref.IN)).astype(np.float32)
    T = g.normal(size=(n, ref.OUT)).astype(np.float32)
    _lib.check("load", L.wgdna_surrogate_load(ctx.h, _lib.ptr(X), _lib.ptr(T), n))
    got = np.zeros(ref.NPARAM, np.float32)
    loss = C.c_double()
    _lib.check("grad", L.wgdna_surrogate_grad(ctx.h, n, _lib.ptr(got), C.byref(loss)))
    want_loss, want = ref.loss_and_grad(p, X, T)
    assert abs(loss.value - want_loss) <= 1e-4 * want_loss
    for (w0, b0), (n_out, n_in) in zip(ref.OFFS, ref.SHAPES):
        for a, b in ((w0, w0 + n_out * n_in), (b0, b0 + n_out)):
            assert np.linalg.norm(got[a:b] - want[a:b]) <= 2e-2 * np.linalg.norm(want[a:b]), (n, a)
    # the sum over CTAs has one order: a second call gives the same bits
    again = np.zeros(ref.NPARAM, np.float32)
    _lib.check("grad", L.wgdna_surrogate_grad(ctx.h, n, _lib.ptr(again), None))
    np.testing.assert_array_equal(again, got)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 128, 129, 300])
def test_prediction_is_standardised_and_back(ctx, n):
    """1e-2 of the largest output, as test_forward_matches_reference (bf16 layer inputs)."""
    L, p, g = _model(ctx, 5)
    norm = np.concatenate([g.normal(size=64), g.uniform(0.5, 2, 64), g.normal(size=80), g.uniform(0.5, 2, 80)]).astype(np.float32)
    _lib.check("norm", L.wgdna_surrogate_norm(ctx.h, None, _lib.ptr(norm)))
    z = g.normal(size=(n, ref.IN))
    X = (norm[:64] + norm[64:128] * z).astype(np.float32)
    G = np.zeros((n, ref.OUT), np.float32)
    _lib.check("predict", L.wgdna_surrogate_predict(ctx.h, _lib.ptr(X), n, _lib.ptr(G)))
    _lib.check("norm", L.wgdna_surrogate_norm(ctx.h, None, _lib.ptr(IDENTITY)))       # the context is shared
    Y, _ = ref.forward(p, ((X - norm[:64]) / norm[64:128]).astype(np.float32))
    Y = Y * norm[208:] + norm[128:208]
    assert np.abs(G - Y).max() <= 1e-2 * np.abs(Y).max()
