"""First calls of a context while the caller's default stream is busy: what they clear or
upload must not wait there, and so land after what follows on the context's own stream."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import wgdna
from wgdna import _lib

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgpu-dna_b200", "csrc")
ON_DEFAULT = re.compile(r"\bcuda(Memset|Memcpy|MemcpyToSymbol)\s*\(")


def on_default_stream(name):
    with open(os.path.join(CSRC, name)) as f:
        return [f"{name}:{k}" for k, line in enumerate(f, 1) if ON_DEFAULT.search(line.split("//")[0])]


def test_surrogate_clears_nothing_on_the_default_stream():
    assert on_default_stream("surrogate_api.cu") == []


@pytest.mark.parametrize("name", ["capi.cu", "irt.cu", "tables.cu"])
def test_context_uploads_nothing_on_the_default_stream(name):
    assert on_default_stream(name) == []


def busy_default_stream():
    """About 0.2 s of products on torch's default stream; returns its end."""
    import torch
    a = torch.zeros((8192, 8192), dtype=torch.bfloat16, device="cuda")
    b = torch.empty_like(a)
    torch.matmul(a, a, out=b)
    torch.cuda.synchronize()
    for _ in range(250):
        torch.matmul(a, a, out=b)
    end = torch.cuda.Event()
    end.record()
    return end


@pytest.mark.gpu
def test_surrogate_parameters_survive_a_busy_default_stream():
    import torch
    L = _lib.lib()
    other = wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000)
    ctx = wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000)
    try:
        # (a process's first call loads the kernels, which waits for everything)
        zero = np.zeros(_lib.SG_NPARAM, np.float32)
        _lib.check("params", L.wgdna_surrogate_params(other.h, None, _lib.ptr(zero)))
        want = np.random.default_rng(3).normal(size=_lib.SG_NPARAM).astype(np.float32)
        got = np.zeros_like(want)
        end = busy_default_stream()
        _lib.check("params", L.wgdna_surrogate_params(ctx.h, None, _lib.ptr(want)))
        assert not end.query(), "the call waited for the default stream"
        torch.cuda.synchronize()
        _lib.check("params", L.wgdna_surrogate_params(ctx.h, _lib.ptr(got), None))
        np.testing.assert_array_equal(got, want)
    finally:
        ctx.close()
        other.close()


@pytest.mark.gpu
def test_context_made_while_the_default_stream_is_busy():
    """Its first transport equals one made in quiet, and the queue of secondaries stays as
    the transport left it."""
    import torch
    out = []
    for busy in (False, True):
        if busy:
            busy_default_stream()
        ctx = wgdna.Context(max_primaries=64, max_rad=2_000_000, max_sec=200_000)
        try:
            ctx.set_tuning(stash_spill=0, stash_keep=0)          # every secondary goes through the queue
            p = wgdna.transport_params(64, 10000.0, 15000.0, 7.5, dna=wgdna.build_dna_target(), seed=4)
            st = _lib.TransportStats()
            _lib.check("transport", _lib.lib().wgdna_transport(ctx.h, C.byref(p), C.byref(st)))
            if busy:
                torch.cuda.synchronize()
            res = np.zeros(64 * 8, np.float32)
            _lib.check("copy", _lib.lib().wgdna_transport_copy_out(ctx.h, _lib.ptr(res), None, None, 0, None))
            out.append((res, int(st.rad_n_stored), np.array(st.counters)))
        finally:
            ctx.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
