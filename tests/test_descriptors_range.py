"""Track descriptors of positions whose distances overflow or are not numbers: the distance
bins keep to their 16, a NaN in the first and an infinity in the last, and the tracks beside
them keep their values."""
import ctypes as C

import numpy as np
import pytest

import wgdna
from wgdna import _lib


class _View:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<f4", "data": (int(ptr), False), "version": 3}


@pytest.mark.gpu
@pytest.mark.parametrize("value,first", [(np.float32(1e20), 15), (np.float32(np.inf), 15), (np.float32(np.nan), 0)])
def test_bins_of_overflowing_distances(value, first):
    import torch
    L, n = _lib.lib(), 9                                 # three blocks of four tracks
    ctx = wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000)
    try:
        p = wgdna.transport_params(n, 1000.0, 15000.0, 7.5, dna=wgdna.build_dna_target(), seed=8)
        st = _lib.TransportStats()
        _lib.check("transport", L.wgdna_transport(ctx.h, C.byref(p), C.byref(st)))
        v = _lib.DeviceView()
        _lib.check("views", L.wgdna_device_views(ctx.h, C.byref(v)))
        rad = torch.as_tensor(_View(v.rad, 4 * st.rad_n_stored), device="cuda").view(-1, 4)
        pid = (rad[:, 3].cpu().numpy().astype(np.int64)) // 8
        k = C.c_uint64()
        before, after = np.zeros((n, 64), np.float32), np.zeros((n, 64), np.float32)
        _lib.check("desc", L.wgdna_track_descriptors(ctx.h, _lib.ptr(before), n, C.byref(k)))
        # every second entry of tracks 3 and 8 at `value`, the others at the origin
        for t in (3, 8):
            at = np.flatnonzero(pid == t)
            xyz = np.zeros((at.size, 3), np.float32)
            xyz[::2, 0] = value
            rad[int(at[0]):int(at[-1]) + 1, :3] = torch.from_numpy(xyz).cuda()
        torch.cuda.synchronize()
        _lib.check("desc", L.wgdna_track_descriptors(ctx.h, _lib.ptr(after), n, C.byref(k)))
        for t in range(n):
            if t not in (3, 8):
                np.testing.assert_array_equal(after[t], before[t])
                continue
            h = after[t, 9:57].reshape(3, 16)
            want = np.zeros((3, 16), np.float32)
            want[0, first] = want[1, 0] = want[2, 0] = 1  # neighbours differ; 4 and 16 apart are alike
            np.testing.assert_allclose(h, want, rtol=1e-6)
    finally:
        ctx.close()
