"""Forces, positions and velocities of a batch too large for the context's
page-locked block (10,922 atoms), read when no device memory is left for a
staging array: they come in pieces, the same values.  (Positions that come in
do need the array: refused, and the calls after that work.)"""
import ctypes

import numpy as np
import pytest

from conftest import build_workspace, load_library

pytestmark = pytest.mark.gpu


class _Full:
    """Takes all memory the device's default pool can give."""

    def __enter__(self):
        self.cu, self.held = ctypes.CDLL("libcuda.so.1"), []
        for shift in range(32, 15, -1):
            p = ctypes.c_uint64(0)
            while self.cu.cuMemAllocAsync(ctypes.byref(p), ctypes.c_size_t(1 << shift), None) == 0:
                self.held.append(p.value)
        assert self.cu.cuStreamSynchronize(None) == 0

    def __exit__(self, *exc):
        for p in self.held:
            self.cu.cuMemFreeAsync(ctypes.c_uint64(p), None)
        assert self.cu.cuStreamSynchronize(None) == 0
        dev, pool = ctypes.c_int(0), ctypes.c_void_p()  # and out of the pool, which keeps what it has
        assert self.cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), dev) == 0
        assert self.cu.cuMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0


def test_state_out_without_staging_memory(gpu_ctx):
    import pdgpu
    from pdgpu import _abi as A
    ws = [build_workspace(a, m, gpu_ctx)[0] for a, m in load_library("lib16_opls_s4")[:9]]
    got = []
    for full in (False, True):
        b = pdgpu.Batch(ws)
        assert b.nAtoms > 10922
        b.setPairPath(1)
        b.calcNewList()
        b.calcForces()
        A.check(A.lib().pdgpu_md_init_velocities(gpu_ctx.ptr, b._id, 300.0, 3))
        f, x, v = (np.zeros((b.nAtoms, 3)) for _ in range(3))
        read = (("pdgpu_get_forces", f), ("pdgpu_get_positions", x), ("pdgpu_get_velocities", v))
        if full:
            with _Full():
                for name, to in read:
                    A.check(getattr(A.lib(), name)(gpu_ctx.ptr, b._id, A.dptr(to)))
                assert A.lib().pdgpu_set_positions(gpu_ctx.ptr, b._id, A.dptr(x)) == A.ERR_NOMEM
                assert A.lib().pdgpu_calc_forces(gpu_ctx.ptr, b._id) == 0
        else:
            for name, to in read:
                A.check(getattr(A.lib(), name)(gpu_ctx.ptr, b._id, A.dptr(to)))
        got.append((f, x, v))
        b.close()
    for w in ws:
        w.close()
    for a, c in zip(*got):
        assert np.abs(a).max() > 0
        np.testing.assert_array_equal(a, c)
