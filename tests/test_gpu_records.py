"""Energy records at the edges of the reductions' blocks: kinetic energies of
initial velocities (256-atom chunks, four at a time) and potential energies
(4,096 items a block).  The record must be the sum of the per-atom values:
1e-12 relative, the FP64 rounding of a few thousand additions."""
import ctypes

import numpy as np
import pytest

from conftest import build_workspace
from test_gpu_edge import _system

pytestmark = pytest.mark.gpu


def _grid(n, gpu_ctx):
    g = int(np.ceil(n ** (1.0 / 3.0)))
    grid = np.array([[i, j, k] for i in range(g) for j in range(g) for k in range(g)], dtype=np.float64)[:n]
    pos = 4.4 * grid + np.random.default_rng(n).normal(0.0, 0.1, (n, 3))
    arrays, meta = _system(pos, np.arange(n) % 300)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.setPairPath(1)
    ws.nlist().calcNewList()
    return arrays, ws, ff


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1024, 1025, 9000])
def test_kinetic_record(n, gpu_ctx):
    import pdgpu
    from pdgpu import _abi as A
    arrays, ws, ff = _grid(n, gpu_ctx)
    A.check(pdgpu.lib().pdgpu_md_init_velocities(ws.ctx.ptr, ws._sys, 300.0, 7))
    ws._pull_velocities()
    ke = 0.5 * np.sum(arrays["mass"] * np.sum(ws.cur.v ** 2, axis=1))
    e = ws._pull_energies()
    assert abs(e[A.ENE_EKIN] - ke) <= 1e-12 * ke
    assert abs(ke - 1.5 * n * 1.38065e-23 * 300.0) <= 1e-12 * ke
    ws.close()


@pytest.mark.parametrize("n", [2, 511, 513, 4096, 4097, 8200])
def test_potential_record(n, gpu_ctx):
    import pdgpu
    from pdgpu import _abi as A
    arrays, ws, ff = _grid(n, gpu_ctx)
    ff.calcForces()
    ep = np.zeros(n)
    A.check(pdgpu.lib().pdgpu_get_atom_epot(ws.ctx.ptr, ws._sys, ep.ctypes.data_as(ctypes.POINTER(ctypes.c_double))))
    assert abs(ws.ene.epot - ep.sum()) <= 1e-12 * np.abs(ep).sum()
    ws.close()
