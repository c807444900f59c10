"""Kinetic energies of initial velocities around a block of the kernel that
adds them (4,096 atoms) and over several: the record is the sum of the atoms'
(1e-12 relative, the FP64 rounding of some thousand additions), and a system
gets the same bits alone and in a batch whose largest member has more blocks."""
import numpy as np
import pytest

from conftest import build_workspace
from test_gpu_edge import _system

pytestmark = pytest.mark.gpu

SIZES = (1, 300, 4095, 4096, 4097, 8192, 8193, 40000)


def _workspace(n, gpu_ctx):
    g = int(np.ceil(n ** (1.0 / 3.0)))
    grid = np.array([[i, j, k] for i in range(g) for j in range(g) for k in range(g)], dtype=np.float64)[:n]
    arrays, meta = _system(4.4 * grid, np.arange(n) % 300)
    return build_workspace(arrays, meta, gpu_ctx)[0], arrays["mass"]


def _init(b, n_sys):
    from pdgpu import _abi as A
    b.setSeeds(np.full(n_sys, 7, dtype=np.uint64))
    A.check(A.lib().pdgpu_md_init_velocities(b.ctx.ptr, b._id, 300.0, 7))
    return b.velocities(), b.energies()[:, A.ENE_EKIN]


def test_kinetic_records_alone_and_in_a_batch(gpu_ctx):
    import pdgpu
    made = [_workspace(n, gpu_ctx) for n in SIZES]
    whole = pdgpu.Batch([ws for ws, _ in made])
    v, e = _init(whole, len(SIZES))
    for s, (ws, mass) in enumerate(made):
        b = pdgpu.Batch([ws])
        v1, e1 = _init(b, 1)
        ke = 0.5 * np.sum(mass * np.sum(v1 ** 2, axis=1))
        assert abs(e1[0] - ke) <= 1e-12 * ke
        assert abs(ke - 1.5 * SIZES[s] * 1.38065e-23 * 300.0) <= 1e-12 * ke
        assert e1[0] == e[s]
        np.testing.assert_array_equal(v1, whole.split(v)[s])
        b.close()
    whole.close()
    for ws, _ in made:
        ws.close()
