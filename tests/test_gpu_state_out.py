"""Forces as the caller gets them: the device forms [n][3] in N from the
accumulators.  Sizes on both sides of a block of the kernel (3 n components,
256 a block), against the oracle's FP64 forces at the same coordinates
(relative RMS 1e-5, the pair arithmetic's bound)."""
import numpy as np
import pytest

from conftest import build_workspace, rel_rms
from test_gpu_edge import _system

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 85, 86, 171, 342])
def test_forces_out_at_block_edges(n, gpu_ctx):
    g = int(np.ceil(n ** (1.0 / 3.0)))
    grid = np.array([[i, j, k] for i in range(g) for j in range(g) for k in range(g)], dtype=np.float64)[:n]
    pos = 4.2 * grid + np.random.default_rng(n).normal(0.0, 0.2, (n, 3))
    arrays, meta = _system(pos, np.arange(n) % 300)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.setPairPath(1)
    ws.nlist().calcNewList()
    ff.calcForces()
    S = O.System(arrays, cutoff=float(meta["cutoff"]), inner=float(meta["inner"]))
    f_ref, _, _ = S.calc_forces(pos, *S.nlist(pos))
    assert rel_rms(ws.cur.f, f_ref) <= 1e-5
    ws.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 10922, 10923])
def test_state_through_the_block_and_past_it(n, gpu_ctx):
    """Positions and velocities in and out around a block of the kernels and
    around the size the page-locked block holds (256 KB: 10,922 atoms): the
    same bits come back, one array at a time and through pdgpu_md_run_io with
    no step to run."""
    import ctypes

    import pdgpu
    from pdgpu import _abi as A
    rng = np.random.default_rng(n)
    x, v = rng.normal(0.0, 200.0, (n, 3)), rng.normal(0.0, 400.0, (n, 3))
    arrays, meta = _system(x, np.arange(n) % 300)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.cur.p[:], ws.cur.v[:] = x, v
    ws._push_positions()
    ws._push_velocities()
    ws.cur.p[:], ws.cur.v[:] = 0.0, 0.0
    ws._pull_positions()
    ws._pull_velocities()
    assert np.array_equal(ws.cur.p, x) and np.array_equal(ws.cur.v, v)
    xo, vo = np.zeros((n, 3)), np.zeros((n, 3))
    p = pdgpu.md_params_default()
    A.check(pdgpu.lib().pdgpu_md_run_io(ws.ctx.ptr, ws._sys, ctypes.byref(p), 0, 0, 0, A.dptr(v), A.dptr(x),
                                        A.dptr(xo), A.dptr(vo), None))
    assert np.array_equal(xo, v) and np.array_equal(vo, x)
    ws.close()
