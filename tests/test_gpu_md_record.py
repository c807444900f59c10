"""MD with the bonded terms and the previous step's energy record behind the
first phase of the evaluation (packs of at most 4,096 atoms, three launches)
and from the start of the step (larger packs, or the evaluation in one
launch): the same kernels on the same inputs, so positions, velocities and
every step's energies have the same bits.  Blocks of one, two and more steps,
as graphs and as plain launches."""
import ctypes

import numpy as np
import pytest

from conftest import build_workspace, load_library

pytestmark = pytest.mark.gpu


def _run(gpu_ctx, b, p, x0, v0, steps):
    from pdgpu import _abi as A
    L = A.lib()
    sid = b._id
    A.check(L.pdgpu_set_positions(gpu_ctx.ptr, sid, A.dptr(x0)))
    A.check(L.pdgpu_set_velocities(gpu_ctx.ptr, sid, A.dptr(v0)))
    nsys = len(b.split(x0))
    h = np.zeros((steps, nsys, 3))
    A.check(L.pdgpu_md_run(gpu_ctx.ptr, sid, ctypes.byref(p), 0, steps, steps, A.dptr(h)))
    x, v = np.zeros_like(x0), np.zeros_like(v0)
    A.check(L.pdgpu_get_positions(gpu_ctx.ptr, sid, A.dptr(x)))
    A.check(L.pdgpu_get_velocities(gpu_ctx.ptr, sid, A.dptr(v)))
    return x, v, h


@pytest.mark.parametrize("members", [1, 2, 8])
@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("steps,every", [(1, 10), (2, 1), (5, 2), (7, 10)])
def test_record_beside_next_step(members, graph, steps, every, gpu_ctx):
    import pdgpu
    from pdgpu import _abi as A
    lib = load_library("lib16_opls_s4")
    ws = [build_workspace(a, m, gpu_ctx)[0] for a, m in (lib * 2)[:members]]
    b = pdgpu.Batch(ws)
    b.setPairPath(1)
    n = sum(w.nAtoms() for w in ws)
    assert (n > 4096) == (members > 1)
    p = A.md_params_default()
    p.Integrator, p.UpdateNList, p.UseGraph = A.INTEGRATOR_LANGEVIN, every, graph
    p.Timestep, p.FricCoeff, p.TargetTemp, p.Seed = 1e-15, 1e12, 300.0, 3
    A.check(A.lib().pdgpu_md_init_velocities(gpu_ctx.ptr, b._id, 300.0, 3))
    x0, v0 = np.zeros((n, 3)), np.zeros((n, 3))
    A.check(A.lib().pdgpu_get_positions(gpu_ctx.ptr, b._id, A.dptr(x0)))
    A.check(A.lib().pdgpu_get_velocities(gpu_ctx.ptr, b._id, A.dptr(v0)))
    assert b.setEvalMode(1) == 1
    one = _run(gpu_ctx, b, p, x0, v0, steps)
    assert b.setEvalMode(0) == 0
    three = _run(gpu_ctx, b, p, x0, v0, steps)
    for u, w in zip(one, three):
        assert np.all(np.isfinite(u))
        assert np.array_equal(u, w)
    b.close()
