"""An MD run enqueues a list period behind the one whose flags it waits for.
It must end as the same steps in calls of one period each, which never have
two: the same bits in positions, velocities and energies, also where the pair
buffers overflow on the way (atoms that close in on each other) and where the
energy turns NaN (the state is then the failed period's, nothing of the next)."""
import ctypes

import numpy as np
import pytest

from conftest import build_workspace
from test_gpu_edge import _system

pytestmark = pytest.mark.gpu

EVERY = 10
STEPS = {"plain": 75, "closing": 75, "nan": 95}


def _setup(gpu_ctx, kind):
    g = 9
    grid = np.array([[i, j, k] for i in range(g) for j in range(g) for k in range(g)], dtype=np.float64)
    grid -= grid.mean(axis=0)
    pos = (5.0 if kind == "plain" else 9.5) * grid + np.random.default_rng(3).normal(0.0, 0.05, grid.shape)
    arrays, meta = _system(pos, np.arange(len(pos)) % 300)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    vel = np.zeros_like(pos)
    if kind != "plain":
        # all at the centre after 110 steps: more pairs from step 60 on than
        # the list rows have room for at first (39,088), a NaN energy after 80
        vel = -pos * 1e-10 / (110 * 1e-15)
    return ws, pos, vel


def _params(graph):
    from pdgpu import _abi as A
    p = A.md_params_default()
    p.Integrator, p.UpdateNList, p.UseGraph = A.INTEGRATOR_VELOCITY_VERLET, EVERY, graph
    p.Timestep, p.Seed = 1e-15, 3
    return p


def _run(gpu_ctx, ws, pos, vel, path, graph, steps, cut):
    """Outputs, the return codes, and the graph launches of each call."""
    from pdgpu import _abi as A
    L = A.lib()
    ws.setPairPath(path)
    A.check(L.pdgpu_set_positions(gpu_ctx.ptr, ws._sys, A.dptr(pos)))
    ws.nlist().calcNewList()
    A.check(L.pdgpu_set_velocities(gpu_ctx.ptr, ws._sys, A.dptr(vel)))
    p = _params(graph)
    h = np.zeros((steps, 3))
    rc, launches, seen = [], [], 0
    for s in range(0, steps, cut):
        rc.append(L.pdgpu_md_run(gpu_ctx.ptr, ws._sys, ctypes.byref(p), s, min(cut, steps - s), steps, A.dptr(h[s:])))
        r = np.zeros(2, dtype=np.int64)
        A.check(L.pdgpu_graph_replays(gpu_ctx.ptr, ws._sys, r.ctypes.data_as(A._I64)))
        launches.append(int(r[0]) - seen)
        seen = int(r[0])
        if rc[-1]:
            break
    x, v = np.zeros_like(pos), np.zeros_like(vel)
    A.check(L.pdgpu_get_positions(gpu_ctx.ptr, ws._sys, A.dptr(x)))
    A.check(L.pdgpu_get_velocities(gpu_ctx.ptr, ws._sys, A.dptr(v)))
    return x, v, h, rc, launches


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("kind", ["plain", "closing", "nan"])
def test_one_run_equals_single_periods(kind, path, graph, gpu_ctx):
    outs = []
    for cut in (EVERY, STEPS[kind]):
        ws, pos, vel = _setup(gpu_ctx, kind)
        outs.append(_run(gpu_ctx, ws, pos, vel, path, graph, STEPS[kind], cut))
        ws.close()
    single, whole = outs
    assert (single[3][-1] != 0) == (whole[3][-1] != 0) == (kind == "nan")
    for a, b in zip(single[:3], whole[:3]):
        np.testing.assert_array_equal(a, b)
    if graph and kind == "closing" and path == 0:
        assert max(single[4]) > 1  # a period ran again on grown list rows
