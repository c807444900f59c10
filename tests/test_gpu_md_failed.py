"""What an MD run that ends in an error leaves behind.  The period behind the
failed one is enqueued already; it must change nothing, its list rebuild
included: the pair structure of the failed period stays, and a caller who puts
good positions back and evaluates without a rebuild gets what the same run in
calls of one period each gives (those never have a second period), bit for
bit.  On list rows and on tiles, in the one-block list build (up to 8,192
atoms) and the general one, on tiles cut from the list (more than 65,536
atoms), in a batch with one failing member, and with the surface term's
error, whose state is finite."""
import ctypes

import numpy as np
import pytest

from conftest import build_workspace, load_fixture, load_library
from test_gpu_edge import _system

pytestmark = pytest.mark.gpu

EVERY = 10


def _lattice(side, spacing):
    g = np.arange(side)
    pos = spacing * np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    return pos + np.random.default_rng(side).normal(0.0, 0.05, pos.shape) - pos.mean(axis=0)


def _handle(gpu_ctx, kind):
    """(handle, closers, good positions, the run's positions, velocities, steps)"""
    import pdgpu
    steps, vel = 15, None  # the period behind the first is a shorter one
    if kind == "surface":
        # closing in from 4.0 A: past 2.9 A an atom has more overlap partners than the term ranks
        pos = _lattice(9, 4.0)
        arrays, meta = _system(pos, np.arange(len(pos)) % 300)
        arrays.update(lcpo_radius=np.full(len(pos), 6.2), lcpo_use=np.ones(len(pos), np.uint8),
                      lcpo_p=np.tile([0.5, -0.3, -0.001, 0.0005], (len(pos), 1)))
        steps, vel = 45, -pos * (0.275 / 15) * 1e-10 / 1e-15
    elif kind == "list":
        pos = _lattice(41, 5.0)
        arrays, meta = _system(pos, np.arange(len(pos)) % 300)
        meta = dict(meta, cutoff="9.0", inner="7.0", vdwcut="9.0", vdwinner="7.0")
    elif kind == "general":
        arrays, meta = load_fixture("c2_16x80_s2")
    else:
        arrays, meta = load_library("lib16_opls_s4")[7]
    pos = np.ascontiguousarray(arrays["pos"])
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    close = [ws]
    bad = pos.copy()
    if kind == "surface":
        sasa = pdgpu.FF_SASA_LCPO(ws)
        sasa.GlobalASP = 0.005
        ff.add(sasa)
        ff.ensuresetup()
    elif kind == "list":
        bad[1] = bad[0]  # two atoms at one point: on tiles a NaN energy
    else:
        bad[10] = np.nan  # an atom with bonds: a NaN energy
    if kind == "batch":
        more = load_library("lib16_opls_s4")[15]
        close.append(build_workspace(*more, gpu_ctx)[0])
        close.insert(0, pdgpu.Batch(close[:]))
        pos, bad = (np.concatenate([x, more[0]["pos"]]) for x in (pos, bad))
    return close[0], close, pos, bad, np.zeros_like(pos) if vel is None else vel, steps


def _state(L, c, s, n):
    """Forces, energies and per-atom energies of the handle as they are."""
    from pdgpu import _abi as A
    f, ep = np.zeros((n, 3)), np.zeros(n)
    A.check(L.pdgpu_get_forces(c, s, A.dptr(f)))
    e = np.zeros(2 * A.ENE_COUNT)
    A.check(L.pdgpu_get_energies(c, s, A.dptr(e), e.size))
    A.check(L.pdgpu_get_atom_epot(c, s, A.dptr(ep)))
    e = e.reshape(2, -1)
    e[:, [A.ENE_EKIN, A.ENE_ETOT]] = 0.0  # the run's last kinetic energies, no part of an evaluation
    return f, e, ep


def _failed_run(gpu_ctx, kind, path, graph, cut):
    """Runs to the error in calls of `cut` steps.  (error, steps asked for
    until then, the state as the run left it, the state of an evaluation from
    good positions, the tile counts, the exported list)"""
    from pdgpu import _abi as A
    L = A.lib()
    h, close, good, x, v, steps = _handle(gpu_ctx, kind)
    cut = cut or steps
    c, s, n = gpu_ctx.ptr, h._device() if hasattr(h, "_device") else h._id, len(good)
    assert h.setPairPath(path) == path
    A.check(L.pdgpu_set_positions(c, s, A.dptr(good)))
    A.check(L.pdgpu_nlist_build(c, s))
    A.check(L.pdgpu_set_positions(c, s, A.dptr(x)))
    A.check(L.pdgpu_set_velocities(c, s, A.dptr(np.ascontiguousarray(v))))
    p = A.md_params_default()
    p.Integrator, p.UpdateNList, p.UseGraph = A.INTEGRATOR_VELOCITY_VERLET, EVERY, graph
    p.Timestep, p.Seed = 1e-15, 3
    for at in range(0, steps, cut):
        rc = L.pdgpu_md_run(c, s, ctypes.byref(p), at, min(cut, steps - at), steps, None)
        if rc:
            break
    left = _state(L, c, s, n)
    A.check(L.pdgpu_set_positions(c, s, A.dptr(good)))
    A.check(L.pdgpu_set_step(c, s, 0))  # (a call that succeeds leaves its last step there)
    A.check(L.pdgpu_calc_forces(c, s))
    again = _state(L, c, s, n)
    counts = np.zeros(5, dtype=np.int64)
    A.check(L.pdgpu_pair_counts(c, s, counts.ctypes.data_as(A._I64)))
    ptr, count = np.zeros(n + 1, np.int32), ctypes.c_int64(0)
    L.pdgpu_nlist_export(c, s, 1, A.iptr(ptr), None, 0, ctypes.byref(count))
    data = np.zeros(count.value, np.int32)
    A.check(L.pdgpu_nlist_export(c, s, 1, A.iptr(ptr), A.iptr(data), count.value, ctypes.byref(count)))
    for q in close:
        q.close()
    return rc, at, left, again, counts, (ptr, data)


CASES = [(k, path, 1) for k in ("small", "general", "batch", "surface") for path in (0, 1)]
CASES += [("small", 0, 0), ("small", 1, 0), ("list", 1, 1)]


@pytest.mark.parametrize("kind,path,graph", CASES)
def test_pairs_after_a_failed_run(kind, path, graph, gpu_ctx):
    single = _failed_run(gpu_ctx, kind, path, graph, EVERY)
    whole = _failed_run(gpu_ctx, kind, path, graph, None)
    assert single[0] == whole[0] != 0 and single[1] == (20 if kind == "surface" else 0)
    assert np.all(np.isfinite(single[3][0])) and np.abs(single[3][0]).max() > 0
    for a, b in zip(single[3] + single[5] + (single[4],), whole[3] + whole[5] + (whole[4],)):
        np.testing.assert_array_equal(a, b)
    assert single[4][4] > 0 if path else single[5][0][-1] > 0


# (past its ranks' limit the surface term keeps whichever candidates came first)
@pytest.mark.parametrize("kind,path,graph", [c for c in CASES if c[:2] != ("surface", 1)])
def test_forces_after_a_failed_run(kind, path, graph, gpu_ctx):
    single = _failed_run(gpu_ctx, kind, path, graph, EVERY)
    whole = _failed_run(gpu_ctx, kind, path, graph, None)
    assert np.abs(np.nan_to_num(single[2][0])).max() > 0
    for a, b in zip(single[2][:2], whole[2][:2]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind,path,graph", [c for c in CASES if c[0] != "surface"])
def test_atom_energies_after_a_failed_run(kind, path, graph, gpu_ctx):
    """Odd and even steps keep them in two buffers: the failed period's last
    step decides, not that of the period behind."""
    single = _failed_run(gpu_ctx, kind, path, graph, EVERY)
    whole = _failed_run(gpu_ctx, kind, path, graph, None)
    assert np.abs(np.nan_to_num(single[2][2])).max() > 0
    np.testing.assert_array_equal(single[2][2], whole[2][2])


def _peptide(gpu_ctx, path):
    arrays, meta = load_library("lib16_opls_s4")[7]
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    assert ws.setPairPath(path) == path
    return ws, ff, np.ascontiguousarray(arrays["pos"])


def _md(gpu_ctx, ws, first, steps, graph=1):
    from pdgpu import _abi as A
    p = A.md_params_default()
    p.Integrator, p.UpdateNList, p.UseGraph = A.INTEGRATOR_VELOCITY_VERLET, EVERY, graph
    p.Timestep, p.Seed = 1e-15, 3
    return A.lib().pdgpu_md_run(gpu_ctx.ptr, ws._sys, ctypes.byref(p), first, steps, 100, None)


@pytest.mark.parametrize("path", [0, 1])
def test_list_of_a_run_that_failed_inside_a_period(path, gpu_ctx):
    """The run starts inside a period on a list made for it (no tile search at
    these positions) and fails there; the period behind would have searched."""
    from pdgpu import _abi as A
    lists = []
    for steps in (5, 25):
        ws, ff, pos = _peptide(gpu_ctx, path)
        ws.nlist().calcNewList()
        assert _md(gpu_ctx, ws, 0, 5) == 0
        moved = 1.05 * pos
        bad = moved.copy()
        bad[10] = np.nan
        A.check(A.lib().pdgpu_set_positions(gpu_ctx.ptr, ws._sys, A.dptr(bad)))
        A.check(A.lib().pdgpu_system_set_params(gpu_ctx.ptr, ws._sys, ctypes.byref(ff._nb()._params())))
        assert _md(gpu_ctx, ws, 5, steps) != 0
        A.check(A.lib().pdgpu_set_positions(gpu_ctx.ptr, ws._sys, A.dptr(moved)))
        lists.append(ws.nlist().getData(shadow=True))
        ws.close()
    for a, b in zip(*lists):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("steps", [10, 5])
def test_atom_energies_after_a_replayed_period(steps, gpu_ctx):
    """A period replayed from its graph, with a single evaluation before it."""
    from pdgpu import _abi as A
    out = []
    for graph in (1, 0):
        ws, ff, pos = _peptide(gpu_ctx, 1)
        ws.nlist().calcNewList()
        for k in range(2):
            assert _md(gpu_ctx, ws, 10 * k, steps, graph) == 0
            if steps < EVERY:  # the rest of the period, so the next call begins one
                assert _md(gpu_ctx, ws, 10 * k + steps, EVERY - steps - 1, graph) == 0
                assert _md(gpu_ctx, ws, 10 * k + EVERY - 1, 1, graph) == 0
            if k == 0:
                A.check(A.lib().pdgpu_calc_forces(gpu_ctx.ptr, ws._sys))
        if steps < EVERY:
            assert _md(gpu_ctx, ws, 20, steps, graph) == 0
        out.append(_state(A.lib(), gpu_ctx.ptr, ws._sys, len(pos))[2])
        ws.close()
    np.testing.assert_array_equal(*out)
