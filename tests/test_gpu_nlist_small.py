"""The list rebuild of one small system (boxes, keys and sort in one block,
row starts added up by the fill) against the general chain, which a pack's
first build always runs: the same rows in the same order.  The row passes add
in row order, so their forces and energies must be the same bits, and the
exported list the same.  Sizes around the warps' segments, the block and the
limit of the small path; grids of one cell, of many, and with more cells than
the table holds for 32 warps; a NaN and an infinite coordinate."""
import numpy as np
import pytest

from conftest import build_workspace
from test_gpu_edge import _system

pytestmark = pytest.mark.gpu


def _positions(n, kind):
    rng = np.random.default_rng(n)
    g = int(np.ceil(n ** (1.0 / 3.0)))
    cube = 3.6 * np.array([[i, j, k] for i in range(g) for j in range(g) for k in range(g)], dtype=np.float64)[:n]
    cube += rng.normal(0.0, 0.1, cube.shape)
    if kind == "chain":       # a long thin box
        return np.stack([3.0 * np.arange(n), rng.normal(0, 2, n), rng.normal(0, 2, n)], 1)
    if kind == "sparse":      # more cells than atoms: the grid is clamped
        return rng.uniform(-3000.0, 3000.0, (n, 3))
    if kind == "nan":
        cube[n // 2, 1] = np.nan
    if kind == "inf":
        cube[n // 3, 2] = np.inf
    return cube[rng.permutation(n)] if kind == "shuffled" else cube


CASES = [(1, "cube"), (2, "cube"), (31, "cube"), (33, "shuffled"), (64, "nan"), (97, "inf"), (1000, "sparse"),
         (1023, "cube"), (1025, "shuffled"), (2600, "chain"), (4097, "shuffled"), (8192, "sparse"),
         (8192, "shuffled"), (8193, "cube")]


@pytest.mark.parametrize("n,kind", CASES)
def test_small_rebuild_equals_general(n, kind, gpu_ctx):
    arrays, meta = _system(_positions(n, kind), np.arange(n) % 300)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.setLanes((8, 8, 8))
    got = []
    for _ in range(3):  # the first build is the general chain, the others the small path
        ws.nlist().calcNewList()
        ff.calcForces()
        f, e = ws.cur.f.copy(), ws._pull_energies()
        ff.calcEnergies()
        got.append((f, e, ws.cur.f.copy(), ws._pull_energies()) + ws.nlist().getData(shadow=True))
    for g in got[1:]:
        for a, b in zip(g, got[0]):
            np.testing.assert_array_equal(a, b)
    ws.close()


def test_small_rebuild_that_outgrows_the_buffer(gpu_ctx):
    """Atoms far apart, then close together: the second list needs far more
    entries than the first sized the buffer for."""
    n = 3000
    spread, dense = _positions(n, "sparse"), _positions(n, "cube")
    arrays, meta = _system(spread, np.arange(n) % 300)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.setLanes((8, 8, 8))
    ws.nlist().calcNewList()
    assert len(ws.nlist().getData(shadow=True)[1]) < n
    ws.cur.p[:] = dense
    ws._push_positions()
    ws.nlist().calcNewList()
    got = ws.nlist().getData(shadow=True)
    arrays2, _ = _system(dense, np.arange(n) % 300)
    ws2, ff2 = build_workspace(arrays2, meta, gpu_ctx)
    ws2.setLanes((8, 8, 8))
    ws2.nlist().calcNewList()
    ref = ws2.nlist().getData(shadow=True)
    assert len(ref[1]) > 48 * n + 4096
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
    ws.close()
    ws2.close()
