"""Conjugate gradients at the edges of the dot products' 256-atom chunks: a
system of one chunk, of exactly one, of one atom more and of several.  Against
the oracle's minimiser: relative RMS 1e-4 of the displacements, twelve steps
along forces of relative RMS error 1e-5 (without the dot products' part of the
direction they are 7e-3 off, from 255 atoms on).  And in one batch, where the
grid is as deep as its largest member: every member's positions have the bits
it gets alone."""
import numpy as np
import pytest

from conftest import build_workspace, rel_rms
from test_gpu_edge import _system

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = (2, 255, 256, 257, 513)
STEPS, STEP_SIZE = 12, 1e7


def _grid(n):
    g = int(np.ceil(n ** (1.0 / 3.0)))
    grid = np.array([[i, j, k] for i in range(g) for j in range(g) for k in range(g)], dtype=np.float64)[:n]
    pos = 4.0 * grid + np.random.default_rng(n).normal(0.0, 0.1, (n, 3))
    return _system(pos, np.arange(n) % 300)


def _params():
    from pdgpu import _abi as A
    p = A.min_params_default()
    p.Algorithm, p.UpdateNList, p.StepSize = A.MIN_CONJUGATE_GRADIENTS, 1, STEP_SIZE
    return p


def _alone(gpu_ctx, n):
    import pdgpu
    arrays, meta = _grid(n)
    ws, _ = build_workspace(arrays, meta, gpu_ctx)
    b = pdgpu.Batch([ws])
    b.setPairPath(1)
    b.calcNewList()
    assert b.minimise(_params(), STEPS)[0] == STEPS
    pos = b.positions()
    b.close()
    ws.close()
    return pos


@pytest.mark.parametrize("n", SIZES)
def test_cg_follows_the_oracle(n, gpu_ctx):
    arrays, meta = _grid(n)
    S = O.System(arrays, cutoff=float(meta["cutoff"]), inner=float(meta["inner"]))
    taken, ref = O.minimise(S, arrays["pos"], STEPS, algorithm="cg", step_size=STEP_SIZE)[:2]
    assert taken == STEPS
    assert rel_rms(_alone(gpu_ctx, n) - arrays["pos"], ref - arrays["pos"]) <= 1e-4


def test_cg_in_a_batch_equals_alone(gpu_ctx):
    import pdgpu
    ws = [build_workspace(*_grid(n), gpu_ctx)[0] for n in SIZES]
    b = pdgpu.Batch(ws)
    b.setPairPath(1)
    b.calcNewList()
    b.minimise(_params(), STEPS)
    for x, n in zip(b.split(b.positions()), SIZES):
        np.testing.assert_array_equal(x, _alone(gpu_ctx, n))
    b.close()
    for w in ws:
        w.close()
