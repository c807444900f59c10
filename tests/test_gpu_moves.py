"""Trial moves around the chunk of rotations the prefix kernel forms at a
time (32): fewer, exactly as many, one more and two chunks, on one chain and
on two (a nest that begins inside a chunk), against the oracle's rotations
one after another (1e-9 A, the bound of the existing trial-move test)."""
import numpy as np
import pytest

from conftest import build_workspace, load_fixture

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,nrot", [("c1_pep64_s0", 1), ("c1_pep64_s0", 31), ("c1_pep64_s0", 32),
                                       ("c1_pep64_s0", 33), ("c1_pep64_s0", 64), ("two_chain_s4", None)])
def test_torsion_prefix_chunks(name, nrot, gpu_ctx):
    arrays, meta = load_fixture(name)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    axes = ws.backboneAxes()[:nrot]
    assert ws.setTorsionMoves(axes) == len(axes)
    ws.saveBasePositions()
    angles = np.random.default_rng(len(axes)).normal(0.0, np.radians(15.0), len(axes))
    ws.perturbTorsions(angles=angles)
    ref = O.apply_torsions(arrays["pos"], arrays["cov12_ptr"], arrays["cov12_idx"], axes, angles)
    assert np.abs(ws.cur.p - ref).max() <= 1e-9
    ws.close()
