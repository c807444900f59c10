"""The tile search where its capacities end: i-clusters with more tiles than
a block stages (256), more bond-order tiles than it stages (24), more
candidate j-clusters than one list round holds, and ragged last clusters.
The tiles must hold the pairs of the list at the same positions, so every
result is the same bits as with the tiles cut from the list."""
import numpy as np
import pytest

from conftest import build_workspace
from test_gpu_edge import _system
from test_gpu_tiles import _counts, _forces_energies

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,spacing,order,special", [
    (3, 3.4, "grid", 0),        # 27 atoms: less than one i-cluster
    (4, 3.4, "grid", 6),        # 64 atoms
    (7, 3.0, "shuffled", 40),   # 343 atoms: a last j-cluster of 7
    (21, 2.2, "shuffled", 60),  # 9,261 atoms: every early i-cluster meets most of the 1,158 j-clusters
])
def test_search_capacities(side, spacing, order, special, gpu_ctx):
    rng = np.random.default_rng(side)
    g = np.arange(side)
    pos = spacing * np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    pos += rng.normal(0.0, 0.1, pos.shape)
    if order == "shuffled":
        pos = pos[rng.permutation(len(pos))]
    n = len(pos)
    arrays, meta = _system(pos, np.arange(n) % 300)
    if special:  # 1-4 partners of the first i-cluster's atoms all over the system
        far = np.linspace(33, n - 1, special).astype(int) if n > 64 else np.arange(40, 40 + special)
        partners = [[] for _ in range(n)]
        for k, j in enumerate(far):
            partners[k % 32].append(int(j))
            partners[int(j)].append(k % 32)
        arrays["cov14_ptr"] = np.cumsum([0] + [len(p) for p in partners]).astype(np.int32)
        arrays["cov14_idx"] = np.array([j for p in partners for j in sorted(p)], dtype=np.int32)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.setPairPath(0)
    ws.nlist().calcNewList()
    ws.setPairPath(1)
    listed = _forces_energies(ws, ff)
    ws.nlist().calcNewList()
    searched = _forces_energies(ws, ff)
    for a, b in zip(searched, listed):
        np.testing.assert_array_equal(a, b)  # (the dense grid's energy is NaN on both sides)
    c = _counts(ws)
    assert c[3] == c[2] // 2 and c[4] > 0
    ws.close()


def test_search_capacities_with_finite_energies(gpu_ctx):
    """The large shuffled system again at a spacing where no pair overlaps so
    far that its energy is not finite: a lost tile, or bond-order rows given to
    the wrong tile, then show in the energies too."""
    rng = np.random.default_rng(5)
    g = np.arange(21)
    pos = 3.4 * np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    pos = (pos + rng.normal(0.0, 0.1, pos.shape))[rng.permutation(21 ** 3)]
    n = len(pos)
    arrays, meta = _system(pos, np.arange(n) % 300)
    partners = [[] for _ in range(n)]
    # 60 pairs inside the cutoff, each in a tile of its own
    dist = np.linalg.norm(pos[:32, None] - pos[None], axis=2)
    near = dist.argmin(axis=0)
    close = [j for j in range(32, n) if 4.0 < dist[near[j], j] < 12.0]
    for j in {j // 8: j for j in close[::-1]}.values():
        if sum(len(p) for p in partners) < 120:
            partners[near[j]].append(int(j))
            partners[j].append(int(near[j]))
    arrays["cov14_ptr"] = np.cumsum([0] + [len(p) for p in partners]).astype(np.int32)
    arrays["cov14_idx"] = np.array([j for p in partners for j in sorted(p)], dtype=np.int32)
    ws, ff = build_workspace(arrays, meta, gpu_ctx)
    ws.setPairPath(0)
    ws.nlist().calcNewList()
    ptr, data = ws.nlist().getData(shadow=True)
    special = (np.asarray(data[:ptr[32]]) >> 24) < 7
    assert special.sum() > 24 and np.diff(ptr[:33]).sum() > 256 * 8
    ws.setPairPath(1)
    listed = _forces_energies(ws, ff)
    ws.nlist().calcNewList()
    searched = _forces_energies(ws, ff)
    for a, b in zip(searched, listed):
        assert np.all(np.isfinite(np.asarray(a)))
        np.testing.assert_array_equal(a, b)
    ws.close()
