"""Rows of the neighbour build at the lengths where its sort changes, and the passes that give a warp several receivers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _build(positions, cell):
    from fastmace_b200.neighbours import CellListNeighbours
    x = torch.tensor(positions, dtype=torch.float64, device="cuda")
    nl = CellListNeighbours(cell, 6.0, "cuda")
    nl.build(x)
    n = nl.num_candidates
    return (nl.candidate_index[:, :n].cpu().numpy(), nl.candidate_unit_shifts[:n].cpu().numpy(), nl.cand_row_ptr.cpu().numpy())


@pytest.mark.parametrize("neighbours", [1, 31, 32, 63, 64, 65, 127, 128, 129, 300, 700])
@pytest.mark.parametrize("extra", [0, 5000])
def test_rows_of_a_cluster(neighbours, extra):
    """Everybody in the cluster sees everybody else; `extra` far atoms take the build from its one-launch form to the
    passes over large lists. The cluster sits across the cell's corner, so its pairs carry images."""
    rng = np.random.default_rng(neighbours)
    m, edge = neighbours + 1, 60.0 + 8.0 * (extra > 0) * 12
    cluster = rng.uniform(-1.5, 1.5, (m, 3))                           # diameter below 6.3 Å; partly outside the cell
    far = np.stack(np.meshgrid(*[np.arange(18)] * 3, indexing="ij"), -1).reshape(-1, 3)[:extra] * 7.0 + 10.0
    positions = np.concatenate([cluster, far])
    (sender, receiver), shifts, row_ptr = _build(positions, edge * np.eye(3))
    assert len(sender) == m * neighbours and row_ptr[len(positions)] == len(sender)
    others = np.array([[j for j in range(m) if j != i] for i in range(m)]).reshape(-1)
    assert np.array_equal(receiver, np.repeat(np.arange(m), neighbours)) and np.array_equal(sender, others)
    d = positions[receiver] - positions[sender] + shifts.astype(np.float64) * edge
    assert (np.linalg.norm(d, axis=1) < 6.3).all()


def test_large_crystal_against_a_tree():
    from scipy.spatial import cKDTree
    from fastmace_b200.structures import nacl
    s = nacl((14, 14, 14), 0.05, 3)
    assert s.natoms >= 4 * 32 * 148
    (sender, receiver), _, _ = _build(s.positions, s.cell)
    pairs = cKDTree(s.positions % s.cell[0, 0], boxsize=s.cell[0, 0]).query_pairs(6.3, output_type="ndarray")
    pairs = np.concatenate([pairs, pairs[:, ::-1]])
    pairs = pairs[np.lexsort((pairs[:, 1], pairs[:, 0]))]
    assert np.array_equal(pairs[:, 0], receiver) and np.array_equal(pairs[:, 1], sender)
