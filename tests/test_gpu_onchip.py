"""The second interaction with its last radial layer on the SM against the kernels that read the radial weights from
memory, where rows end anywhere in a tile or a range of edges, rows are empty and warps run out of edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gas(atoms, seed):
    """Clusters and single atoms far from everything, the first and the last atom among them: rows of 0 to 40 edges."""
    from fastmace_b200.structures import Structure
    rng = np.random.default_rng(seed)
    positions, side = [], 14 * int(np.ceil((atoms / 8) ** (1 / 3)) + 1)
    for corner in np.stack(np.meshgrid(*[np.arange(0, side, 14.0)] * 3, indexing="ij"), -1).reshape(-1, 3):
        count = min(int(rng.choice([1, 2, 3, 9, 20, 41])), atoms - 1 - len(positions))
        grid = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
        cells = rng.permutation(len(grid))[:count] if positions else [0]
        positions += [corner + 1.9 * grid[k] + rng.uniform(-0.3, 0.3, 3) for k in cells]
    positions = positions[:atoms - 1] + [np.array([side - 7.0] * 3)]
    assert len(positions) == atoms
    return Structure(np.array(positions), side * np.eye(3), rng.choice([11, 17], atoms))


@pytest.mark.parametrize("atoms,chunk", [(301, None), (333, None), (777, None), (777, 1 << 12)])
def test_weights_on_chip_and_streamed_agree(atoms, chunk):
    """Both routes are fp32 sums with radial weights of 22 bits and differ from float64 by up to 4e-6 of the norm."""
    from fastmace_b200.forcefield import B200ForceField
    from fastmace_b200.model import MEDIUM, init_weights
    s = _gas(atoms, atoms)
    options = {} if chunk is None else dict(chunk_edges=chunk, edge_adjoint=False)
    ff = B200ForceField(MEDIUM, init_weights(MEDIUM, 1), s.numbers, s.cell, compute_stress=True, **options)
    assert ff.packed.struct.layer[1].extra_images
    energy, forces, stress = ff.evaluate(s, stress=True)
    degree = np.bincount(ff.neighbours.edge_index[1, :int(ff.edge_count)].cpu().numpy(), minlength=atoms)
    assert degree[0] == degree[-1] == 0 and degree.max() > 16 and (degree % 2 == 1).any()
    ff.packed.struct.layer[1].extra_images = 0
    other_energy, other_forces, other_stress = ff.evaluate(s, stress=True)
    assert abs(energy - other_energy) <= 1e-6 * max(abs(other_energy), 1.0)
    assert np.linalg.norm(forces - other_forces) <= 8e-6 * np.linalg.norm(other_forces)
    assert np.linalg.norm(stress - other_stress) <= 8e-6 * np.linalg.norm(other_stress)
    assert not forces[0].any() and not forces[-1].any()
    assert (forces != other_forces).any()                            # two routes indeed
