"""The streamed tensor-product kernels of a whole edge list at the edges of their dispatch: the last size whose receivers are
shared by several groups and the first that is not, receivers without edges, rows of one edge, lists shorter than a batch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("atoms", [2, 11, 296, 297])
def test_energy_forces_stress_of_a_gas_with_lone_atoms(model, atoms):
    """Bound: two interactions of fp32 sums, 1e-5 of the norm (the cells of the benchmark are off by 0.7e-6 to 2e-6)."""
    from fastmace_b200.forcefield import B200ForceField
    from fastmace_b200.model import SPECS, init_weights
    from fastmace_b200.structures import Structure
    from oracle import mace_oracle, neighbours_oracle
    spec = SPECS[model]
    weights = init_weights(spec, 3)
    rng = np.random.default_rng(atoms)
    edge = max(14.0, (atoms * 40.0) ** (1 / 3))
    positions = rng.uniform(0, edge, (atoms, 3))
    cell = np.diag([edge, edge, edge + 40.0])
    positions[atoms // 2] = [edge / 2, edge / 2, edge + 20.0]          # nobody within the cutoff
    if atoms > 4:
        positions[1:3] = [[0.0, 0.0, edge + 20.0], [2.5, 0.0, edge + 20.0 ]]       # a pair by itself: rows of one edge
    if atoms == 2:
        positions = np.array([[1.0, 1.0, 1.0], [3.0, 2.0, 1.5]])
    numbers = rng.choice([11, 17], atoms)
    s = Structure(positions, cell, numbers)
    ff = B200ForceField(spec, weights, numbers, cell, compute_stress=True)
    energy, forces, stress = ff.evaluate(s, stress=True)
    assert ff.edge_local and ff.work.chunk_edges >= ff.edge_capacity
    snd, rcv, u = neighbours_oracle.build(positions, cell, spec.r_cut, 0.0)
    assert int(ff.edge_count) == len(snd) > 0
    e, f, st = mace_oracle.evaluate(spec, weights, positions, cell, numbers, snd, rcv, u)
    assert abs(energy - float(e)) <= 1e-5 * atoms
    assert np.linalg.norm(forces - f.numpy()) <= 1e-5 * np.linalg.norm(f.numpy())
    assert np.linalg.norm(stress - st.numpy()) <= 1e-5 * np.linalg.norm(st.numpy())
    assert int(ff.status) == 0
