"""Lists evaluated in chunks: rows that straddle chunk boundaries or have no edges, chunks behind the last edge, the sender
gradients of one chunk at a time, and the kernels that remain where not even those fit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(model, atoms=150):
    from fastmace_b200.model import SPECS, init_weights
    spec = SPECS[model]
    rng = np.random.default_rng(5)
    edge = (atoms * 50.0) ** (1 / 3)
    cell = np.diag([edge, edge, edge + 30.0])
    positions = rng.uniform(0, edge, (atoms, 3))
    positions[[0, 70, atoms - 1], :] = [[1, 1, edge + 15.0], [1, 9, edge + 15.0], [9, 1, edge + 15.0]]     # rows without edges
    numbers = rng.choice([11, 17], atoms)
    return spec, init_weights(spec, 4), torch.tensor(positions, device="cuda"), numbers, cell


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("chunk", [37, 256, 1000])
@pytest.mark.parametrize("edge_adjoint", [None, False])
def test_chunks_give_what_the_whole_list_gives(model, chunk, edge_adjoint):
    """Bound: the same fp32 terms summed in another order, 1e-5 of the norm."""
    from fastmace_b200.forcefield import B200ForceField
    spec, weights, x, numbers, cell = _case(model)
    whole = B200ForceField(spec, weights, numbers, cell, positions=x, compute_stress=True)(x)
    ff = B200ForceField(spec, weights, numbers, cell, positions=x, compute_stress=True, chunk_edges=chunk, edge_adjoint=edge_adjoint)
    assert ff.edge_local == (edge_adjoint is None) and int(ff.work.dx_edges) == (0 if edge_adjoint is None else chunk)
    for _ in range(2):                                    # the second call finds the first one's buffers
        out = ff(x)
        for a, b in zip(out, whole):
            assert (a.double() - b.double()).norm() <= 1e-5 * b.double().norm()
    ff.check_status()


@pytest.mark.parametrize("model", ["small", "medium", "large"])
def test_evaluation_from_both_ends_without_hand_over_buffers(model):
    from fastmace_b200.forcefield import B200ForceField
    spec, weights, x, numbers, cell = _case(model)
    whole = B200ForceField(spec, weights, numbers, cell, positions=x, compute_stress=True)(x)
    ff = B200ForceField(spec, weights, numbers, cell, positions=x, compute_stress=True, chunk_edges=1000, edge_adjoint=False)
    ff.work.mirror, ff.work.edge_q, ff.work.edge_dx = None, None, None
    for a, b in zip(ff(x), whole):
        assert (a.double() - b.double()).norm() <= 1e-5 * b.double().norm()
    ff.check_status()


@pytest.mark.parametrize("model", ["small", "medium", "large"])
@pytest.mark.parametrize("chunk", [37, 200, 1000, 4096])
@pytest.mark.parametrize("n_owned,n_inner", [(-1, -1), (40, 91)])
def test_sender_gradients_of_one_chunk_at_a_time_are_the_bits_of_the_whole_list(model, chunk, n_owned, n_inner):
    """A row's terms come in the same order whether they are collected behind each chunk or at the end; with an inner halo
    the rows behind it hand over nothing."""
    from fastmace_b200.forcefield import B200ForceField
    spec, weights, x, numbers, cell = _case(model)
    outputs = []
    for edge_adjoint in (None, False):
        ff = B200ForceField(spec, weights, numbers, cell, positions=x, compute_stress=True, chunk_edges=chunk,
                            edge_adjoint=edge_adjoint, n_owned=n_owned, n_inner=n_inner)
        assert int(ff.work.dx_edges) == (0 if edge_adjoint is None else min(chunk, ff.edge_capacity))
        ff(x)
        ff.buf["d_x"].fill_(float("nan"))                # every row is written anew
        out = ff(x)
        outputs.append([t.clone() for t in out] + [ff.buf["d_x"][:n_inner if n_inner > 0 else len(numbers)].clone()])
        ff.check_status()
    assert all(torch.equal(a, b) for a, b in zip(*outputs))
