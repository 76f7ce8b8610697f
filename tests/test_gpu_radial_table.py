"""The table-driven edge kernel against the float64 radial functions and against the MLP kernel it stands in for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _features(model, structure, table=True):
    from fastmace_b200 import _lib
    from fastmace_b200.forcefield import B200ForceField
    from fastmace_b200.model import SPECS, init_weights
    import ctypes
    spec = SPECS[model]
    x = torch.tensor(structure.positions, dtype=torch.float64, device="cuda")
    ff = B200ForceField(spec, init_weights(spec, 1), structure.numbers, structure.cell, positions=x)
    if not table:
        for layer in range(2):
            ff.packed.struct.layer[layer].rad_tab = None
    else:
        assert ff.packed.struct.layer[0].rad_tab and ff.packed.struct.layer[1].rad_tab
    _lib.check(ff.lib.fmb_edge_features(ff.packed.pointer(), ff.neighbours.pointer(), ctypes.byref(ff.work), x.data_ptr(),
                                        _lib.current_stream()), "fmb_edge_features")
    torch.cuda.synchronize()
    n = int(ff.edge_count)
    return ff, n, {k: ff.buf[k].cpu() for k in ("edge_vec", "edge_sh", "edge_hidden")}


@pytest.mark.parametrize("model,atoms", [("small", 1), ("medium", 2), ("medium", 9), ("large", 130)])
def test_features_of_the_table_kernel(model, atoms):
    """Edge counts from a handful (less than a warp's 16) to many blocks, none a multiple of a block. The values are off
    by the acceptance bound of the table (2e-7, 4e-7 of the largest magnitude) plus six fp32 roundings; the MLP kernel by
    its 3xTF32 layers."""
    from fastmace_b200.packing import radial_hidden_float64
    from fastmace_b200.structures import Structure
    rng = np.random.default_rng(atoms)
    edge = max(6.5, (atoms * 14.0) ** (1 / 3))
    s = Structure(rng.uniform(0, edge, (atoms, 3)), edge * np.eye(3) * (0.85 if atoms == 1 else 1.0),
                  rng.choice([11, 17], atoms) if atoms > 2 else np.full(atoms, 11))
    ff, n, got = _features(model, s)
    assert n > 0
    r = got["edge_vec"][:n, 3].double()
    largest = []
    for layer in range(2):
        ws = [ff.packed.tensors[f"l{layer}.rad.{i}"].cpu() for i in range(3)]
        largest.append([t.abs().max() for t in radial_hidden_float64(*ws, torch.linspace(0.1, 5.9, 400).double(), 6.0)])
        value, tangent = radial_hidden_float64(*ws, r, 6.0)
        assert (got["edge_hidden"][layer, 0, :n] - value).abs().max() <= 6e-7 * max(value.abs().max(), largest[layer][0])
        assert (got["edge_hidden"][layer, 1, :n] - tangent).abs().max() <= 1.2e-6 * max(tangent.abs().max(), largest[layer][1])
        assert not got["edge_hidden"][layer, :, n:].any()                 # nothing is written behind the edges
    _, m, other = _features(model, s, table=False)
    assert m == n
    assert torch.equal(other["edge_vec"][:n], got["edge_vec"][:n]) and torch.equal(other["edge_sh"][:n], got["edge_sh"][:n])
    for layer in range(2):
        for part in range(2):
            a, b = got["edge_hidden"][layer, part, :n], other["edge_hidden"][layer, part, :n]
            # the MLP kernel's fp32 envelope sums terms up to 35, off by 35 * 6e-8 of its maximum, before three layers
            assert (a - b).abs().max() <= 2e-5 * max(b.abs().max(), largest[layer][part])


def test_two_atoms_in_one_place_are_an_error():
    from fastmace_b200._lib import Fmb200Error
    from fastmace_b200.forcefield import B200ForceField
    from fastmace_b200.model import MEDIUM, init_weights
    from fastmace_b200.structures import nacl
    s = nacl((2, 2, 2), 0.05, 1)
    s.positions[5] = s.positions[0]
    ff = B200ForceField(MEDIUM, init_weights(MEDIUM, 1), s.numbers, s.cell)
    with pytest.raises(Fmb200Error):
        ff.evaluate(s)
