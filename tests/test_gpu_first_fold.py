"""The adjoint of the first-layer fold for odd numbers of species: 64 columns per species leave half a column tile, which the
packed image pads with zeros and the kernels do not store."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ELEMENTS = (11, 17, 8, 14, 26, 29, 47)


@pytest.mark.parametrize("species,atoms", [
    (1, 100), (3, 100), (5, 64), (7, 40),                     # up to 37 tiles of 128 columns: tiles of 32
    (1, 500), (3, 250), (5, 150), (7, 128),                   # up to 74: of 64
    (1, 1000), (3, 500), (5, 300), (7, 250),                  # up to 148: of 128
    (1, 2000), (3, 900), (5, 700), (7, 600),                  # beyond: persistent
])
def test_gradient_of_the_outer_products_and_nothing_beside_it(species, atoms):
    """A force call leaves the operand in d_msg and the product in d_mid. Bound: a truncation of 2^-23 per accumulating
    instruction (16 of them) and the remainders dropped by the split (3 products of 2^-22; 8 x 2^-23 in all), relative to the
    sum of magnitudes."""
    from fastmace_b200.forcefield import B200ForceField
    from fastmace_b200.model import SMALL, init_weights
    rng = np.random.default_rng(atoms)
    side = int(np.ceil(atoms ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:atoms]
    positions = torch.tensor(4.0 * grid + rng.uniform(-0.5, 0.5, (atoms, 3)), device="cuda")
    numbers = np.array(ELEMENTS)[np.arange(atoms) % species]
    ff = B200ForceField(SMALL, init_weights(SMALL, 2), numbers, np.eye(3) * max(4.0 * side, 14.0), positions=positions,
                        atom_capacity=atoms + 3)
    assert ff.packed.struct.layer[0].extra_images
    product, width = ff.buf["d_mid"].reshape(-1), 64 * species
    product.fill_(7.0)
    ff(positions)
    ff.check_status()
    d_msg = ff.buf["d_msg"][:atoms].double()
    got = product[:atoms * 16 * width].reshape(atoms, 16, width).double()
    weights = ff.packed.tensors["l0.first_t"].double().reshape(4, 128, width)
    for l in range(4):
        a, b = d_msg[:, l * l:(l + 1) ** 2], weights[l]
        assert a.norm() > 0
        off = (got[:, l * l:(l + 1) ** 2] - a @ b).abs()
        assert (off <= (16 + 8) * 2.0 ** -23 * (a.abs() @ b.abs()) + 1e-30).all()
    behind = product[atoms * 16 * width:][:64]
    # one species: the second interaction's gradient [atoms][16][128] came before and reaches further
    assert (behind != 0).all() if species == 1 else (behind == 7.0).all()
