"""What a host built against the header may rely on: buffers it may use between phases, and fields it may leave unset."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _crystal():
    from fastmace_b200.model import MEDIUM, init_weights
    from fastmace_b200.structures import nacl
    return MEDIUM, init_weights(MEDIUM, 1), nacl((4, 4, 3), 0.05, 1)


def _outputs(ff):
    return [t.clone() for t in (ff.energy, ff.forces, ff.stress)]


@pytest.mark.parametrize("chunk", [None, 1 << 12])
def test_weight_buffer_is_free_between_the_second_and_the_last_phase(chunk):
    """Ranks played on one device may share tp_w once the second interaction's adjoint is through."""
    from fastmace_b200.forcefield import B200ForceField
    spec, weights, s = _crystal()
    x = torch.tensor(s.positions, device="cuda")
    ff = B200ForceField(spec, weights, s.numbers, s.cell, compute_stress=True, positions=x, n_owned=s.natoms, n_inner=s.natoms,
                        halo_exchange=True, chunk_edges=chunk)
    results = []
    for spoil in (False, True):
        for index in range(3):
            ff.phase(index, x)
            if spoil and index == 1:
                ff.buf["tp_w"].fill_(float("nan"))
        results.append(_outputs(ff))
    ff.check_status()
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("left", [1, 3, -1])
def test_a_layer_whose_padding_was_left_unset_selects_no_extra_image(left):
    """Hosts of the same header version knew fmb_layer_t.extra_images as padding."""
    from fastmace_b200.forcefield import B200ForceField
    spec, weights, s = _crystal()
    x = torch.tensor(s.positions, device="cuda")
    ff = B200ForceField(spec, weights, s.numbers, s.cell, compute_stress=True, positions=x)
    results = []
    for value in (0, left):
        for layer in ff.packed.struct.layer:
            layer.extra_images = value
        ff(x)
        results.append(_outputs(ff))
    ff.check_status()
    assert all(torch.equal(a, b) for a, b in zip(*results))
