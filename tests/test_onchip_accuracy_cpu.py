"""Which layers are packed as fp16 pairs for the kernels that keep the last radial layer on the SM."""
import pytest
import torch


@pytest.mark.parametrize("factor,packed", [(1.0, True), (2.0 ** -10, True), (2.0 ** -18, False), (0.0, True)])
def test_a_layer_is_packed_only_where_fp16_pairs_hold_what_tf32_pairs_hold(factor, packed):
    """One channel far below the others: 2^-17 of the layer's largest weight is where the remainders lose bits."""
    from fastmace_b200._lib import IMAGE_ONCHIP
    from fastmace_b200.model import MEDIUM, init_weights
    from fastmace_b200.packing import PackedModel
    weights = dict(init_weights(MEDIUM, 1))
    weights["l1.rad.3"] = weights["l1.rad.3"].clone()
    weights["l1.rad.3"][:, 400] *= factor
    layer = PackedModel(MEDIUM, weights, [11, 17], "cpu").struct.layer[1]
    assert bool(layer.extra_images & IMAGE_ONCHIP) == packed


def test_accuracy_is_that_of_the_products():
    """The criterion itself against float64 products of the split operands, entry by entry of the layout, for features that
    vanish at the cutoff like those of a radial MLP."""
    from fastmace_b200.packing import onchip_image, onchip_is_accurate
    g = torch.Generator().manual_seed(3)
    w4, shape = torch.randn(64, 1280, generator=g) / 8, torch.randn(50, 64, generator=g).double()
    r = 6.0 - torch.logspace(-2.5, 0.7, 50, dtype=torch.float64)
    features, tangents = shape * (6.0 - r)[:, None] ** 4, 4.0 * shape * (6.0 - r)[:, None] ** 3
    size = float(shape.abs().max())
    long = (5.5, 6.0, 8 * size, 16 * size)                    # scales 32768 / 2^10 = 32 and 16: 4 a d^4 is their largest
    image = onchip_image(w4, 1024.0, 2048.0, long)
    assert onchip_is_accurate(w4, image, r, features, tangents)
    common = onchip_image(w4, 1024.0, 2048.0)                 # one scale for all lengths
    assert not onchip_is_accurate(w4, common, r, features, tangents)
    exchanged = w4.clone()
    exchanged[[7, 8], 1111] = w4[[8, 7], 1111]                # the image of another layer
    assert not onchip_is_accurate(exchanged, image, r, features, tangents)
