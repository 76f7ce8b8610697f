"""The last radial layer as the kernels that keep it in tensor memory read it."""
import pytest
import torch

from fastmace_b200.packing import ONCHIP_HEADER, onchip_image


@pytest.mark.parametrize("paths", [10])
def test_image_holds_the_layer_to_22_bits(paths):
    w4 = torch.randn(64, paths * 128, generator=torch.Generator().manual_seed(paths)) / 8
    flat = onchip_image(w4, 3.0, 50.0)
    assert float(flat[0]) == 2.0 ** 13 and float(flat[1]) == 2.0 ** 9        # 3 and 50 reach half of the fp16 range
    scale = 1.0 / (float(flat[2]) * float(flat[0]))
    image = flat[ONCHIP_HEADER:].view(torch.float16).double().reshape(2, paths // 2, 2, 8, 128, 8)
    rows = image.sum(2).transpose(2, 3).reshape(2, paths, 64, 64) / scale
    want = w4.double().t().reshape(paths, 2, 64, 64).transpose(0, 1)
    assert (rows - want).abs().max() <= 2.0 ** -22 * w4.abs().max()
