"""The tabulated hidden radial features against the float64 function they stand for."""
import math

import pytest
import torch

from fastmace_b200.model import SPECS, init_weights
from fastmace_b200.packing import radial_hidden_float64, radial_table


def _weights(model, layer, scale=1.0):
    w = init_weights(SPECS[model], 1)
    ws = [w[f"l{layer}.rad.{i}"] for i in range(3)]
    return [(scale * m / math.sqrt(m.shape[0])).to(torch.float32) for m in ws]


def test_tangent_is_the_derivative():
    ws = _weights("medium", 0)
    r = torch.tensor([1e-3, 0.3, 1.7, 2.82, 4.0, 5.9], dtype=torch.float64)
    h = 1e-5
    up, down = (radial_hidden_float64(*ws, r + s * h, 6.0)[0] for s in (1, -1))
    tangent = radial_hidden_float64(*ws, r, 6.0)[1]
    assert (tangent - (up - down) / (2 * h)).abs().max() < 1e-7 * tangent.abs().max()


@pytest.mark.parametrize("model,layer,r_cut,scale", [("small", 0, 6.0, 1.0), ("medium", 1, 6.0, 1.0),
                                                     ("large", 1, 4.3, 1.0), ("medium", 0, 6.0, 2.0)])
def test_table_reproduces_the_mlp(model, layer, r_cut, scale):
    """Between the nodes too, and with steeper functions (larger weights) on finer intervals. Bounds: those the table is
    accepted with, times three for points that were not probed."""
    ws = _weights(model, layer, scale)
    table, per = radial_table(*ws, r_cut)
    assert table.dtype == torch.float32 and table.shape[0] >= per * r_cut
    r = torch.rand(4001, dtype=torch.float64, generator=torch.Generator().manual_seed(3)) * (r_cut - 0.01) + 0.005
    i = torch.floor(r * per).long()
    u = (2 * (r * per - i) - 1)[:, None]
    c = table.double()[i]
    powers = torch.cat([u ** k for k in range(6)], 1)
    slopes = torch.cat([k * u ** max(k - 1, 0) for k in range(6)], 1) * (2 * per)
    value, tangent = radial_hidden_float64(*ws, r, r_cut)
    assert ((powers[:, :, None] * c).sum(1) - value).abs().max() <= 6e-7 * value.abs().max()
    assert ((slopes[:, :, None] * c).sum(1) - tangent).abs().max() <= 1.2e-6 * tangent.abs().max()
    if scale > 1:
        assert per > 32


def test_a_function_no_table_serves_is_refused():
    assert radial_table(*_weights("medium", 0, 400.0), 6.0) is None


def test_table_is_accurate_at_every_length():
    """One feature 2e5 at contact and next to nothing from 1.5 Å on, beside steep ones of order one: what the table is off
    by at a bond's length must be measured against the features there. Bounds: those of the acceptance, times three for
    points that were not probed."""
    r_cut = 6.0
    r = torch.linspace(0.05, 5.9, 400, dtype=torch.float64)
    k, x = torch.arange(1, 9) * math.pi / r_cut, (r / r_cut)[:, None]
    basis = math.sqrt(2 / r_cut) * torch.sin(r[:, None] * k) / r[:, None] * (1 + x ** 5 * (-21 + 35 * x - 15 * x * x))
    peak = torch.linalg.lstsq(basis, (2 * (1 - r).clamp(min=0) ** 2)[:, None]).solution[:, 0].float()
    w0, w1, w2 = torch.zeros(8, 64), torch.zeros(64, 64), torch.zeros(64, 64)
    w0[:, 0], w0[:, 1] = peak, -peak                       # silu(z) + silu(-z) is about z^2 / 2: quadratic where z is small
    w1[0:2, 0], w1[0:2, 1], w2[0:2, 0] = 1.0, -1.0, 1e5
    w0[:, 2:10], w0[:, 10:18] = torch.eye(8), -torch.eye(8)
    g = torch.Generator().manual_seed(0)
    w1[2:18, 2:34] = 10 * torch.randn(16, 32, generator=g)
    w2[2:34, 1:64] = torch.randn(32, 63, generator=g) / 50
    found = radial_table(w0, w1, w2, r_cut)
    assert found is not None
    table, per = found
    r = torch.rand(20001, dtype=torch.float64, generator=torch.Generator().manual_seed(3)) * (r_cut - 0.01) + 0.005
    i = torch.floor(r * per).long()
    u = (2 * (r * per - i) - 1)[:, None]
    c = table.double()[i]
    got = sum(c[:, q] * u ** q for q in range(6))
    d_got = sum(q * c[:, q] * u ** (q - 1) for q in range(1, 6)) * (2 * per)
    value, tangent = radial_hidden_float64(w0, w1, w2, r, r_cut)
    for low in torch.arange(0, r_cut, 0.25):
        at = (r >= low) & (r < low + 0.25)
        assert (got - value)[at].abs().max() <= 6e-7 * value[at].abs().max(), float(low)
        assert (d_got - tangent)[at].abs().max() <= 1.2e-6 * tangent[at].abs().max(), float(low)
