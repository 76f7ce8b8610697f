"""The tile widths and the persistent form of the node linears' GEMM at their edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1, 128, 32), (129, 128, 96), (4700, 128, 128),      # up to 37 tiles of 128 columns: 32-column tiles, one to four stages
    (2300, 256, 160), (9400, 128, 64),                   # up to 74: 64-column tiles, K not a multiple of the stages
    (9601, 128, 416), (3100, 640, 128),                  # up to 148: 128-column tiles
    (19073, 128, 32), (9601, 384, 96), (40007, 128, 320),    # beyond: persistent, tiles of one and of many chunks
])
def test_gemm_tiles(m, n, k):
    """Bound: a truncation of 2^-23 per accumulating instruction (K / 8 of them) and the remainders dropped by the split
    (3 products of 2^-22), relative to the sum of magnitudes. Rows behind the last stay untouched; a row that is not
    a number spoils itself only."""
    from fastmace_b200 import _lib
    from fastmace_b200.packing import tensor_core_image
    lib = _lib.load()
    g = torch.Generator().manual_seed(m + n + k)
    a, b = torch.randn(m, k, generator=g).cuda(), torch.randn(k, n, generator=g)
    image = tensor_core_image([b]).cuda()
    b = b.cuda()
    status = torch.zeros((), dtype=torch.int32, device="cuda")
    bad = m // 2
    a[bad, k // 3] = float("nan")
    c = torch.full((m + 3, n), 7.0, device="cuda")
    for accumulate in (0, 1):
        _lib.check(lib.fmb_gemm(a.data_ptr(), b.data_ptr(), image.data_ptr(), None, c.data_ptr(), m, n, k, accumulate, 2,
                                status.data_ptr(), _lib.current_stream()), "gemm")
        keep = torch.arange(m, device="cuda") != bad
        ref = (accumulate + 1) * (a.double() @ b.double())[keep]
        size = (accumulate + 1) * (a.abs() @ b.abs())[keep].double()
        assert ((c[:m][keep].double() - ref).abs() <= (k / 8 + 8) * 2 ** -23 * size + 1e-30).all()
        assert c[bad].isnan().all() and (c[m:] == 7.0).all()
    assert int(status.item()) == 0


@pytest.mark.parametrize("m", [77, 40000])
def test_operands_up_to_the_end_of_fp32(m):
    """Activations of 1e38 to 3e38 with a product that fits: every step of the split stays finite. Bound: 3xTF32 of sums
    of one sign, K = 128."""
    from fastmace_b200 import _lib
    from fastmace_b200.packing import tensor_core_image
    g = torch.Generator().manual_seed(m)
    a = ((1 + 2 * torch.rand(m, 128, generator=g)) * 1e38).cuda()
    b = ((0.5 + torch.rand(128, 128, generator=g)) * 1e-3).cuda()
    image = tensor_core_image([b.cpu()]).cuda()
    c, status = torch.zeros(m, 128, device="cuda"), torch.zeros((), dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().fmb_gemm(a.data_ptr(), b.data_ptr(), image.data_ptr(), None, c.data_ptr(), m, 128, 128, 0, 2,
                                    status.data_ptr(), _lib.current_stream()), "gemm")
    want = a.double() @ b.double()
    assert bool(torch.isfinite(c).all()) and int(status) == 0
    assert float(((c.double() - want) / want).abs().max()) <= 2e-6
