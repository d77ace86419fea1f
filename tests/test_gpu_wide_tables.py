"""GEMMs whose weights the L2 does not keep (above 16 MB): row blocks of a column tile follow each other.  Row counts that leave part of a row
block, that are odd numbers of row blocks and that go round the grid several times, with a last column tile that is not whole; against 64-bit
sums.  384 products in 24 steps of a truncating accumulator: 2 x 24 x 2^-23 of the absolute sum, and the result's own rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precise,n", [(False, 22016), (False, 22112), (True, 3744)])
@pytest.mark.parametrize("rows", [129, 301, 1031, 3840])
def test_against_wide_sums(precise, n, rows):
    from kfold_b200 import _lib as L, functional as F, packing
    dev, k = torch.device("cuda:0"), 384
    gen = torch.Generator(device=dev).manual_seed(rows + n)
    dt = torch.float32 if precise else torch.bfloat16
    x = torch.randn(rows, k, generator=gen, device=dev).to(dt)
    w = (torch.randn(n, k, generator=gen, device=dev) * k ** -0.5).to(dt)
    b = torch.randn(n, generator=gen, device=dev)
    packed = packing.split3_weights(w) if precise else w
    assert packed.numel() * 2 > 16 << 20
    out = (F.linear_fp32 if precise else F.linear)(x, packed, b)
    assert out.dtype == dt and out.shape == (rows, n)
    for c in range(0, n, 4096):
        s = slice(c, min(c + 4096, n))
        ref = x.double() @ w[s].double().T + b[s].double()
        terms = x.double().abs() @ w[s].double().abs().T + b[s].double().abs()
        bound = 48 * 2.0 ** -23 * terms + (2.0 ** -23 if precise else 2.0 ** -8) * ref.abs()
        assert ((out[:, s].double() - ref).abs() <= bound).all(), c
    assert L.device_status() == 0
