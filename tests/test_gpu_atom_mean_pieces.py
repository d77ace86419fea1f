"""The mean over a token's atoms by pieces of 16 and 8 bytes and by single channels: widths on either side of each rule, results that start
between pieces and whose neighbours stay as they are; sums of up to 40 bf16 values are held to float32's rounding of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,d,off", [(torch.bfloat16, 4, 0), (torch.bfloat16, 12, 0), (torch.bfloat16, 12, 2), (torch.bfloat16, 124, 4),
                                         (torch.bfloat16, 128, 0), (torch.bfloat16, 128, 4), (torch.bfloat16, 128, 1), (torch.bfloat16, 132, 0),
                                         (torch.bfloat16, 136, 0), (torch.bfloat16, 136, 4), (torch.bfloat16, 768, 0), (torch.bfloat16, 768, 1),
                                         (torch.bfloat16, 131, 3), (torch.float32, 12, 0), (torch.float32, 132, 1), (torch.float32, 130, 0)])
def test_widths_and_offsets(dtype, d, off):
    from kfold_b200 import _lib as L
    dev, batch, n_atom, n_token = torch.device("cuda:0"), 2, 200, 31
    gen = torch.Generator(device=dev).manual_seed(d + off)
    index = torch.cat([torch.zeros(40, dtype=torch.long, device=dev), torch.randint(2, 30, (160,), generator=gen, device=dev)]).sort().values
    index = index.view(1, n_atom)
    mask = (torch.rand(1, n_atom, generator=gen, device=dev) < 0.8)
    x = torch.randn(batch, n_atom, d, generator=gen, device=dev).to(dtype)
    buf = torch.full((off + batch * n_token * d + 16,), 7.0, device=dev, dtype=dtype)
    out = buf[off:off + batch * n_token * d].view(batch, n_token, d)
    L.check(L.lib().kfb_atoms_to_tokens(L.ptr(x), L.ptr(index), L.ptr(mask.view(torch.uint8)), L.ptr(out), None, 0, batch, n_atom, n_token, d, batch, 1,
                                        L.dtype_code(dtype), L.stream_ptr()))
    member = ((index[0][None, :] == torch.arange(n_token, device=dev)[:, None]) & mask[0]).double()
    count = member.sum(1).clamp(min=1.0)[:, None]
    pos = x.double().clamp(min=0.0)
    ref = member @ pos / count
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    assert ((out.double() - ref).abs() <= ulp * ref.abs() + 40 * 2.0 ** -23 * ref.abs()).all()
    assert (buf[:off] == 7.0).all() and (buf[off + batch * n_token * d:] == 7.0).all()
    assert L.device_status() == 0
