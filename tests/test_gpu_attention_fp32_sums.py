"""Float32 triangle attention's sums over keys.  Every position holds the same row, so that each key has the weight 1 and the same values, and a
sum in one accumulator rounds the same way for hundreds of keys: of 512, 256 at half a last place in the last binade alone, 0.29 x 256 x 2^-24 =
4.4e-6 root mean square over values.  In sums of eight keys it is an eighth of that for each binade, 4/3 of it for all: 7e-7, beside 5e-7 of the
products' six parts: 1.5e-6 is the bound."""
import pytest
import torch

from oracle import pairformer_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,heads", [(512, 128, 4), (511, 96, 4), (448, 64, 4)])
@pytest.mark.parametrize("starting", [True, False])
def test_equal_keys(monkeypatch, n, c, heads, starting):
    from kfold_b200 import _lib as L, modules as M
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(n + c)
    att = (M.TriangleAttentionStartingNode if starting else M.TriangleAttentionEndingNode)(c, heads).to(dev)
    with torch.no_grad():
        for name, p in att.named_parameters():
            p.normal_(0.0, p.shape[-1] ** -0.5 if p.dim() == 2 else 0.1, generator=gen).add_(1.0 if name.endswith("norm.weight") else 0.0)
        row = torch.randn(c, generator=gen, device=dev)
        z = row.expand(1, n, n, c).contiguous()
        mask = torch.ones(1, n, n, dtype=torch.bool, device=dev)
        out = att(z, mask)
        weights = {k: v.detach().double() for k, v in att.state_dict().items()}
        monkeypatch.setattr(torch.Tensor, "float", torch.Tensor.double)        # the oracle in 64 bits
        ref = O.triangle_attention(row.double().expand(1, 8, 8, c), mask[:, :8, :8], weights, heads, starting)
        monkeypatch.undo()
    err = out.double() - ref[0, 0, 0]
    assert float((err.pow(2).mean() / ref.pow(2).mean()).sqrt()) < 1.5e-6
    assert L.device_status() == 0
