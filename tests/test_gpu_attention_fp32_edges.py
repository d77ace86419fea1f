"""Float32 attention of many rows at the edges of its blocks (64 queries with one warp, 128 with two) and with a bias that does not start on a
16-byte boundary, which is copied in pieces of four bytes: the bits of one that does."""
import pytest
import torch

from helpers import err_stats
from oracle import pairformer_oracle as O
from test_gpu_parity import PRECISE_MAX_TOL, PRECISE_RMS_TOL, _oracle_on

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


@pytest.mark.parametrize("n", [80, 120, 128, 136, 192, 256])
@pytest.mark.parametrize("starting", [True, False])
def test_block_edges(dev, n, starting):
    from kfold_b200 import _lib as L, functional as F, packing
    import synth
    c, heads = 128, 4
    z, pm, _ = synth.pair_inputs(n, n, c, 1, valid=n - n // 9)
    w = synth.triatt_weights(synth._Rng(n + c), c, heads)
    out = F.triangle_attention(z.to(dev), pm.to(dev), packing.pack_triatt(w, heads, dev, precise=True), starting).cpu()
    ref = _oracle_on(dev, O.triangle_attention, z, pm, w, heads, starting)
    mx, r = err_stats(out, ref)
    assert mx < PRECISE_MAX_TOL and r < PRECISE_RMS_TOL, f"{mx:.3e} {r:.3e}"
    assert L.device_status() == 0


@pytest.mark.parametrize("l,heads,d", [(48, 12, 32), (72, 16, 24), (136, 24, 16)])
def test_a_bias_off_its_boundary(dev, l, heads, d):
    from kfold_b200 import _lib as L
    lib, c = L.lib(), heads * d
    batch = -(-2 * 148 // heads) + 1
    gen = torch.Generator(device=dev).manual_seed(l)
    x = torch.randn(batch, l, c, generator=gen, device=dev)
    w_proj = (torch.randn(4 * c, 6 * c, generator=gen, device=dev) * c ** -0.5).bfloat16()
    w_out = (torch.randn(c, 6 * c, generator=gen, device=dev) * c ** -0.5).bfloat16()
    mask = (torch.rand(batch, l, generator=gen, device=dev) > 0.2).to(torch.uint8)
    bias = torch.randn(heads * l * l, generator=gen, device=dev)
    need = lib.kfb_apb_workspace_bytes_precise(batch, l, c)
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    outs = []
    for off in (0, 1, 2):
        pb = torch.empty(bias.numel() + 4, device=dev)[off:off + bias.numel()]
        pb.copy_(bias)
        out = torch.empty(batch, l, c, device=dev)
        L.check(lib.kfb_apb_fwd(L.ptr(x), L.ptr(pb), L.ptr(mask), L.ptr(w_proj), None, L.ptr(w_out), None, None, 1, 0, L.ptr(out), None, L.ptr(ws), need,
                                batch, l, c, heads, batch, L.KFB_FP32_PRECISE, L.stream_ptr()))
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]) and bool(torch.isfinite(outs[0]).all())
    assert L.device_status() == 0
