"""Triangle attention's LayerNorm and projections in one launch from 16 tiles of four runs on, in two below: on either side of the line, with
one and with several complexes, the q, k, g, V^T of either are the bits of the row-shard entry point."""
import pytest
import torch

from test_gpu_pair_project import _inputs, _pieces, _up

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n,one", [(1, 24, False), (1, 60, False), (1, 61, True), (1, 64, True), (2, 30, False), (2, 31, True), (3, 27, True),
                                         (7, 9, True)])
@pytest.mark.parametrize("ending", [0, 1])
def test_route(batch, n, one, ending):
    from kfold_b200 import _lib as L, packing
    import synth
    dev, lib, c, heads = torch.device("cuda:0"), L.lib(), 128, 4
    pk = packing.pack_triatt(synth.triatt_weights(synth._Rng(heads + n), c, heads), heads, dev)
    np_ = _up(n, 16)
    x, xpad, mask, _ = _inputs(dev, batch, n, np_, c)
    need = lib.kfb_triatt_workspace_bytes(batch, n, c, heads)
    ws = torch.full((need,), 0x55, dtype=torch.uint8, device=dev)
    out = torch.empty_like(x)
    L.profile_enable(True)
    L.check(lib.kfb_triatt_fwd(ending, L.ptr(x), L.ptr(mask), L.ptr(pk["ln_w"]), L.ptr(pk["ln_b"]), L.ptr(pk["w_proj"]), L.ptr(pk["w_out"]), L.ptr(out),
                               None, L.ptr(ws), need, batch, n, c, heads, 1e-5, L.KFB_BF16, L.stream_ptr()))
    torch.cuda.synchronize()
    tags = L.profile_report()
    L.profile_enable(False)
    assert ("triatt_project" in tags) == one and ("triatt_proj" in tags) != one
    _, qkg, vt, bias = _pieces(ws, (batch, n, n, c), (batch, n, n, 384), (batch, n, 128, np_), (batch, heads, n, np_))
    for b in range(batch):
        src = xpad[b].transpose(0, 1).contiguous() if ending else xpad[b]
        xn = torch.empty(np_ * np_ * c, dtype=torch.bfloat16, device=dev)
        qkg_ref = torch.empty(np_, np_, 384, dtype=torch.bfloat16, device=dev)
        vt_ref = torch.empty(np_, 128, np_, dtype=torch.bfloat16, device=dev)
        bias_ref = torch.empty(heads, np_, np_, dtype=torch.bfloat16, device=dev)
        L.check(lib.kfb_triatt_project(L.ptr(src), L.ptr(pk["ln_w"]), L.ptr(pk["ln_b"]), L.ptr(pk["w_proj"]), L.ptr(xn), L.ptr(qkg_ref), L.ptr(vt_ref),
                                       L.ptr(bias_ref), np_, np_, c, heads, 0, 1e-5, L.KFB_BF16, L.stream_ptr()))
        assert torch.equal(qkg[b], qkg_ref[:n, :n])
        assert torch.equal(vt[b][..., :n], vt_ref[:n, :, :n])
    assert (vt[..., n:] == 0).all() and (bias[..., n:] == 0).all()
    assert L.device_status() == 0
