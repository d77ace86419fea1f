"""The pair track's input projections in one kernel: bit for bit what LayerNorm and the projection GEMMs write (the row-shard entry points
still take those), at the edges of its runs (64 positions), tiles (two runs of a CTA, four of a pair) and units, with fewer tiles than pairs
and with more, transposed walks, ragged rows and several batches.  Projections are local to a position, so a ragged tensor is compared with
the padded one's part."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def _status():
    from kfold_b200 import _lib as L
    yield
    assert L.device_status() == 0


def _up(v, a):
    return (v + a - 1) // a * a


def _pieces(ws, *shapes):
    """The workspace's pieces in order, each on a 256-byte boundary."""
    out, off = [], 0
    for shape in shapes:
        count = 1
        for d in shape:
            count *= d
        out.append(ws[off:off + 2 * count].view(torch.bfloat16).view(shape))
        off += _up(2 * count, 256)
    return out


def _inputs(dev, batch, n, np_, c):
    gen = torch.Generator(device=dev).manual_seed(1000 * c + 10 * n + batch)
    x = torch.randn(batch, n, n, c, generator=gen, device=dev).mul_(1.5).add_(0.3).bfloat16()
    pad = torch.zeros(batch, np_, np_, c, device=dev, dtype=torch.bfloat16)
    pad[:, :n, :n] = x
    mask = torch.rand(batch, n, n, generator=gen, device=dev) > 0.2
    mpad = torch.zeros(batch, np_, np_, device=dev, dtype=torch.bool)
    mpad[:, :n, :n] = mask
    return x, pad, mask, mpad


@pytest.mark.parametrize("c,batch,n", [(128, 1, 24), (128, 2, 27), (128, 1, 63), (128, 1, 65), (128, 3, 64), (128, 1, 129), (128, 1, 200), (128, 1, 251),
                                       (256, 1, 24), (256, 2, 31), (256, 1, 64), (256, 1, 127), (256, 1, 193)])
@pytest.mark.parametrize("incoming", [0, 1])
def test_triangle_multiplication(dev, c, batch, n, incoming):
    from kfold_b200 import _lib as L, packing
    import synth
    lib = L.lib()
    pk = packing.pack_trimul(synth.trimul_weights(synth._Rng(c + n), c), dev)
    np_ = _up(n, 8)
    x, xpad, mask, mpad = _inputs(dev, batch, n, np_, c)
    need = lib.kfb_trimul_workspace_bytes(batch, n, c)
    ws = torch.zeros(need, dtype=torch.uint8, device=dev)
    out = torch.empty_like(x)
    before = L.launch_count()
    L.check(lib.kfb_trimul_fwd(incoming, L.ptr(x), L.ptr(mask), L.ptr(pk["ln_in_w"]), L.ptr(pk["ln_in_b"]), L.ptr(pk["w_in"]), L.ptr(pk["w_gout"]),
                               L.ptr(pk["ln_out_w"]), L.ptr(pk["ln_out_b"]), L.ptr(pk["w_pout"]), L.ptr(out), None, L.ptr(ws), need, batch, n, c, 1e-5,
                               L.KFB_BF16, L.stream_ptr()))
    assert L.launch_count() - before == 3
    _, ab, gl, _ = _pieces(ws, (batch, n, np_, c), (2 * c, batch, n, np_), (batch, n, n, c), (c, batch, n, np_))
    xn = torch.empty(batch * np_ * np_ * c, dtype=torch.bfloat16, device=dev)
    ab_ref = torch.empty(2 * c, batch, np_, np_, dtype=torch.bfloat16, device=dev)
    gl_ref = torch.empty(batch, np_, np_, c, dtype=torch.bfloat16, device=dev)
    L.check(lib.kfb_trimul_project(L.ptr(xpad), L.ptr(mpad), L.ptr(pk["ln_in_w"]), L.ptr(pk["ln_in_b"]), L.ptr(pk["w_in"]), L.ptr(pk["w_gout"]),
                                   L.ptr(xn), L.ptr(ab_ref), L.ptr(gl_ref), batch, np_, np_, c, incoming, 0, 1, 1e-5, L.KFB_BF16, L.stream_ptr()))
    assert torch.equal(ab[..., :n], ab_ref[:, :, :n, :n])
    assert torch.equal(gl, gl_ref[:, :n, :n])


@pytest.mark.parametrize("heads,n", [(4, 17), (2, 64), (4, 65), (2, 100), (4, 130), (4, 251)])
@pytest.mark.parametrize("ending", [0, 1])
def test_triangle_attention(dev, heads, n, ending):
    from kfold_b200 import _lib as L, packing
    import synth
    lib, c, batch = L.lib(), 128, 1
    pk = packing.pack_triatt(synth.triatt_weights(synth._Rng(heads + n), c, heads), heads, dev)
    np_ = _up(n, 16)
    x, xpad, mask, _ = _inputs(dev, batch, n, np_, c)
    need = lib.kfb_triatt_workspace_bytes(batch, n, c, heads)
    ws = torch.full((need,), 0x55, dtype=torch.uint8, device=dev)
    out = torch.empty_like(x)
    L.check(lib.kfb_triatt_fwd(ending, L.ptr(x), L.ptr(mask), L.ptr(pk["ln_w"]), L.ptr(pk["ln_b"]), L.ptr(pk["w_proj"]), L.ptr(pk["w_out"]), L.ptr(out),
                               None, L.ptr(ws), need, batch, n, c, heads, 1e-5, L.KFB_BF16, L.stream_ptr()))
    _, qkg, vt, bias = _pieces(ws, (n, n, c), (n, n, 384), (n, 128, np_), (heads, n, np_))
    src = xpad[0].transpose(0, 1).contiguous() if ending else xpad[0]
    xn = torch.empty(np_ * np_ * c, dtype=torch.bfloat16, device=dev)
    qkg_ref = torch.empty(np_, np_, 384, dtype=torch.bfloat16, device=dev)
    vt_ref = torch.empty(np_, 128, np_, dtype=torch.bfloat16, device=dev)
    bias_ref = torch.empty(heads, np_, np_, dtype=torch.bfloat16, device=dev)
    L.check(lib.kfb_triatt_project(L.ptr(src), L.ptr(pk["ln_w"]), L.ptr(pk["ln_b"]), L.ptr(pk["w_proj"]), L.ptr(xn), L.ptr(qkg_ref), L.ptr(vt_ref),
                                   L.ptr(bias_ref), np_, np_, c, heads, 0, 1e-5, L.KFB_BF16, L.stream_ptr()))
    assert torch.equal(qkg, qkg_ref[:n, :n])
    assert torch.equal(vt[..., :n], vt_ref[:n, :, :n])
    assert (vt[..., n:] == 0).all() and (bias[..., n:] == 0).all()
    if heads == 2:      # natural units on both sides
        assert torch.equal(bias[..., :n], bias_ref[:, :n, :n])
    else:               # log2 units: both sides round once, bias_ref before the factor
        got, want = bias[..., :n].float(), bias_ref[:, :n, :n].float() * 1.4426950408889634
        assert ((got - want).abs() <= 2.0 ** -7 * want.abs()).all()
