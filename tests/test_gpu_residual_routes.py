"""Output projections onto a float32 residual stream: a row's result, bit for bit, is that of the same row among many more (whose tiles are
several waves and K goes by in one accumulator), for every width of the one-wave tiles and on either side of where K is shared; then what the
gate, the bias and the residual each add, one without the other."""
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


# (in the order of the columns of a tile: 64, 96, 128, 192, 256)
@pytest.mark.parametrize("c,hidden,samples,l", [
    (768, 768, 1, 129), (768, 768, 1, 384), (768, 1536, 1, 385), (768, 1536, 1, 513), (768, 1536, 1, 768), (768, 1536, 5, 96), (1024, 1024, 1, 301),
    (320, 640, 1, 700), (64, 128, 1, 65), (768, 1536, 5, 384), (768, 768, 7, 257), (128, 256, 1, 9000), (1024, 2048, 2, 1023), (768, 768, 5, 520),
    (768, 1536, 5, 700), (1024, 1024, 5, 800)])
@pytest.mark.parametrize("with_resid", [True, False])
def test_a_row_does_not_depend_on_the_rows_beside_it(dev, c, hidden, samples, l, with_resid):
    from kfold_b200 import _lib as L
    lib = L.lib()
    gen = torch.Generator(device=dev).manual_seed(c + hidden + l)
    w1 = (torch.randn(2 * hidden, c, generator=gen, device=dev) * c ** -0.5).bfloat16()
    w2 = (torch.randn(c, hidden, generator=gen, device=dev) * hidden ** -0.5).bfloat16()
    gate = torch.randn(l, c, generator=gen, device=dev).bfloat16()
    many = max(2 * samples, -(-40000 // l))
    x = torch.randn(many * l, c, generator=gen, device=dev).bfloat16()
    resid = torch.randn(many * l, c, generator=gen, device=dev)

    def call(s):
        rows = s * l
        out = torch.empty(rows, c, device=dev)
        need = lib.kfb_cond_transition_workspace_bytes(rows, hidden)
        ws = torch.empty(need, dtype=torch.uint8, device=dev)
        L.check(lib.kfb_cond_transition_fwd(L.ptr(x), L.ptr(w1), L.ptr(w2), L.ptr(gate), c, L.ptr(out), L.ptr(resid) if with_resid else None, L.ptr(ws),
                                            need, rows, c, hidden, s, l, L.KFB_FP32, L.stream_ptr()))
        return out

    few, all_rows = call(samples), call(many)
    assert torch.equal(few, all_rows[:samples * l])


@pytest.mark.parametrize("batch,l", [(1, 200), (3, 192), (5, 384), (5, 768)])
def test_gate_bias_and_residual_by_themselves(dev, batch, l):
    """768 channels, 16 heads; a gate of sigmoid 1 (logit 60) multiplies by one, so that it and no gate give the same bits."""
    from kfold_b200 import _lib as L
    lib, c, heads, dp = L.lib(), 768, 16, 64
    gen = torch.Generator(device=dev).manual_seed(batch * l)
    x = torch.randn(batch, l, c, generator=gen, device=dev).bfloat16()
    pb = torch.randn(1, heads, l, l, generator=gen, device=dev).bfloat16()
    mask = torch.ones(batch, l, dtype=torch.uint8, device=dev)
    w_proj = (torch.randn(4 * heads * dp, c, generator=gen, device=dev) * c ** -0.5).bfloat16()
    w_out = (torch.randn(c, c, generator=gen, device=dev) * c ** -0.5).bfloat16()
    bias = torch.randn(c, generator=gen, device=dev)
    resid = torch.randn(batch, l, c, generator=gen, device=dev)
    ones = torch.full((batch, l, c), 60.0, device=dev).bfloat16()
    need = lib.kfb_apb_workspace_bytes(batch, l, c, heads)
    ws = torch.empty(need, dtype=torch.uint8, device=dev)

    def call(b, g, r):
        out = torch.empty(batch, l, c, device=dev)
        L.check(lib.kfb_apb_fwd(L.ptr(x), L.ptr(pb), L.ptr(mask), L.ptr(w_proj), None, L.ptr(w_out), L.ptr(b), L.ptr(g), 1, 0, L.ptr(out), L.ptr(r),
                                L.ptr(ws), need, batch, l, c, heads, batch, L.KFB_FP32, L.stream_ptr()))
        return out

    bare = call(None, ones, None)
    full = call(bias, None, resid)
    assert torch.equal(full, call(bias, ones, resid))
    assert torch.equal(call(None, None, resid), bare + resid)
    assert torch.equal(full, (bare + bias) + resid)
