"""Output projections onto the float32 residual stream, at the edges of their runs (64 rows), tiles (128 rows of a CTA, 256 of a pair) and
widths, rows that do not divide, gates shared by the samples, in place: against 64-bit sums of the same bf16 operands."""
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


@pytest.mark.parametrize("c,groups,samples,l", [(128, 1, 1, 700), (128, 2, 3, 130), (192, 1, 2, 257), (320, 1, 4, 65), (768, 1, 1, 1), (768, 1, 1, 641),
                                                (768, 1, 5, 63), (768, 1, 5, 193), (768, 1, 5, 768), (768, 2, 2, 301), (1024, 1, 4, 321), (1024, 1, 5, 800)])
@pytest.mark.parametrize("in_place", [False, True])
def test_gate_and_residual(dev, c, groups, samples, l, in_place):
    from kfold_b200 import _lib as L, packing
    import synth
    lib, hidden = L.lib(), 2 * c
    pk = packing.pack_cond_transition(synth.conditioned_transition_weights(synth._Rng(c + l), c, 64), dev)
    rows = groups * samples * l
    gen = torch.Generator(device=dev).manual_seed(rows + c)
    x = torch.randn(rows, c, generator=gen, device=dev).bfloat16()
    gate = torch.randn(groups * l, c + 8, generator=gen, device=dev).bfloat16()        # wider rows, as a stack's table has
    resid = torch.randn(rows, c, generator=gen, device=dev)
    buf = torch.full((rows * c + 64,), 7.0, device=dev)
    out = buf[:rows * c].view(rows, c)
    if in_place:
        out.copy_(resid)
    need = lib.kfb_cond_transition_workspace_bytes(rows, hidden)
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    L.check(lib.kfb_cond_transition_fwd(L.ptr(x), L.ptr(pk["w_swiglu"]), L.ptr(pk["w_out"]), L.ptr(gate), c + 8, L.ptr(out),
                                        L.ptr(out if in_place else resid), L.ptr(ws), need, rows, c, hidden, samples, l, L.KFB_FP32, L.stream_ptr()))
    h = ws[:rows * hidden * 2].view(torch.bfloat16).view(rows, hidden).double()
    g = torch.sigmoid(gate[:, :c].double()).view(groups, 1, l, c).expand(groups, samples, l, c).reshape(rows, c)
    update = (h @ pk["w_out"].double().T) * g
    # the gate's hardware tanh: 2^-11 of its argument's half range; sums in float32: 1e-6 of the terms
    bound = 2.0 ** -10 * update.abs() + 2e-5 * (h.abs() @ pk["w_out"].double().abs().T) + 1e-6 * resid.abs()
    assert ((out.double() - (resid.double() + update)).abs() <= bound + 1e-6).all()
    assert (buf[rows * c:] == 7.0).all()
