"""The pair track's transition in one kernel, at the edges of its tiles (128 rows of a CTA, 256 of a pair), at more tiles than pairs, at the
fewest hidden channels, with and without residual, in place; against the oracle and, bit for bit, against the three launches that a
destination off by eight bytes still takes."""
import pytest
import torch

from helpers import err_stats
from oracle import pairformer_oracle as O
from test_gpu_parity import _check, _oracle_on

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def _status():
    from kfold_b200 import _lib as L
    yield
    assert L.device_status() == 0


def _call(x, out, resid, pk):
    from kfold_b200 import _lib as L
    lib = L.lib()
    rows, c, hidden = x.shape[0], pk["c"], pk["hidden"]
    need = lib.kfb_transition_workspace_bytes(rows, c, hidden)
    ws = torch.empty(need, dtype=torch.uint8, device=x.device)
    before = L.launch_count()
    L.check(lib.kfb_transition_fwd(L.ptr(x), L.ptr(pk["ln_w"]), L.ptr(pk["ln_b"]), L.ptr(pk["w_swiglu"]), L.ptr(pk["w_out"]), L.ptr(out),
                                   L.ptr(resid), L.ptr(ws), need, rows, c, hidden, 1e-5, L.KFB_BF16, L.stream_ptr()))
    return L.launch_count() - before


@pytest.mark.parametrize("c,factor,rows", [(128, 4, 1), (128, 4, 127), (128, 4, 128), (128, 4, 129), (128, 1, 256), (128, 1, 57001), (128, 4, 37889),
                                           (256, 4, 1), (256, 4, 255), (256, 4, 257), (256, 1, 57001), (256, 2, 18944)])
def test_one_launch(dev, c, factor, rows):
    from kfold_b200 import packing
    import synth
    w = synth.transition_weights(synth._Rng(c + rows), c, factor)
    pk = packing.pack_transition(w, dev)
    x = torch.randn(rows, c, generator=torch.Generator().manual_seed(rows)).mul_(1.5).add_(0.3).bfloat16()
    xd = x.to(dev)
    other = torch.randn(rows, c, generator=torch.Generator().manual_seed(rows + 1)).bfloat16().to(dev)
    ref = _oracle_on(dev, O.transition, x.float()[None], w)[0]
    for resid in (None, xd, other):
        buf = torch.full((rows * c + 16,), 7.0, device=dev, dtype=torch.bfloat16)
        out = buf[:rows * c].view(rows, c)
        assert _call(xd, out, resid, pk) == 1
        _check(*err_stats(out.float().cpu(), ref if resid is None else ref + resid.float().cpu()), f"transition c={c} rows={rows}")
        assert (buf[rows * c:] == 7.0).all()
        off = torch.empty(rows * c + 8, device=dev, dtype=torch.bfloat16)[4:4 + rows * c].view(rows, c)
        assert _call(xd, off, resid, pk) == 3
        assert torch.equal(off, out)
    assert _call(xd, xd, xd, pk) == 1        # in place
    _check(*err_stats(xd.float().cpu(), ref + x.float()), f"transition in place c={c} rows={rows}")
