"""Float32-accurate triangle attention of many rows: queries at the edges of a lane's pair (32), a warp's rows (64) and a block (256), keys at
the edges of a group (8) and a tile (32), each head dim, rows without any valid key; both directions, against the oracle.  (A token count that
is no multiple of eight is padded with masked tokens, which a row without any valid key averages too: those rows are left out there.)"""
import pytest
import torch

from helpers import err_stats
from oracle import pairformer_oracle as O
from test_gpu_parity import PRECISE_MAX_TOL, PRECISE_RMS_TOL, _oracle_on

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


@pytest.mark.parametrize("c,heads,n", [(128, 4, 74), (128, 4, 96), (128, 4, 127), (128, 4, 160), (128, 4, 193), (128, 4, 257), (64, 4, 75), (64, 4, 129),
                                       (96, 4, 80), (96, 4, 131)])
@pytest.mark.parametrize("starting", [True, False])
def test_against_oracle(dev, c, heads, n, starting):
    from kfold_b200 import _lib as L, functional as F, packing
    import synth
    z, pm, _ = synth.pair_inputs(n, n, c, 1, valid=n - n // 7)
    pm = pm & (torch.rand(pm.shape, generator=torch.Generator().manual_seed(n)) > 0.2)
    w = synth.triatt_weights(synth._Rng(n + c), c, heads)
    out = F.triangle_attention(z.to(dev), pm.to(dev), packing.pack_triatt(w, heads, dev, precise=True), starting).cpu()
    assert L.device_status() == 0
    ref = _oracle_on(dev, O.triangle_attention, z, pm, w, heads, starting)
    if not starting:
        out, ref, pm = out.transpose(1, 2), ref.transpose(1, 2), pm.transpose(1, 2)
    rows = pm[0].any(-1) if n % 8 else torch.ones(n, dtype=torch.bool)
    mx, r = err_stats(out[:, rows], ref[:, rows])
    assert mx < PRECISE_MAX_TOL and r < PRECISE_RMS_TOL, f"{mx:.3e} {r:.3e}"
