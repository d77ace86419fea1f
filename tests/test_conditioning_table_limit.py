"""The float32 conditioning tables of an atom stack grow with atoms, entries and blocks: beyond a limit each block computes its own rows,
which are freed behind it."""
import pytest
import torch

from kfold_b200 import modules as M


class _Tables(Exception):
    pass


class _Blocks(Exception):
    pass


@pytest.mark.parametrize("blocks,entries,atoms", [(1, 1, 32), (2, 1, 64), (3, 2, 96)])
def test_tables_only_within_the_limit(monkeypatch, blocks, entries, atoms):
    def raises(what):
        def f(*a, **k):
            raise what
        return f

    c = 64
    monkeypatch.setattr(M, "_check_inference", lambda x: None)
    monkeypatch.setattr(M.F, "window_bias", lambda z, lw, lb, w, eps: torch.zeros(w.shape[0], *z.shape[:-1]))
    monkeypatch.setattr(M._ConditioningBank, "tables", raises(_Tables))
    monkeypatch.setattr(M.AdaLN, "gate_shift", raises(_Blocks))
    stack = M.LocalTransformerStack(c, c, 16, 2, blocks)
    rows_bytes = blocks * entries * atoms * (3 * 2 * c + 2 * c) * 4
    for limit, what in ((rows_bytes, _Tables), (rows_bytes - 1, _Blocks), (None, _Tables)):
        if limit is not None:
            monkeypatch.setattr(M.LocalTransformerStack, "table_limit", limit)
        else:
            monkeypatch.setattr(M.LocalTransformerStack, "table_limit", 1 << 30)
        with torch.no_grad(), pytest.raises(what):
            stack(torch.zeros(entries, 3, atoms, c), torch.zeros(entries, 1, atoms, c), torch.zeros(entries, 1, atoms // 32, 32, 128, 16),
                  torch.ones(entries, 1, atoms, dtype=torch.bool))
