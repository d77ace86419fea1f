"""Which conditioning row a kernel is told to read for which entry, without a GPU: a kernel has no way of knowing how many rows its
tables have, so the host must not ask it to share fewer than there are."""
import itertools

import pytest
import torch

from kfold_b200 import functional as F
from kfold_b200 import modules as M

L, C, CS = 4, 16, 8


@pytest.mark.parametrize("lead", [(), (3,), (1, 5), (2, 3), (2, 1), (2, 3, 2)])
def test_every_broadcast_of_the_conditioning(lead):
    """All patterns of missing and size-one dims: the entry that the kernel reads (entry // share) is the one that broadcasting
    gives, and it exists."""
    a = torch.zeros(*lead, L, C)
    leads = {t[k:] for t in itertools.product(*[(1, d) for d in lead]) for k in range(len(lead) + 1)}
    for s_lead, rows in itertools.product(sorted(leads), (L, 1)):
        s = torch.randn(*s_lead, rows, CS)
        got, share = M._shared_conditioning(a, s)
        flat = got.reshape(-1, L, CS)
        entries = a.numel() // (L * C)
        assert flat.shape[0] * share == entries, (lead, s_lead, rows)
        want = s.expand(*lead, L, CS).reshape(-1, L, CS)
        assert all(torch.equal(flat[e // share], want[e]) for e in range(entries)), (lead, s_lead, rows)


def test_a_conditioning_that_does_not_broadcast_is_refused():
    for s in (torch.zeros(2, 5, CS), torch.zeros(3, L, CS), torch.zeros(2, 1, 2, L, CS)):
        with pytest.raises((ValueError, RuntimeError)):
            M._shared_conditioning(torch.zeros(1, 2, L, C), s)


@pytest.fixture()
def no_gpu_needed(monkeypatch):
    monkeypatch.setattr(F, "_require_cuda", lambda *t: None)

    def lib():
        raise AssertionError("the native library was called")

    monkeypatch.setattr(F.L, "lib", lib)


def test_tables_with_too_few_rows_are_refused(no_gpu_needed):
    a = torch.zeros(2, 2, L, C)
    pk = {"c": C, "hidden": 32, "heads": 2}
    for entries, share in ((1, 2), (2, 1), (4, 2)):      # tables of `entries` entries, told that `share` consecutive entries use one
        with pytest.raises(ValueError):
            F.adaln(a, torch.zeros(entries, L, 2 * C), share)
        with pytest.raises(ValueError):
            F.conditioned_transition(a, pk, torch.zeros(entries, L, C), share)
        with pytest.raises(ValueError):
            F.attention_pair_bias(a, torch.zeros(2, 1, 2, L, L), torch.ones(2, 1, L, dtype=torch.bool), pk,
                                  out_gate=torch.zeros(entries, L, C), gate_share=share)
    with pytest.raises(ValueError):
        F.adaln(a, torch.zeros(4, L, C), 1)


@pytest.mark.parametrize("s_lead,expected", [((2, 1), 1), ((2, 3), 3), ((1, 3), 3), ((1, 1), None)])
def test_token_stack_conditioning_entries(monkeypatch, no_gpu_needed, s_lead, expected):
    """Entries of conditioning per complex that the native call is told of: 1, or one per sample; one for all complexes is run
    block by block."""
    calls = []
    monkeypatch.setattr(M, "_check_inference", lambda x: None)
    monkeypatch.setattr(M.F, "token_stack", lambda a, s, pb, mask, plan, groups, samples, s_samples, *r: calls.append(
        (groups, samples, s_samples, s.numel() // (s.shape[-1] * s.shape[-2]))) or a)
    monkeypatch.setattr(M.CachedGlobalTransformerBlock, "forward", lambda self, a, *r, **k: calls.append(None) or a)
    stack = M.CachedGlobalTransformerStack(64, CS, 2, 1)
    monkeypatch.setattr(M._ConditioningBank, "tables", lambda self, s, adalns, gates: ([None] * len(adalns), [None] * len(gates)))
    with torch.no_grad():
        stack(torch.zeros(2, 3, 8, 64, dtype=torch.bfloat16), torch.zeros(*s_lead, 8, CS), torch.zeros(2, 1, 1, 2, 8, 8),
              torch.ones(2, 1, 8, dtype=torch.bool))
    assert calls == [None if expected is None else (2, 3, expected, 2 * expected)]
