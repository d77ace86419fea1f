"""What the native calls are told about their tensors.  Which conditioning row a kernel is told to read for which entry, without a GPU: a kernel has no way of knowing how many rows its
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


# ------------------------------------------------------------------------------------------------ shapes of the stacks' native calls
def _token_args():
    return {"a": torch.zeros(2, 3, 8, 64, dtype=torch.bfloat16), "s": torch.zeros(2, 1, 8, CS), "pair_bias": torch.zeros(2, 1, 2, 2, 8, 8),
            "mask": torch.ones(2, 1, 8, dtype=torch.bool)}


def _atom_args():
    return {"a": torch.zeros(2, 3, 64, 64, dtype=torch.bfloat16), "s": torch.zeros(2, 1, 64, 64), "z": torch.zeros(2, 1, 2, 32, 128, 16),
            "mask": torch.ones(2, 1, 64, dtype=torch.bool)}


def _cut(t, dim, by):
    return t.narrow(dim, 0, t.shape[dim] - by) if by > 0 else torch.cat([t, t.narrow(dim, 0, -by)], dim)


@pytest.mark.parametrize("which,arg,dim,by", [
    ("token", "a", -1, 8), ("token", "s", -1, 1), ("token", "s", -1, -2), ("token", "pair_bias", -1, 1), ("token", "pair_bias", -1, -4),
    ("token", "pair_bias", -2, 2), ("token", "pair_bias", -3, 1), ("token", "pair_bias", -4, 1), ("token", "mask", -1, 1),
    ("token", "mask", -1, -3), ("token", "s", -2, 1), ("atom", "a", -1, 8), ("atom", "s", -1, 8), ("atom", "s", -2, 4), ("atom", "z", -4, -1),
    ("atom", "z", -2, 8), ("atom", "z", -3, 1), ("atom", "z", -1, 4), ("atom", "mask", -1, 32), ("atom", "mask", -1, -64)])
def test_a_wrong_extent_is_refused(monkeypatch, no_gpu_needed, which, arg, dim, by):
    """One argument shorter or longer than the others say, along one dim: the kernels address by the extents they are told."""
    monkeypatch.setattr(M, "_check_inference", lambda x: None)
    if which == "token":
        stack, args = M.CachedGlobalTransformerStack(64, CS, 2, 2), _token_args()
    else:
        stack, args = M.LocalTransformerStack(64, 64, 16, 2, 2), _atom_args()
        if arg != "z" or dim == -4:      # the window biases are another call's concern
            monkeypatch.setattr(M.F, "window_bias", lambda z, lw, lb, w, eps: torch.zeros(w.shape[0], *z.shape[:-1]))
    args[arg] = _cut(args[arg], dim, by)
    with torch.no_grad(), torch.autocast("cpu", dtype=torch.bfloat16), pytest.raises((ValueError, RuntimeError, IndexError)):
        stack(**args)


@pytest.mark.parametrize("which", ["token", "atom"])
def test_right_extents_reach_the_native_call(monkeypatch, no_gpu_needed, which):
    monkeypatch.setattr(M, "_check_inference", lambda x: None)
    stack, args = ((M.CachedGlobalTransformerStack(64, CS, 2, 2), _token_args()) if which == "token"
                   else (M.LocalTransformerStack(64, 64, 16, 2, 2), _atom_args()))
    monkeypatch.setattr(M.F, "window_bias", lambda z, lw, lb, w, eps: torch.zeros(w.shape[0], *z.shape[:-1]))
    with torch.no_grad(), torch.autocast("cpu", dtype=torch.bfloat16):
        with pytest.raises(AssertionError, match="the native library was called"):
            stack(**args)
        if which == "token":      # a mask of one value per complex is spread over its tokens
            args["mask"] = torch.ones(2, 1, 1, dtype=torch.bool)
            with pytest.raises(AssertionError, match="the native library was called"):
                stack(**args)


def test_projections_of_other_widths_are_refused(no_gpu_needed):
    with pytest.raises(ValueError):
        F.linear(torch.zeros(4, 16), torch.zeros(8, 24))
    with pytest.raises(ValueError):
        F.window_bias(torch.zeros(2, 32, 128, 16), None, None, torch.zeros(4, 8))


@pytest.mark.parametrize("cls", ["PairformerBlock", "ConfidencePairSingleBlock"])
@pytest.mark.parametrize("b,s_lead,mask_lead,one", [(2, (2,), (2,), True), (2, (2,), (1,), False), (2, (2,), (), False), (1, (1, 3), (1, 1), False)])
def test_blocks_take_what_their_operators_take(monkeypatch, no_gpu_needed, cls, b, s_lead, mask_lead, one):
    """A mask shared by the complexes and a single track with a sample dim go operator by operator, as they did before a block
    was one call; their shapes are the operators' to judge."""
    from kfold_b200 import confidence
    n, calls = 32, []
    for mod in (M, confidence):
        monkeypatch.setattr(mod, "_check_inference", lambda x: None)
    monkeypatch.setattr(M.F, "pair_block", lambda z, pm, plan, s=None, mask=None, precise=False: calls.append("block") or ((z, s) if s is not None else z))
    monkeypatch.setattr(M.F, "pair_bias", lambda z, *a: torch.zeros(z.shape[0], 2, n, n))
    for name in ("_TriangleMultiplication", "_TriangleAttention", "Transition"):
        monkeypatch.setattr(getattr(M, name), "forward", lambda self, x, *a, **k: calls.append(type(self).__name__) or x)
    monkeypatch.setattr(M.SelfAttentionPairBias, "forward", lambda self, a, s, pb, mask, residual=False: calls.append((tuple(a.shape), tuple(mask.shape))) or a)
    blk = M.PairformerBlock(64, 64, 2, 2) if cls == "PairformerBlock" else confidence.ConfidencePairSingleBlock(64, 64, 2)
    z, s = torch.zeros(b, n, n, 64, dtype=torch.bfloat16), torch.zeros(*s_lead, n, 64, dtype=torch.bfloat16)
    mask = torch.ones(*mask_lead, n, dtype=torch.bool)
    with torch.no_grad():
        zo, so = blk(z, s, torch.ones(b, n, n, dtype=torch.bool), mask)
    assert zo.shape == z.shape and so.shape == s.shape
    assert (calls == ["block"]) is one and (one or (tuple(s.shape), tuple(mask.shape)) in calls)
