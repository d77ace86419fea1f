"""What a module keeps between calls: when its packed weights are stale, without a GPU."""
import copy
import io

import pytest
import torch
from torch import nn

from kfold_b200 import modules as M
from kfold_b200.plans import ParamState


def _in_place(m):
    with torch.no_grad():
        m.linear_out.weight.mul_(2.0)


def _replaced(m):
    m.linear_out.weight = nn.Parameter(torch.zeros_like(m.linear_out.weight))


def _added_parameter(m):
    m.linear_out.bias = nn.Parameter(torch.zeros(m.linear_out.weight.shape[0]))


def _removed_parameter(m):
    m.layernorm.bias = None


def _replaced_module(m):
    m.layernorm = M.LayerNorm(64)


def _added_module(m):
    m.linear_out.adapter = M.LinearNoBias(64, 8)


def _loaded(m):
    m.load_state_dict({k: v.clone() for k, v in m.state_dict().items()})


@pytest.mark.parametrize("change", [_in_place, _replaced, _added_parameter, _removed_parameter, _replaced_module, _added_module, _loaded])
def test_every_change_of_the_weights_is_noticed(change):
    m = M.Transition(64, 2)
    state = ParamState(m)
    assert state.current() and state.current()
    change(m)
    assert not state.current()
    assert ParamState(m).current()


# ------------------------------------------------------------------------------------------------ when the one native call is made
DEV = torch.device("cpu")


def _owners():
    from kfold_b200.confidence import ConfidencePairSingleBlock
    pair = (DEV, torch.bfloat16, False)
    return {
        "TriangularBlock": (M.TriangularBlock(64), pair, ["tri_mul_out", "tri_mul_in", "transition_z"]),
        "PairformerBlock": (M.PairformerBlock(64, 64, 2, 2), pair,
                            ["tri_mul_out", "tri_att_start", "tri_att_end", "transition_z", "attention", "transition"]),
        "ConfidencePairSingleBlock": (ConfidencePairSingleBlock(64, 64, 2), pair,
                                      ["pair_block", "pair_block.tri_mul_in", "pair_block.transition_z", "attention", "transition"]),
        "CachedGlobalTransformerStack": (M.CachedGlobalTransformerStack(64, 32, 2, 2), (DEV, False),
                                         ["blocks.1", "blocks.0.attention", "blocks.1.transition", "blocks.1.attention.adaln_a"]),
        "LocalTransformerStack": (M.LocalTransformerStack(64, 64, 16, 2, 2), (DEV, False), ["blocks.0.transition", "blocks.1.attention"]),
    }


PATHS = [(name, path) for name, (_, _, paths) in _owners().items() for path in paths]


@pytest.mark.parametrize("name,path", PATHS)
def test_submodules_that_are_hooked_or_replaced_are_called(name, path):
    """The native call of a block or stack is made only while its submodules are what it stands for."""
    owner, key, _ = _owners()[name]
    sub = owner.get_submodule(path)
    parent, _, leaf = path.rpartition(".")
    parent = owner.get_submodule(parent)
    read_only = path.endswith("adaln_a")      # its weights are read, it is not called in either case
    with torch.no_grad():
        plan = owner._plan_for(*key)
        assert plan is not None and owner._plan_for(*key) is plan
        for register in (sub.register_forward_hook, sub.register_forward_pre_hook):
            handle = register(lambda *a: None)
            assert (owner._plan_for(*key) is None) is not read_only
            handle.remove()
            assert owner._plan_for(*key) is plan
        everywhere = nn.modules.module.register_module_forward_hook(lambda *a: None)
        assert owner._plan_for(*key) is None
        everywhere.remove()
        sub.forward = lambda *a, **k: a[0]
        assert (owner._plan_for(*key) is None) is not read_only
        del sub.forward
        assert owner._plan_for(*key) is plan
        patched = type("Patched", (type(sub),), {"forward": lambda self, x, *a, **k: x})
        subclassed = patched.__new__(patched)
        subclassed.__dict__.update(sub.__dict__)      # the same parameters under another forward
        for new in (subclassed, nn.Identity()):
            setattr(parent, leaf, new)
            assert owner._plan_for(*key) is None
        setattr(parent, leaf, sub)
        assert owner._plan_for(*key) is not None


NORMS = {"TriangularBlock": ["tri_mul_out.layernorm_in", "tri_mul_in.layernorm_in", "transition_z.layernorm"],
         "PairformerBlock": ["tri_mul_out.layernorm_in", "tri_mul_in.layernorm_in", "tri_att_start.layer_norm", "tri_att_end.layer_norm",
                             "transition_z.layernorm", "layernorm_z", "attention.layernorm_a", "transition.layernorm"],
         "ConfidencePairSingleBlock": ["pair_block.tri_mul_out.layernorm_in", "pair_block.tri_mul_in.layernorm_in",
                                       "pair_block.transition_z.layernorm", "layernorm_z", "attention.layernorm_a", "transition.layernorm"],
         "CachedGlobalTransformerStack": [f"blocks.{i}.{m}.layernorm_s" for i in range(2) for m in ("attention.adaln_a", "transition.adaln")],
         "LocalTransformerStack": [f"blocks.{i}.{m}.layernorm_s" for i in range(2)
                                   for m in ("attention.adaln_a_q", "attention.adaln_a_k", "transition.adaln")]}


@pytest.mark.parametrize("name", sorted(NORMS))
def test_one_epsilon_per_native_call(name):
    """A native call has one epsilon for all its LayerNorms: it is made where they agree, with the value they have at the time."""
    owner, key, _ = _owners()[name]
    eps = lambda plan: (plan.struct if hasattr(plan, "struct") else plan.cond).eps
    with torch.no_grad():
        assert eps(owner._plan_for(*key)) == pytest.approx(1e-5)
        for path in NORMS[name]:
            norm = owner.get_submodule(path)
            norm.eps = 1e-3
            assert owner._plan_for(*key) is None, f"{path}: another epsilon than the others'"
            norm.eps = 1e-5
        for path in NORMS[name]:
            owner.get_submodule(path).eps = 1e-3
        assert eps(owner._plan_for(*key)) == pytest.approx(1e-3)


@pytest.mark.parametrize("l,pitch", [(16, 16), (16, 24), (20, 24), (20, 20)])
def test_a_bias_for_blocks_called_one_by_one_is_converted_once(l, pitch):
    """Each block's bias is contiguous, so that no block copies it again, and it is kept for the next call."""
    stack = M.CachedGlobalTransformerStack(64, 32, 2, 3)
    bias = torch.randn(2, 1, 3, 2, l, pitch)[..., :l]
    pb = stack._prepared_bias(bias, per_block=True)
    assert all(pb[i].is_contiguous() for i in range(3)) and stack._prepared_bias(bias, per_block=True) is pb
    assert torch.equal(pb.float(), bias.movedim(-4, 0).bfloat16().float())
    assert stack._prepared_bias(bias).stride(-2) % 8 == 0      # the stack's own form


@pytest.mark.parametrize("name", sorted(_owners()))
def test_a_module_that_has_run_can_be_copied_and_saved(name):
    """What a module keeps for its native calls (addresses among it) stays with it: a copy, or what is loaded from a file, makes
    its own, from its own weights."""
    owner, key, _ = _owners()[name]
    with torch.no_grad():
        plan = owner._plan_for(*key)
        buf = io.BytesIO()
        torch.save(owner, buf)
        buf.seek(0)
        for other in (copy.deepcopy(owner), torch.load(buf, weights_only=False)):
            made = other._plan_for(*key)
            assert made is not None and made is not plan and owner._plan_for(*key) is plan
            mine = {t.data_ptr() for t in plan.keep if t is not None}
            assert not mine & {t.data_ptr() for t in made.keep if t is not None}
            next(other.parameters()).zero_()
            assert other._plan_for(*key) is not made and owner._plan_for(*key) is plan


def test_a_copy_knows_no_complex_by_its_address(monkeypatch):
    """The bias that a stack has converted is kept by the address of its source, which it holds; a copy must not keep the address
    alone."""
    monkeypatch.setattr(M.F, "window_bias", lambda z, lw, lb, w, eps: torch.randn(w.shape[0], *z.shape[:-1]))
    token, atom = M.CachedGlobalTransformerStack(64, 32, 2, 2), M.LocalTransformerStack(64, 64, 16, 2, 2)
    bias, z = torch.randn(1, 2, 2, 8, 8), torch.randn(1, 2, 32, 128, 16)
    first, windows = token._prepared_bias(bias), atom._window_biases(z, torch.bfloat16)
    t2, a2 = copy.deepcopy(token), copy.deepcopy(atom)
    assert t2._bias_key is None and a2._bias_all_key is None
    assert token._bias_src is bias and atom._window_biases(z, torch.bfloat16) is windows and first.shape == (2, 1, 2, 8, 8)
