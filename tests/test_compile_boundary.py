"""torch.compile stops at every method that calls the native library: ctypes calls and addresses are nothing it can trace."""
import inspect

import pytest
import torch
from torch import nn

from kfold_b200 import confidence, modules, trunk

ENTRIES = sorted({(cls.__qualname__, name, fn) for mod in (modules, confidence, trunk)
                  for cls in vars(mod).values() if inspect.isclass(cls) and issubclass(cls, nn.Module) and cls.__module__ == mod.__name__
                  for name, fn in vars(cls).items()
                  if inspect.isfunction(fn) and "_check_inference(" in inspect.getsource(inspect.unwrap(fn))}, key=lambda e: e[:2])


def test_the_entries_are_found():
    assert {"TriangularBlock", "PairformerBlock", "ConfidencePairSingleBlock", "CachedGlobalTransformerStack"} <= {e[0] for e in ENTRIES}


def test_the_token_pair_bias_is_not_traced():
    assert modules._token_pair_bias._torchdynamo_disable


@pytest.mark.parametrize("cls,name,fn", ENTRIES, ids=lambda v: v if isinstance(v, str) else "")
def test_native_entries_are_not_traced(cls, name, fn):
    assert getattr(fn, "_torchdynamo_disable", False), f"{cls}.{name} would be traced by torch.compile"


def test_a_compiled_triangular_block_runs_its_native_call_untraced(monkeypatch):
    """The call of a compiled block reaches the native call as it is written, with tensors that have addresses."""
    seen = []

    def pair_block(z, pair_mask, plan, precise=False):
        seen.append((torch.compiler.is_compiling(), z.data_ptr(), plan))
        return z

    monkeypatch.setattr(modules, "_check_inference", lambda x: None)
    monkeypatch.setattr(modules.F, "pair_block", pair_block)
    blk = modules.TriangularBlock(64)
    z, mask = torch.zeros(1, 32, 32, 64, dtype=torch.bfloat16), torch.ones(1, 32, 32, dtype=torch.bool)
    graphs = []

    def backend(gm, inputs):
        graphs.append(gm)
        return gm.forward

    with torch.no_grad():
        out = torch.compile(blk, backend=backend)(z, mask)
    assert out.data_ptr() == z.data_ptr()
    assert seen == [(False, z.data_ptr(), blk._plan)] and not graphs
