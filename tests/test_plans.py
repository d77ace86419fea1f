"""What a module keeps between calls: when its packed weights are stale, without a GPU."""
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
