"""What a module keeps between calls: its packed weights, and a cheap way to see whether they are still those of its parameters.

A forward call has to notice a parameter that was replaced, moved or changed in place (``load_state_dict``, ``.to(device)``, an
optimiser step), but walking ``module.parameters()`` of a 24-block stack costs more host time than launching its kernels does.
`ParamState` remembers where the parameters live (the modules' own dictionaries) and reads their addresses and versions from
there: about 0.15 us per parameter.
"""
from __future__ import annotations

import threading
from itertools import chain

import torch
from torch.nn.modules import module as _nn_module

__all__ = ["ParamState", "StandsFor", "NativeCall", "Unshared", "handed_out", "HandedOut"]

_recording = threading.local()


def handed_out(kept):
    """Every place that keeps device memory between calls (workspaces, packed weights, what is derived from the tensors of one
    complex) passes what it gives to a call through here, so that a CUDA graph can hold what its kernels point to."""
    seen = getattr(_recording, "seen", None)
    if seen is not None:
        seen[id(kept)] = kept
    return kept


class HandedOut:
    """``with HandedOut() as h:`` collects in `h.kept` everything that calls of this thread were handed meanwhile."""

    def __init__(self):
        self.kept = {}

    def __enter__(self):
        self._outer = getattr(_recording, "seen", None)
        _recording.seen = self.kept
        return self

    def __exit__(self, *exc):
        _recording.seen = self._outer
        if self._outer is not None:
            self._outer.update(self.kept)
        return False

    def tensors(self) -> list:
        """The tensors among it: themselves, the values of a dict or a sequence, the `keep` list of a plan."""
        out, todo = {}, list(self.kept.values())
        while todo:
            t = todo.pop()
            if isinstance(t, torch.Tensor):
                out[id(t)] = t
            elif isinstance(t, dict):
                todo += t.values()
            elif isinstance(t, (list, tuple)):
                todo += t
            else:
                todo += getattr(t, "keep", ())
        return list(out.values())


class StandsFor:
    """The submodules whose `forward` a native call of the whole block or stack stands for.

    The native call reads their weights and never calls them.  That is the same thing only while they are what the framework
    made them: of exactly that class, without a `forward` of their own and without forward hooks, which would not fire.
    Given as `module, class` or `module, (class, {child: ...})` pairs, children being looked at below a plain module only; a child
    whose name ends in `*` is read and not called without the native call either, so that its class is all that matters.
    `norms()`, asked when all are plain, lists the LayerNorms for which the call has one epsilon: they have to agree on it."""

    __slots__ = ("_submodules", "_classes", "_called", "_norms")

    def __init__(self, *pairs, norms):
        self._submodules, self._classes, self._called, todo = [], [], [], list(pairs)
        while todo:
            m, cls, *read_only = todo.pop()
            children = {}
            if isinstance(cls, tuple):
                cls, children = cls
            self._submodules.append(m)
            self._classes.append(cls)
            if type(m) is cls:
                if not any(read_only):
                    self._called.append(m.__dict__)
                todo += [(m._modules.get(name.rstrip("*")), sub, name[-1] == "*") for name, sub in children.items()]
        self._norms = norms() if self.plain() else []

    def plain(self) -> bool:
        """Whether every submodule is of the expected class itself."""
        return list(map(type, self._submodules)) == self._classes and not any(["forward" in d for d in self._called])

    def eps(self):
        """The epsilon of the LayerNorms, None where they differ."""
        seen = {n.eps for n in self._norms}
        return seen.pop() if len(seen) == 1 else None

    def holds(self):
        """The epsilon of the native call if it may be made -- plain submodules, nobody listens to them, one epsilon -- else None."""
        if _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks or list(map(type, self._submodules)) != self._classes:
            return None
        if any([d["_forward_hooks"] or d["_forward_pre_hooks"] or "forward" in d for d in self._called]):
            return None
        return self.eps()


class Unshared:
    """Mixin, before nn.Module, of a module that keeps things which are of use to it alone (addresses, views of its dictionaries):
    `_unshared` names the attributes that a copy and a saved file go without.  The class has defaults for them."""

    _unshared = ()

    def __getstate__(self):
        return {k: v for k, v in super().__getstate__().items() if k not in self._unshared}


class NativeCall(Unshared):
    """Mixin of a block or stack that runs as one native call: `_plan_for(*key)` gives the plan of that call, or None where the
    submodules have to be called one by one.  The class provides `_stands_for()` and `_make_plan(*key)`; a plan has
    `fits(*key)` and `set_eps(eps)`, for an epsilon is no parameter and may be changed between calls."""

    _plan = None
    _unshared = ("_plan",)

    def _plan_for(self, *key):
        plan = self._plan
        if plan is None or not plan.fits(*key):
            stands = self._stands_for()
            eps = stands.holds()
            plan = self._plan = None if eps is None else self._make_plan(*key)
            if plan is not None:
                plan.stands = stands      # the submodules are still these for as long as the plan fits
        else:
            eps = plan.stands.holds()
        if eps is None:
            return None
        plan.set_eps(eps)
        return handed_out(plan)


def _version(p):
    try:
        return p._version
    except RuntimeError:      # inference tensors carry no version counter
        return None


_data_ptr = torch.Tensor.data_ptr


class ParamState:
    """Addresses and in-place versions of every parameter below `modules`, as they were when this was made."""

    __slots__ = ("_parameters", "_modules", "_empty", "_children", "_seen")

    def __init__(self, *modules):
        # views of the modules' own dictionaries: a parameter or a submodule that is added where there was none shows in them too
        dicts = [(m._parameters, m._modules) for root in modules for m in root.modules()]
        self._parameters, self._modules = [p.values() for p, _ in dicts if p], [c.values() for _, c in dicts if c]
        self._empty = [d for pair in dicts for d in pair if not d]
        self._children, self._seen = list(chain.from_iterable(self._modules)), self._read()

    def _read(self):
        ps = [p for p in chain.from_iterable(self._parameters) if p is not None]
        try:
            return list(map(_data_ptr, ps)), [p._version for p in ps]
        except RuntimeError:
            return list(map(_data_ptr, ps)), [_version(p) for p in ps]

    def current(self) -> bool:
        """Whether nothing changed since."""
        return self._read() == self._seen and not any(self._empty) and list(chain.from_iterable(self._modules)) == self._children
