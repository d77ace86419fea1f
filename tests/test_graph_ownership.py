"""What a captured call points to stays alive and is used by nothing else for as long as the call lives.

A CUDA graph records addresses.  The CPU tests replace the CUDA objects and look at who holds the memory; the GPU tests replay
graphs whose memory later calls would have taken."""
import contextlib
import gc
import weakref

import pytest
import torch

from helpers import err_stats


# ------------------------------------------------------------------------------------------------ ownership, without a GPU
class _Input:
    """Stands for a CUDA tensor as far as GraphedCall's constructor looks at one."""
    is_cuda, device = True, torch.device("cuda:0")

    def clone(self):
        return _Input()


class _Stream:
    cuda_stream = 7

    def wait_stream(self, other):
        pass

    synchronize = lambda self: None


class _Graph:
    capture_begin = capture_end = lambda self: None


@pytest.fixture()
def fake_cuda(monkeypatch):
    from kfold_b200 import functional as F, graphs
    monkeypatch.setattr(torch.cuda, "CUDAGraph", _Graph)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: _Stream())
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(graphs, "_capture_stream", lambda device: _Stream())
    monkeypatch.setattr(F.L, "raw_stream", lambda index=None: 7)
    F.release_workspaces()
    yield
    F.release_workspaces()


def _call_of(nbytes, seen):
    """A call with a workspace of `nbytes`; `seen` gets a weak reference to the one it was given last."""
    from kfold_b200 import functional as F

    def fn(x):
        seen["ws"] = weakref.ref(F._workspace(torch.device("cpu"), nbytes))
        return x

    return fn


def test_two_live_graphs_own_their_workspaces(fake_cuda):
    from kfold_b200 import functional as F
    from kfold_b200.graphs import GraphedCall
    first, second, third = {}, {}, {}
    a = GraphedCall(_call_of(1000, first), _Input())
    b = GraphedCall(_call_of(1000000, second), _Input())      # needs more: the workspace kept for the stream is replaced
    c = GraphedCall(_call_of(10, third), _Input())            # needs less: fits in any workspace that is still handed out
    F.release_workspaces()
    gc.collect()
    alive = [s["ws"]() for s in (first, second, third)]
    assert all(ws is not None for ws in alive), "a live graph's workspace was freed"
    assert len({ws.data_ptr() for ws in alive}) == 3, "two live graphs share a workspace"
    del alive, a
    gc.collect()
    assert first["ws"]() is None and second["ws"]() is not None, "a workspace outlives its graph"
    del b, c


def test_a_large_stack_workspace_is_given_back(fake_cuda, monkeypatch):
    """The workspace of a stack call above the bound lives as long as the call; a smaller one, and an operator's, is kept."""
    from kfold_b200 import functional as F, modules as M
    sizes = {}

    class Lib:
        kfb_token_stack_workspace_bytes = kfb_atom_stack_workspace_bytes = lambda self, *a: sizes["need"]
        kfb_token_stack_fwd = kfb_atom_stack_fwd = lambda self, *a: 0

    monkeypatch.setattr(F.L, "lib", lambda: Lib())
    monkeypatch.setattr(F.L, "stream_ptr", lambda: 7)
    monkeypatch.setattr(F, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(M, "_check_inference", lambda x: None)
    monkeypatch.setattr(M.F, "window_bias", lambda z, lw, lb, w, eps: torch.zeros(w.shape[0], *z.shape[:-1]))
    monkeypatch.setattr(F, "MOST_KEPT_BYTES", 1 << 20)
    token, atom = M.CachedGlobalTransformerStack(64, 8, 2, 1), M.LocalTransformerStack(64, 64, 16, 2, 1)
    for stack, args in ((token, (torch.zeros(1, 8, 64), torch.zeros(1, 8, 8), torch.zeros(1, 1, 2, 8, 8), torch.ones(1, 8).bool())),
                        (atom, (torch.zeros(1, 64, 64), torch.zeros(1, 64, 64), torch.zeros(1, 2, 32, 128, 16), torch.ones(1, 64).bool()))):
        F.release_workspaces()
        for need, kept in ((1 << 16, True), (1 << 22, False)):
            sizes["need"] = need
            before = dict(F._workspaces)
            with torch.no_grad(), torch.autocast("cpu", dtype=torch.bfloat16):
                stack(*args)
            assert any(ws.numel() >= need for ws in F._workspaces.values()) is kept
            assert kept or F._workspaces == before


def test_a_graph_holds_what_modules_replace(fake_cuda):
    """Packed weights, converted biases and plans that the captured call was handed, and what the function closes over."""
    from kfold_b200.graphs import GraphedCall
    from kfold_b200.plans import handed_out

    class Plan:
        def __init__(self):
            self.keep = [torch.zeros(8)]

    cache = {"bias": torch.zeros(4), "packed": {"w": torch.zeros(2)}, "plan": Plan(), "pair": (torch.zeros(1), None)}
    closed_over = torch.zeros(3)
    refs = [weakref.ref(t) for t in (cache["bias"], cache["packed"]["w"], cache["plan"].keep[0], cache["pair"][0], closed_over)]

    def build():
        bias_of_complex = closed_over

        def fn(x):
            assert bias_of_complex.numel() == 3
            for v in cache.values():
                handed_out(v)
            return x

        return GraphedCall(fn, _Input())

    g = build()
    cache.clear()
    del closed_over
    gc.collect()
    # `closed_over` is a cell of build() too: drop the function itself
    del build
    gc.collect()
    assert all(r() is not None for r in refs)
    del g
    gc.collect()
    assert all(r() is None for r in refs)


def test_modules_record_what_they_hand_out():
    """Every cache of the modules goes through plans.handed_out: a packed weight, a projection, a bias, a plan."""
    from kfold_b200 import modules as M
    from kfold_b200.plans import HandedOut
    dev = torch.device("cpu")
    stack = M.CachedGlobalTransformerStack(64, 32, 2, 1)
    bias = torch.zeros(1, 1, 2, 8, 8)
    proj = M._ProjectionCache()
    with torch.no_grad(), HandedOut() as h:
        plan = stack._plan_for(dev, False)
        prepared = stack._prepared_bias(bias)
        w = proj.get(stack.blocks[0].attention.linear_q, dev, False)
        pk = stack.blocks[0].attention._apb_packed(dev)
    kept = {t.data_ptr() for t in h.tensors()}
    assert {t.data_ptr() for t in plan.keep if t is not None} <= kept
    assert prepared.data_ptr() in kept and w.data_ptr() in kept and pk["w_proj"].data_ptr() in kept


def test_a_capture_without_memory_is_tried_again(fake_cuda, monkeypatch):
    """An allocation that fails under capture: the failed capture is ended, the cache emptied outside of it, the call captured
    once more; a second failure, and any other error, is the caller's."""
    from kfold_b200.graphs import GraphedCall
    events = []

    class Graph:
        def __init__(self):
            self.n = sum(e[0] == "begin" for e in events)

        def capture_begin(self):
            events.append(("begin", self.n))

        def capture_end(self):
            events.append(("end", self.n))
            if self.n == bad_end:
                raise RuntimeError("capture invalidated")

    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: events.append(("empty",)))

    def failing(times, error):
        def fn(x):
            if events and events[-1][0] == "begin" and sum(e[0] == "begin" for e in events) <= times:
                raise error
            return x
        return fn

    for bad_end in (None, 0):
        events.clear()
        g = GraphedCall(failing(1, torch.OutOfMemoryError("no memory")), _Input())
        assert events == [("begin", 0), ("end", 0), ("empty",), ("begin", 1), ("end", 1)] and g._graph.n == 1
    bad_end = None
    events.clear()
    with pytest.raises(torch.OutOfMemoryError):
        GraphedCall(failing(2, torch.OutOfMemoryError("no memory")), _Input())
    assert events[-1] == ("end", 1)
    events.clear()
    with pytest.raises(ValueError):
        GraphedCall(failing(1, ValueError("the call's own")), _Input())
    assert events == [("begin", 0), ("end", 0)]


# ------------------------------------------------------------------------------------------------ replays, on a GPU
def _token_call(dev, l, seed):
    from kfold_b200 import modules as M
    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=dev)
    with torch.device(dev):
        stack = M.CachedGlobalTransformerStack(256, 384, 8, 2)
    a, s, bias = rnd(1, 2, l, 256), rnd(1, 1, l, 384), rnd(1, 1, 2, 8, l, l)
    mask = torch.ones(1, 1, l, dtype=torch.bool, device=dev)

    def fn(a_, s_):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return stack(a_, s_, bias, mask)

    return fn, a, s


@pytest.mark.gpu
def test_graphs_of_growing_complexes_stay_valid():
    """A graph for a small complex, then one for a larger one, then calls of a third network on the capture stream: the replays
    of the first two give their eager results to the bit, also after the kept workspaces were dropped."""
    from kfold_b200 import _lib as L, functional as F
    from kfold_b200.graphs import GraphedCall, _capture_stream
    dev = torch.device("cuda:0")
    with torch.no_grad():
        built = []
        for l, seed in ((40, 1), (333, 2)):
            fn, a, s = _token_call(dev, l, seed)
            built.append((GraphedCall(fn, a, s), a, s, fn(a, s).clone()))
        F.release_workspaces()
        fn, a, s = _token_call(dev, 200, 3)
        with torch.cuda.stream(_capture_stream(dev)):     # allocations and kernels on the stream that the captures ran on
            for _ in range(3):
                fn(a * 100, s)
            junk = [torch.full((1 << 18,), float("nan"), device=dev) for _ in range(64)]
        torch.cuda.synchronize()
        for _ in range(2):
            for graphed, a, s, ref in built:
                assert torch.equal(graphed(a, s), ref)
        del junk
    assert L.device_status() == 0


@pytest.mark.gpu
def test_a_stack_with_a_workspace_of_its_own(monkeypatch):
    """Eager and captured, with nothing kept for the stack: the same result to the bit, and no workspace left behind."""
    from kfold_b200 import _lib as L, functional as F
    from kfold_b200.graphs import GraphedCall
    dev = torch.device("cuda:0")
    with torch.no_grad():
        fn, a, s = _token_call(dev, 77, 9)
        ref = fn(a, s).clone()
        monkeypatch.setattr(F, "MOST_KEPT_BYTES", 0)
        F.release_workspaces()
        assert torch.equal(fn(a, s), ref) and not F._workspaces
        graphed = GraphedCall(fn, a, s)
        junk = [torch.full((1 << 18,), float("nan"), device=dev) for _ in range(32)]
        for _ in range(2):
            assert torch.equal(graphed(a, s), ref)
        del junk
    assert L.device_status() == 0


@pytest.mark.gpu
def test_one_network_two_complexes_both_graphs_live():
    """The window biases and the converted pair bias of the first complex leave the modules' caches when the second is captured."""
    from kfold_b200 import modules as M
    from kfold_b200 import _lib as L
    from kfold_b200.graphs import GraphedCall
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(5)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=dev)
    with torch.no_grad():
        with torch.device(dev):
            stack = M.LocalTransformerStack(128, 128, 16, 4, 2)
        built = []
        for atoms in (64, 96):
            a, s, z = rnd(1, 2, atoms, 128), rnd(1, 1, atoms, 128), rnd(1, 1, atoms // 32, 32, 128, 16)
            mask = torch.ones(1, 1, atoms, dtype=torch.bool, device=dev)

            def fn(a_, s_, z=z, mask=mask):
                with torch.autocast("cuda", dtype=torch.bfloat16):
                    return stack(a_, s_, z, mask)

            built.append((GraphedCall(fn, a, s), a, s, fn(a, s).clone()))
        stack.reset_caches()
        junk = [torch.full((1 << 16,), float("nan"), device=dev) for _ in range(64)]
        for graphed, a, s, ref in built:
            out = graphed(a, s)
            assert torch.equal(out, ref), err_stats(out, ref)
        del junk
    assert L.device_status() == 0


@pytest.mark.gpu
def test_a_capture_beside_a_full_cache():
    """A capture that needs the memory which the allocator has cached, under a limit that the allocator itself enforces."""
    from kfold_b200 import _lib as L
    from kfold_b200.graphs import GraphedCall
    dev = torch.device("cuda:0")
    big = 1 << 30
    gc.collect()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(dev).total_memory
    x = torch.randn(1 << 20, device=dev)

    def fn(t):
        twice = t * 2
        scratch = torch.empty(big, dtype=torch.uint8, device=dev)      # freed to the capture stream's cache by the warm-up
        del scratch
        return twice

    with torch.no_grad():
        try:
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(dev) + 1.5 * big) / total, dev)
            graphed = GraphedCall(fn, x)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0, dev)
        assert torch.equal(graphed(x), x * 2)
        torch.cuda.synchronize()
    assert L.device_status() == 0
