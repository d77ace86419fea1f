"""CUDA-graph replay of a fixed-shape call.

The sampler of K-Fold calls its token transformer 200 times per prediction with tensors of the same shape
(src/kfold/model/modules/ecsi.py:468-560).  One step of the network is about 240 kernel launches of a few microseconds
each, so for small complexes it is bound by the host that issues them; captured once into a CUDA graph and replayed it is not
(bench.py --sampler-step prints both).  The library is capturable as it is: it allocates nothing, never synchronises, and
every temporary of the Python layer comes from torch's caching allocator, which gives a capture its own pool.
"""
from __future__ import annotations

import gc
import threading

import torch

from . import functional as F
from .plans import HandedOut

_local = threading.local()


def _capture_stream(device: torch.device) -> torch.cuda.Stream:
    """This thread's side stream for warm-up and capture on `device`.  One stream for all captures: memory the allocator has
    cached for it, that of a workspace whose graph is gone included, serves the next capture instead of being allocated anew."""
    streams = _local.__dict__.setdefault("streams", {})
    index = torch.cuda.current_device() if device.index is None else device.index
    if index not in streams:
        streams[index] = torch.cuda.Stream(index)
    return streams[index]


def _capture(fn, inputs):
    graph = torch.cuda.CUDAGraph()
    graph.capture_begin()
    try:
        output = fn(*inputs)
    except BaseException:
        try:
            graph.capture_end()
        except RuntimeError:      # the capture had become invalid: the error that made it so is the one to report
            pass
        raise
    graph.capture_end()
    return graph, output


class GraphedCall:
    """``GraphedCall(fn, *example_inputs)`` captures ``fn(*example_inputs)`` once; ``self(*inputs)`` copies the inputs into
    the captured buffers, replays the graph and returns the captured output tensor(s) (overwritten by the next call).

    ``fn`` must be free of host synchronisation and of data-dependent control flow, and every call must use the shapes,
    dtypes and devices of the example.  Tensors that never change between calls (weights, a cached pair bias, masks) can
    be closed over by ``fn`` instead of being passed as inputs, which saves their copy.

    The stacks keep what they derive from per-complex tensors (the converted token pair bias, the window biases of the atom
    transformers) in caches that already hold their result when the capture runs, so those kernels are NOT part of the
    graph: the pair tensor ``z``, the window pair tensor ``p`` and ``pair_bias`` must be closed over by ``fn``, never passed
    as inputs that later calls replace -- a replay would keep using the bias of the captured tensors.  For a new complex
    build a new GraphedCall; the earlier one stays valid.

    A graph holds addresses, so a GraphedCall owns what lies at them for as long as it lives: ``fn`` and what it closes over, its
    workspaces (from then on no other call is given them) and everything that the modules called keep between calls -- packed
    weights, the converted pair bias, the window biases -- even after a module has replaced it.  What a *parameter* points to is
    not held: weights must not be replaced while the graph is in use.
    """

    def __init__(self, fn, *example_inputs: torch.Tensor, warmup: int = 2):
        if not example_inputs or not all(t.is_cuda for t in example_inputs):
            raise ValueError("GraphedCall needs CUDA tensors as example inputs")
        self._fn = fn
        self._inputs = [t.clone() for t in example_inputs]
        dev = example_inputs[0].device
        with torch.cuda.device(dev), torch.no_grad():
            # Warm-up and capture on one side stream.  torch.cuda.graph() would collect Python garbage and return the
            # allocator's cached blocks to the driver first; with a model of a few hundred parameters in memory that is
            # 0.1 s and more, and every later allocation pays for it again, so the capture is begun and ended directly, and
            # only one that finds no memory is tried again after that.
            current, side = torch.cuda.current_stream(), _capture_stream(dev)
            side.wait_stream(current)
            with torch.cuda.stream(side):          # warm-up outside the capture: weight packing, workspace allocation
                for _ in range(max(warmup, 1)):
                    fn(*self._inputs)
                side.synchronize()
                with HandedOut() as used:
                    try:
                        self._graph, self._output = _capture(fn, self._inputs)
                    except torch.OutOfMemoryError:
                        # the allocator returns no cached block to the driver while a capture is under way: what the calls
                        # before have left in its cache may be the memory that is missing
                        gc.collect()
                        torch.cuda.empty_cache()
                        self._graph, self._output = _capture(fn, self._inputs)
            current.wait_stream(side)
        self._kept, self._streams = used.tensors(), set()
        F.withdraw_workspaces(self._kept)

    def __call__(self, *inputs: torch.Tensor):
        if len(inputs) != len(self._inputs):
            raise ValueError(f"expected {len(self._inputs)} inputs, got {len(inputs)}")
        for dst, src in zip(self._inputs, inputs):
            if dst.shape != src.shape or dst.dtype != src.dtype:
                raise ValueError(f"input {tuple(src.shape)} {src.dtype} does not match the captured {tuple(dst.shape)} {dst.dtype}")
            if dst.data_ptr() != src.data_ptr():
                dst.copy_(src, non_blocking=True)
        stream = torch.cuda.current_stream(self._inputs[0].device)
        if stream.cuda_stream not in self._streams:
            # the kernels of a replay use this memory on a stream that it was not allocated on: it goes back to its own only
            # when the replays that are under way at that time have ended
            for t in self._kept + self._inputs:
                t.record_stream(stream)
            self._streams.add(stream.cuda_stream)
        self._graph.replay()
        return self._output
