"""Stream capture without the garbage collector.

An engine that is no longer referenced keeps its CUDA graphs in reference cycles until the collector runs. If that happens
in the middle of another engine's capture, the destruction of the old graphs invalidates the capture.
"""
from __future__ import annotations

import contextlib
import gc
import threading

import torch

_LOCK = threading.Lock()
_HOLDERS = 0
_WAS_ON = False


@contextlib.contextmanager
def no_collection():
    """Keeps the collector off while any thread is inside; the last one out restores what the first one found. (Collecting
    beforehand instead costs 9 to 68 ms per engine and does not keep a collection from starting inside.)"""
    global _HOLDERS, _WAS_ON
    with _LOCK:
        if _HOLDERS == 0:
            _WAS_ON = gc.isenabled()
            gc.disable()
        _HOLDERS += 1
    try:
        yield
    finally:
        with _LOCK:
            _HOLDERS -= 1
            if _HOLDERS == 0 and _WAS_ON:
                gc.enable()


@contextlib.contextmanager
def graph(g: torch.cuda.CUDAGraph):
    """`torch.cuda.graph(g)` with the collector off."""
    with no_collection(), torch.cuda.graph(g):
        yield
