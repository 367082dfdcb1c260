"""Recording of CUDA graphs."""
from __future__ import annotations

import contextlib
import gc
import threading

import torch

_recording = threading.RLock()


@contextlib.contextmanager
def captured(graph):
    """``torch.cuda.graph(graph)`` without garbage collections in between. A collection may find an engine that was dropped while part of
    a reference cycle; releasing its graphs is a call that no stream of the process may see while one of them is recording, and the
    recording is lost (launches return cudaErrorStreamCaptureInvalidated). Collections are a switch of the process, and torch collects and
    synchronises when it begins a recording: threads record one after the other."""
    with _recording:
        collecting = gc.isenabled()
        gc.disable()
        try:
            with torch.cuda.graph(graph):
                yield
        finally:
            if collecting:
                gc.enable()
