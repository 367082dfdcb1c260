"""Recording of CUDA graphs."""
import gc
import threading
import time

import pytest
import torch

from eredu_b200.utils.capture import captured


@pytest.mark.parametrize("on, fails", [(True, False), (True, True), (False, False)])
def test_no_collection_inside_a_recording(monkeypatch, on, fails):
    seen = []

    class Recording:
        def __init__(self, graph):
            seen.append(graph)

        def __enter__(self):
            seen.append(gc.isenabled())

        def __exit__(self, *error):
            seen.append(gc.isenabled())

    monkeypatch.setattr(torch.cuda, "graph", Recording)
    before = gc.isenabled()
    try:
        (gc.enable if on else gc.disable)()
        try:
            with captured("a graph"):
                seen.append(gc.isenabled())
                if fails:
                    raise ValueError
        except ValueError:
            assert fails
        assert seen == ["a graph", False, False, False] and gc.isenabled() == on
    finally:
        (gc.enable if before else gc.disable)()


def test_threads_record_one_after_the_other(monkeypatch):
    """The first to end its recording must not turn collections on under the second."""
    inside, seen = [], []

    class Recording:
        def __init__(self, graph):
            self.graph = graph

        def __enter__(self):
            inside.append(self.graph)

        def __exit__(self, *error):
            inside.remove(self.graph)

    monkeypatch.setattr(torch.cuda, "graph", Recording)
    first_is_in, second_has_begun = threading.Event(), threading.Event()

    def first():
        with captured("first"):
            first_is_in.set()
            second_has_begun.wait(10)
            time.sleep(0.05)            # the second thread is at its recording by now
            seen.append((list(inside), gc.isenabled()))

    def second():
        first_is_in.wait(10)
        second_has_begun.set()
        with captured("second"):
            time.sleep(0.1)             # beyond the end of the first
            seen.append((list(inside), gc.isenabled()))

    before = gc.isenabled()
    gc.enable()
    try:
        threads = [threading.Thread(target=f) for f in (first, second)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(20)
        assert seen == [(["first"], False), (["second"], False)] and gc.isenabled()
    finally:
        (gc.enable if before else gc.disable)()
