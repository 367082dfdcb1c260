"""Recording of CUDA graphs."""
import gc

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
