"""No garbage collection inside the capture of a decode step."""

import gc
import threading

import pytest
import torch


class Cycle:
    def __init__(self, note):
        self.me, self.note = self, note

    def __del__(self):
        self.note()


@pytest.fixture
def eager_collector():
    """The collector runs at every other allocation."""
    thresholds, was_on = gc.get_threshold(), gc.isenabled()
    gc.collect()
    gc.enable()
    gc.set_threshold(1, 1, 1)
    yield
    gc.set_threshold(*thresholds)
    gc.enable() if was_on else gc.disable()


def test_the_collector_is_held_while_any_thread_is_inside(eager_collector):
    from reskv_b200.models.llama import _collector_held

    notes, entered, leave = [], threading.Event(), threading.Event()

    def other():
        with _collector_held():
            entered.set()
            leave.wait(10)

    thread = threading.Thread(target=other)
    with _collector_held():
        thread.start()
        assert entered.wait(10)
    Cycle(lambda: notes.append(1))
    keep = [[] for _ in range(100)]  # the other thread is still inside
    assert not notes and not gc.isenabled()
    leave.set()
    thread.join()
    assert gc.isenabled()
    keep += [[] for _ in range(100)]
    assert notes
    gc.disable()  # off before: stays off
    with pytest.raises(ZeroDivisionError), _collector_held():
        1 / 0
    assert not gc.isenabled()


@pytest.mark.gpu
def test_no_finaliser_runs_inside_the_capture(eager_collector, monkeypatch):
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.models import LlamaShape, ResKVLlama

    shape = LlamaShape(hidden=256, layers=2, heads=8, kv_heads=2, ffn=512, vocab=320)
    model = ResKVLlama(shape, ResKVKernelConfig(num_clusters=8, kmeans_iterations=2), seed=3)
    ids = torch.randint(0, 320, (1, 200), device="cuda")
    model.prefill(ids, reserve=8)
    model.begin_graph_decode(1)
    body, capturing = model._step_body, []

    def littering_body(tok):
        for _ in range(20):
            Cycle(lambda: capturing.append(torch.cuda.is_current_stream_capturing()))
        return body(tok)

    monkeypatch.setattr(model, "_step_body", littering_body)
    for token in range(3):
        model.decode_graph(torch.tensor([token], device="cuda"))
    monkeypatch.undo()
    gc.collect()
    torch.cuda.synchronize()
    assert capturing and not any(capturing)
