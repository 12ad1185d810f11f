"""The native host calls let other Python threads run: a launch that waits because the stream's queue is full, and a verdict
that is dropped while its kernel is still queued, hold no interpreter lock."""

import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BUSY_CYCLES = 1_500_000_000  # 0.8 s of a spinning kernel at 1.9 GHz


class Pulse(threading.Thread):
    """Longest time between two turns of a thread that only sleeps."""

    def __init__(self):
        super().__init__()
        self.done, self.gap = threading.Event(), 0.0

    def run(self):
        last = time.perf_counter()
        while not self.done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            self.gap, last = max(self.gap, now - last), now


def _longest_gap(work):
    """(longest gap of another thread, duration) while ``work`` runs behind a busy stream."""
    torch.cuda.synchronize()
    pulse = Pulse()
    pulse.start()
    start = time.perf_counter()
    torch.cuda._sleep(BUSY_CYCLES)
    try:
        work()
        took = time.perf_counter() - start
    finally:
        pulse.done.set()
        pulse.join()
        torch.cuda.synchronize()
    return pulse.gap, took


def test_a_launch_that_waits_lets_other_threads_run():
    from reskv_b200 import ResKVKernelConfig, attention, compress
    from reskv_b200.synthetic import gaussian, mixture

    cache = compress(mixture(1, 2, 200, seed=1, device=DEV), mixture(1, 2, 200, seed=2, device=DEV),
                     ResKVKernelConfig(num_clusters=8, kmeans_iterations=2))
    q = gaussian(1, 8, 1, 128, seed=3, device=DEV)
    attention(q, cache, position=200)
    gap, took = _longest_gap(lambda: [attention(q, cache, position=200) for _ in range(2000)])  # 4000 launches
    assert took > 0.3, "the queue never filled"
    assert gap < 0.2


def test_a_dropped_verdict_lets_other_threads_run_and_does_not_wait():
    from reskv_b200._extension import load_extension

    ids = torch.zeros((1, 2, 64), dtype=torch.int32, device=DEV)
    ops = load_extension("compression")

    def drop_many():
        for _ in range(20):  # more than are kept
            ticket = ops.take_ids(ids, ids, 4, 4)
            del ticket

    drop_many()
    gap, took = _longest_gap(drop_many)
    assert gap < 0.2 and took < 0.4
    for _ in range(20):
        assert ops.take_ids(ids, ids, 4, 4)[2]()
    assert not ops.take_ids(ids + 4, ids, 4, 4)[2]()


def test_calls_of_several_threads_give_the_bits_of_calls_in_turn():
    from reskv_b200 import ResKVKernelConfig, attention, compress
    from reskv_b200.cache import ResKVLayerCache
    from reskv_b200.compression import cluster
    from reskv_b200.synthetic import gaussian, mixture

    cfg = ResKVKernelConfig(sparsity=0.75, num_clusters=8, kmeans_iterations=2, max_clusters=16)

    def request(seed):
        key, value = (mixture(1, 2, 300, seed=seed + i, device=DEV) for i in (0, 1))
        given = compress(key, value, cfg, clustering=(cluster(key, 8, 2), cluster(value, 8, 2, value=True)))
        layer, out = ResKVLayerCache(cfg, 0), []
        layer.update(key, value, {"raw_keys": key})
        for step in range(80):  # a decode group is compressed on the way
            token, q = gaussian(1, 2, 1, 128, seed=seed + step, device=DEV), gaussian(1, 8, 1, 128, seed=step, device=DEV)
            position = layer.length
            keys, values = layer.update(token, token, {"raw_keys": token})
            out.append(attention(q, layer.compressed, position=position, recent=(q, keys, values)))
        return torch.cat([*out, attention(q, given, position=300)])

    want = [request(100 * i) for i in range(6)]
    got = [None] * 6

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = request(100 * i)
            torch.cuda.current_stream().synchronize()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(g is not None and torch.equal(g, w) for g, w in zip(got, want))
