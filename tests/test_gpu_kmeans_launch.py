"""The one launch that makes all Lloyd iterations: captured in a graph, several at once on streams of their own (every one
wants all SMs and its CTAs wait for one another), and against one iteration per call by the kernel of another form."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _sides(b, h, t, seed):
    from reskv_b200.synthetic import mixture

    return [mixture(b, h, t, seed=seed + i, device=DEV) for i in range(2)]


def _pair(sides, count, iterations):
    from reskv_b200._extension import load_extension

    return [x for side in load_extension("compression").kmeans_pair(*sides, count, iterations) for x in side]


# one CTA per unit, several CTAs per unit, several units per CTA, two segments of a unit in a CTA
@pytest.mark.parametrize("b,h,t", [(8, 8, 2000), (1, 8, 8128), (40, 8, 130), (16, 8, 3000), (1, 1, 20000)])
@pytest.mark.parametrize("iterations", [1, 2, 5])
def test_replay_of_a_captured_call(b, h, t, iterations):
    sides = _sides(b, h, t, 1)
    want = _pair(sides, 32, iterations)
    side_stream = torch.cuda.Stream()
    side_stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side_stream):
        _pair(sides, 32, iterations)
    torch.cuda.current_stream().wait_stream(side_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _pair(sides, 32, iterations)
    for _ in range(2):
        for x in got:
            x.zero_()
        graph.replay()
        assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_calls_in_flight_together():
    jobs = [_sides(b, 8, t, 10 * i) for i, (b, t) in enumerate([(8, 2000), (1, 8128), (8, 2000), (16, 1000)])]
    want = [_pair(sides, 32, 10) for sides in jobs]
    streams = [torch.cuda.Stream() for _ in jobs]
    torch.cuda.synchronize()
    got = []
    for _ in range(5):
        for sides, stream in zip(jobs, streams):
            with torch.cuda.stream(stream):
                got.append(_pair(sides, 32, 10))
    torch.cuda.synchronize()
    for i, result in enumerate(got):
        assert all(torch.equal(x, y) for x, y in zip(result, want[i % len(jobs)]))


@pytest.mark.parametrize("b,h,t", [(2, 8, 2000), (1, 8, 8128), (40, 8, 130)])
def test_iterations_agree_with_the_other_form(b, h, t):
    """Centres within one FP16 unit in the last place of the mma.sync form's, ids equal where no token lies between two."""
    from reskv_b200.compression import cluster

    for value, x in enumerate(_sides(b, h, t, 5)):
        for iterations in (2, 3):
            cen, ids = cluster(x, 32, iterations, value=bool(value))
            want_cen, want_ids = cluster(x, 32, iterations, value=bool(value), warp_mma=True)
            assert (ids != want_ids).float().mean().item() < 1e-3
            bits = lambda c: c.view(torch.int16).int()
            same_sign = torch.signbit(cen) == torch.signbit(want_cen)
            assert ((bits(cen) - bits(want_cen)).abs()[same_sign] <= 1).float().mean().item() > 0.999
