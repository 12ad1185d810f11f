"""The native host path of ``attention``: a dense window read in place (the leading tokens of a longer buffer, one
buffer per side, evenly spaced units) gives the bits of its dense copy; layouts that cannot be addressed are copied."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,h", [(1, 1), (1, 3), (3, 1), (2, 4)])
@pytest.mark.parametrize("tr,cap", [(1, 1), (1, 96), (95, 96), (33, 40)])
def test_window_views_equal_their_dense_copies(b, h, tr, cap):
    from reskv_b200 import ResKVKernelConfig, attention, compress
    from reskv_b200.synthetic import gaussian, mixture

    t = 200
    cfg = ResKVKernelConfig(sparsity=0.5, num_clusters=8, kmeans_iterations=2)
    cache = compress(mixture(b, h, t, seed=1, device=DEV), mixture(b, h, t, seed=2, device=DEV), cfg)
    q, qr = (gaussian(b, 4 * h, 1, 128, seed=s, device=DEV) for s in (3, 4))
    buf = torch.full((2, b, h, cap, 128), float("nan"), dtype=torch.float16, device=DEV)  # surroundings must not be read
    buf[:, :, :, :tr] = gaussian(2, b, h, tr, 128, seed=5, device=DEV)
    k, v = buf[0].narrow(2, 0, tr), buf[1].narrow(2, 0, tr)
    want = attention(q, cache, position=t + tr, recent=(qr, k.contiguous(), v.contiguous()))
    assert want.isfinite().all()
    got = attention(q, cache, position=t + tr, recent=(qr, k, v))
    assert torch.equal(got, want)
    # keys and values with different strides, and heads stored behind tokens
    swapped = k.transpose(1, 2).contiguous().transpose(1, 2)
    assert torch.equal(attention(q, cache, position=t + tr, recent=(qr, swapped, v)), want)


def test_argument_errors_keep_their_messages():
    from reskv_b200 import ResKVKernelConfig, attention, compress
    from reskv_b200.synthetic import gaussian, mixture

    cfg = ResKVKernelConfig(num_clusters=4, kmeans_iterations=1)
    cache = compress(mixture(1, 2, 64, seed=1, device=DEV), mixture(1, 2, 64, seed=2, device=DEV), cfg)
    q = gaussian(1, 8, 1, 128, seed=3, device=DEV)
    for query, message in ((q.cpu(), "FP16 CUDA"), (q.float(), "FP16 CUDA"), (q[:, :6], "ratios"), (q.repeat(2, 1, 1, 1), "batch")):
        with pytest.raises(ValueError, match=message):
            attention(query, cache, position=64)
    with pytest.raises(ValueError, match="precedes"):
        attention(q, cache, position=62)
    with pytest.raises(ValueError, match="inv_freq"):
        attention(q, cache, position=64, inv_freq=torch.ones(32, device=DEV))
    k = torch.zeros(1, 2, 5, 128, device=DEV)
    with pytest.raises(ValueError, match="FP16 on the query device"):
        attention(q, cache, position=64, recent=(q, k, k))
    with pytest.raises(ValueError, match="shapes"):
        attention(q, cache, position=64, recent=(q, k.half(), k[:, :, :4].half()))
