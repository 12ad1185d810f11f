"""The prompt's dense tail in the window: one launch for dense prompts and token slices of longer buffers, plain copies for
everything else (other types, strides and alignments, tensors that need gradients)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _views(x, how):
    """``x`` again, laid out another way."""
    b, h, t, d = x.shape
    if how == "slice":
        buf = torch.full((b, h, t + 9, d), 3.0, dtype=x.dtype, device=DEV)
        buf[:, :, 4 : 4 + t] = x
        return buf[:, :, 4 : 4 + t]
    if how == "transposed":  # [B,T,H,D] as a projection leaves it
        return x.transpose(1, 2).contiguous().transpose(1, 2)
    if how == "misaligned":
        buf = torch.zeros(x.numel() + 3, dtype=x.dtype, device=DEV)
        buf[3:] = x.flatten()
        return buf[3:].view(x.shape)
    return x


@pytest.mark.parametrize("how", ["dense", "slice", "transposed", "misaligned"])
@pytest.mark.parametrize("b,h,t,sinks", [(1, 1, 1, 0), (1, 8, 33, 4), (3, 2, 95, 0), (2, 4, 300, 4), (1, 8, 200, 0), (2, 1, 96, 32)])
def test_window_holds_sinks_and_tail(b, h, t, sinks, how):
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache
    from reskv_b200.synthetic import gaussian

    cfg = ResKVKernelConfig(recent_size=32, group_size=64, kmeans_iterations=1, num_clusters=16)
    key, raw, value = (gaussian(b, h, t, 128, seed=i, device=DEV) for i in range(3))
    kept = min(sinks, t)
    n = max(0, t - 32 - kept) // 64 * 64
    cache = ResKVLayerCache(cfg, sinks)
    packed = "dense" if how == "misaligned" else how  # the packers take no misaligned rows
    keys, values = cache.update(_views(key, how), _views(value, packed), {"raw_keys": _views(raw, packed)})
    for got, x in ((keys, key), (values, value), (cache.raw_keys[:, :, : cache.live], raw)):
        assert torch.equal(got, torch.cat((x[:, :, :kept], x[:, :, kept + n :]), 2))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_other_types_are_copied(dtype):
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache

    x = torch.randn(2, 2, 20, 128, device=DEV).to(dtype)
    cache = ResKVLayerCache(ResKVKernelConfig())
    keys, values = cache.update(x, x + 1, {"raw_keys": x + 2})
    assert torch.equal(keys, x) and torch.equal(values, x + 1) and torch.equal(cache.raw_keys[:, :, :20], x + 2)


def test_gradients_flow_through_the_window_as_before():
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache

    x = torch.randn(1, 2, 20, 128, device=DEV).half().requires_grad_()
    cache = ResKVLayerCache(ResKVKernelConfig())
    keys, _ = cache.update(x, x, {"raw_keys": x})
    keys.float().sum().backward()
    assert torch.equal(x.grad, torch.ones_like(x))
