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


def test_tangents_flow_through_the_window_as_before():
    import torch.autograd.forward_ad as fw
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache

    x, t = (torch.randn(1, 2, 20, 128, device=DEV).half() for _ in range(2))
    cache = ResKVLayerCache(ResKVKernelConfig())
    with fw.dual_level():
        dual = fw.make_dual(x, t)
        for got in cache.update(dual, dual, {"raw_keys": dual}):
            primal, tangent = fw.unpack_dual(got)
            assert torch.equal(primal, x) and tangent is not None and torch.equal(tangent, t)


def test_operations_are_seen_by_a_dispatch_mode_as_before():
    from torch.utils._python_dispatch import TorchDispatchMode
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache

    class Count(TorchDispatchMode):
        copies = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.copies += func is torch.ops.aten.copy_.default
            return func(*args, **(kwargs or {}))

    x = torch.randn(1, 2, 20, 128, device=DEV).half()
    with Count() as seen:
        keys, values = ResKVLayerCache(ResKVKernelConfig()).update(x, x + 1, {"raw_keys": x + 2})
    assert torch.equal(keys, x) and torch.equal(values, x + 1) and seen.copies == 3


def test_wrapped_tensors_of_a_transform_are_copied_as_before():
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache

    x, t = (torch.randn(1, 2, 20, 128, device=DEV).half() for _ in range(2))
    window = lambda k: ResKVLayerCache(ResKVKernelConfig()).update(k, k, {"raw_keys": k})[0]
    primal, tangent = torch.func.jvp(window, (x,), (t,))
    assert torch.equal(primal, x) and torch.equal(tangent, t)


def test_a_tensor_without_memory_is_copied_as_before():
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.cache import ResKVLayerCache

    x = torch.randn(1, 2, 20, 128, device=DEV).half()
    zero = torch._efficientzerotensor((1, 2, 20, 128), dtype=torch.float16, device=DEV)
    keys, values = ResKVLayerCache(ResKVKernelConfig()).update(x, zero, {"raw_keys": zero})
    assert torch.equal(keys, x) and not values.any()
