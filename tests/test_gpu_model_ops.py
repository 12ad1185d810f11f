"""Fused kernels of the model's prompt pass against plain FP32 tensor operations."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("b,t,hq,hkv", [(1, 1, 1, 1), (2, 3, 4, 1), (1, 65, 8, 2), (3, 17, 8, 8)])
def test_rope_prompt_splits_and_rotates(b, t, hq, hkv):
    from reskv_b200._extension import _stream, bound_library, check

    g = torch.Generator(device=DEV).manual_seed(t)
    qkv = torch.randn(b, t, (hq + 2 * hkv) * 128, generator=g, device=DEV).half()
    angle = torch.arange(t, device=DEV).float()[:, None] * (500000.0 ** (-torch.arange(64, device=DEV).float() / 64))
    cos, sin = angle.cos().contiguous(), angle.sin().contiguous()
    guard = 64  # rows behind the outputs that must stay as they are
    sizes = [b * hq * t * 128] + [b * hkv * t * 128] * 3
    bufs = [torch.full((n + guard,), 7.0, dtype=torch.float16, device=DEV) for n in sizes]
    check(bound_library(qkv.device).reskv_rope_prompt(qkv.data_ptr(), b, t, hq, hkv, cos.data_ptr(), sin.data_ptr(),
                                                      *(x.data_ptr() for x in bufs), _stream(qkv.device)))
    q, k, v = (x.reshape(b, t, -1, 128).transpose(1, 2) for x in qkv.split((hq * 128, hkv * 128, hkv * 128), -1))

    def rotate(x):
        lo, hi = x.float()[..., :64], x.float()[..., 64:]
        return torch.cat((lo * cos - hi * sin, hi * cos + lo * sin), -1)

    for buf, n, want, exact in zip(bufs, sizes, (rotate(q), k, rotate(k), v), (False, True, False, True)):
        assert (buf[n:] == 7.0).all()
        got = buf[:n].view(want.shape).float()
        if exact:
            assert torch.equal(got, want.float())
        else:
            torch.testing.assert_close(got, want, atol=2e-3, rtol=1e-3)


def test_a_second_generation_captures_again_in_the_same_pool():
    """Two generations with different prompts on one model: the second capture gives the eager logits, too."""
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.models import LlamaShape, ResKVLlama

    cfg = ResKVKernelConfig(num_clusters=4, max_clusters=8, group_size=16, recent_size=8, kmeans_iterations=2)
    model = ResKVLlama(LlamaShape(hidden=256, layers=2, heads=8, kv_heads=2, ffn=512, vocab=320), cfg, seed=5)
    gen = torch.Generator().manual_seed(1)
    for batch, length in ((2, 70), (1, 100), (2, 41)):
        ids = torch.randint(0, 320, (batch, length), generator=gen).cuda()
        eager = [model.prefill(ids, reserve=40)]
        for i in range(20):
            eager.append(model.decode(ids[:, i]))
        model.prefill(ids, reserve=40)
        model.begin_graph_decode(batch)
        for i in range(20):
            torch.testing.assert_close(model.decode_graph(ids[:, i]), eager[i + 1], atol=2e-2, rtol=2e-2)
