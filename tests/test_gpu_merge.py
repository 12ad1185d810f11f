"""The merge kernel at its edges: window lengths around its blocks of 16 and its round of 128 tokens, one to many partial
slots, all head ratios, against FP32 attention over the reconstructed cache."""

import pytest
import torch

from helpers import assert_attention_close, np16, oracle_attention

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _as_oracle(ct):
    p = ct.plan
    return dict(layout=p.layout, bits=p.bits, centroids=np16(ct.centroids), ids=np16(ct.cluster_ids),
                payload=np16(ct.payload), metadata=np16(ct.metadata), scale=None)


@pytest.mark.parametrize("batch,ratio", [(37, 4), (38, 4), (75, 4), (18, 8), (19, 8), (38, 8)])
def test_heads_per_block(batch, ratio):
    """Around the sizes at which a block takes two and four query heads instead of one."""
    _check(batch, 2, ratio, 17, 64, 32)


@pytest.mark.parametrize("ratio", [1, 4, 8])
@pytest.mark.parametrize("tr", [1, 15, 16, 17, 127, 128, 129, 300])
@pytest.mark.parametrize("t,clusters", [(64, 1), (1500, 32), (700, 64)])
def test_window_and_slots(ratio, tr, t, clusters):
    _check(1, 2, ratio, tr, t, clusters)


def _check(b, h, ratio, tr, t, clusters):
    from reskv_b200 import ResKVKernelConfig, attention, compress
    from reskv_b200.synthetic import gaussian, mixture

    cen = gaussian(b, h, clusters, 128, seed=3, device=DEV)
    ids = torch.randint(clusters, (b, h, t), generator=torch.Generator().manual_seed(t), dtype=torch.int32).to(DEV)
    cache = compress(mixture(b, h, t, seed=1, device=DEV), mixture(b, h, t, seed=2, device=DEV),
                     ResKVKernelConfig(sparsity=0.5, max_clusters=64), clustering=((cen, ids), (cen, ids)))
    q, qr = (gaussian(b, h * ratio, 1, 128, seed=s, device=DEV) for s in (4, 5))
    k, v = (gaussian(b, h, tr, 128, seed=s, device=DEV) for s in (6, 7))
    out = attention(q, cache, position=t + tr, recent=(qr, k, v))
    want = oracle_attention(q.cpu(), _as_oracle(cache.key), _as_oracle(cache.value), position=t + tr,
                            recent=(qr.cpu(), k.cpu(), v.cpu()))
    assert_attention_close(out, want)
