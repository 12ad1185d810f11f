"""Token counts around the edges of the tensor-core decode kernel's passes (two sub-tiles of 128 tokens, the last pass
split in halves of whole eights), segments (32 tokens) and copies, for rows of every width and both column layouts,
against FP32 attention over the reconstructed cache; tokens beyond the end hold NaN."""

import pytest
import torch

from helpers import assert_attention_close, np16, oracle_attention

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _as_oracle(ct):
    p = ct.plan
    return dict(layout=p.layout, bits=p.bits, centroids=np16(ct.centroids), ids=np16(ct.cluster_ids),
                payload=np16(ct.payload), metadata=None if ct.metadata is None else np16(ct.metadata),
                scale=None if ct.scale is None else np16(ct.scale))


@pytest.mark.parametrize("ratio", [1, 4, 8])
@pytest.mark.parametrize("sparsity,bits,layout", [(0.5, 16, "unstructured"), (0.75, 16, "structured"), (0.5, 4, "unstructured"),
                                                  (0.75, 2, "unstructured"), (0.75, 4, "structured")])
@pytest.mark.parametrize("t", [7, 9, 17, 31, 63, 129, 255, 257, 271, 513])
def test_pass_edges(t, sparsity, bits, layout, ratio):
    from reskv_b200 import ResKVKernelConfig, attention, compress
    from reskv_b200.synthetic import gaussian

    b, h, clusters = 1, 2, 40
    cen = gaussian(b, h, clusters, 128, seed=3, device=DEV, std=0.2)
    ids = torch.randint(clusters, (b, h, t), generator=torch.Generator().manual_seed(t), dtype=torch.int32).to(DEV)
    key, value = (gaussian(b, h, t, 128, seed=s, device=DEV, std=0.5) for s in (1, 2))
    cache = compress(key, value,
                     ResKVKernelConfig(sparsity=sparsity, bits=bits, layout=layout), clustering=((cen, ids), (cen, ids)))
    want_parts = _as_oracle(cache.key), _as_oracle(cache.value)
    cache = cache.reserve(t + 300)
    for side in (cache.key, cache.value):
        for buf in side._buffers:
            if buf is not None and buf.is_floating_point():
                buf[:, :, t:] = float("nan")
    q = gaussian(b, h * ratio, 1, 128, seed=4, device=DEV)
    out = attention(q, cache, position=t + 5, start_position=2)
    assert_attention_close(out, oracle_attention(q.cpu(), *want_parts, position=t + 5, start_position=2))
    for splits in (1, 3):  # fixed splits: one segment per CTA, one or several passes
        from dataclasses import replace

        for side in (cache.key, cache.value):
            side.plan = replace(side.plan, splits=splits)
        got = attention(q, cache, position=t + 5, start_position=2)
        assert_attention_close(got, oracle_attention(q.cpu(), *want_parts, position=t + 5, start_position=2))
